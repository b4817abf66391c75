"""Fields at the ends of their arguments' ranges: a negative delta (the entry points take any finite
one) beside clusters of no extent, distances whose squares leave FP64's range, and screened fields
that grow with the distance (kappa < 0, which the entry points take too)."""
import numpy as np
import pytest

from test_gpu_field_direct_edges import check, coulomb_field, curl_field
from test_gpu_field_far import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nterms", [3, 9, 10])
@pytest.mark.parametrize("scale", [1.0, 1e10])
def test_negative_delta_beside_clusters_of_one_particle(ctx, orc, nterms, scale):
    """A lattice at spacing `scale`, delta = -0.3 scale^2, a particle a leaf: a cluster of no extent
    and a large negative delta.  r^2 of a pair is at least 0.64 scale^2, so r^2 + delta loses
    0.94 / 0.34 = 2.8 of its roundings, and its power 3/2 four: 1e-5 in place of 2e-6."""
    rng = np.random.default_rng(nterms)
    g = np.stack(np.meshgrid(*[np.arange(9.0)] * 3, indexing="ij")).reshape(3, -1)
    x, y, z = (g + rng.uniform(-0.1, 0.1, g.shape)) * scale
    compare(ctx, orc, x, y, z, rng.uniform(-1, 1, g.shape[1]), 1, nterms, 0.5, -0.3 * scale ** 2, 1e-5)


@pytest.mark.parametrize("n", [1, 20, 33, 49, 70, 150])
def test_distances_whose_squares_overflow(ctx, n):
    """n particles near the origin and n some 1e160 away, 1e150 apart: a pair of the two kinds, or of
    two of the far ones, adds 0."""
    import bit_b200 as B
    rng = np.random.default_rng(n)
    p = rng.uniform(-1, 1, (3, 2 * n))
    p[:, n:] = 1e160 * (1.0 + 1e-10 * p[:, n:])
    q = rng.uniform(-1, 1, 2 * n)
    near = slice(0, n)
    for maxmemb in (2 * n, n):
        t = ctx.treemake(*p, maxmemb)
        t.treemoments(q, 2)
        for got, want in ((t.treeforce(0.0, 1e-3), coulomb_field(*p[:, near], q[near], 1e-3)),
                          (t.field(B.FIELD_SCREENED, acc=0.0, kappa=1.5), curl_field(*p[:, near], q[near], 1.5))):
            got = np.stack(got)
            assert not np.any(got[:, n:])
            check(got[:, near], want, 1e-12)
        t.treeempty()


@pytest.mark.parametrize("extent", [10.0, 690.0, 703.0, 760.0])
@pytest.mark.parametrize("n", [40, 300])
def test_screened_field_that_grows(ctx, n, extent):
    """kappa < 0 to where exp(-kappa R) nears FP64's largest number, e^709.78, and past it, where the
    field is infinite (or infinities of either sign meet); kappa R rounds as in the tests of the
    strong screening, so 1e-12 of the terms' sizes."""
    import bit_b200 as B
    rng = np.random.default_rng(n)
    p = rng.uniform(0, 1, (3, n))
    p[:, 0], p[:, 1] = 0.0, 1.0
    kappa = -3.0
    p *= extent / 3.0 / np.sqrt(3.0)
    q = rng.uniform(-1, 1, n) * 1e-6
    t = ctx.treemake(*p, 40)
    t.treemoments(q, 2)
    fx, fy, fz = t.field(B.FIELD_SCREENED, acc=0.0, kappa=kappa)
    t.treeempty()
    d = (p[:, :, None] - p[:, None, :]).astype(np.longdouble)
    r = np.sqrt((d * d).sum(0))
    np.fill_diagonal(r, 1.0)
    w = q * np.exp(-np.longdouble(kappa) * r) / (r * r) * (kappa + 1 / r)
    np.fill_diagonal(w, 0.0)
    most = np.max(-kappa * r, axis=1)
    inside, outside = most < 709.5, most > 710.0
    assert np.any(outside) == (extent > 710)
    for got, terms in ((fx, -d[1] * w), (fy, d[0] * w)):
        assert np.all(np.abs(got - terms.sum(1))[inside] <= 1e-12 * np.abs(terms).sum(1)[inside])
        assert not np.any(np.isfinite(got[outside]))
    assert not np.any(fz)
