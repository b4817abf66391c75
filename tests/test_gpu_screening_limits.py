"""Screening so strong that exponentials come near the end of their range.  The near field takes
an exponential without an underflow check where kappa times the system's extent is below 700, on
small systems of large kappa too; the target's own source adds nothing whatever kappa is.

Against sums in numpy's long double: kappa R is at most about 715 and rounds to 1.1e-16 of itself
in a few steps, so a term is within 715 * 4 * 1.1e-16 = 3.2e-13 of its value, and the tolerance
is 1e-12 of the sum of the terms' sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(n, kappa, extent, seed):
    """n particles in a box whose diagonal times kappa is `extent`."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(0, 1, (3, n))
    p[:, 0], p[:, 1] = 0.0, 1.0
    return p * (extent / kappa / np.sqrt(3.0)), rng.uniform(-1, 1, n)


def terms(p, q, kappa, delta=0.0):
    """Differences, distances and q e^(-kappa R) of every pair, without the diagonal's."""
    d = (p[:, :, None] - p[:, None, :]).astype(np.longdouble)
    r = np.sqrt((d * d).sum(0) + np.longdouble(delta))
    np.fill_diagonal(r, 1.0)
    e = q * np.exp(-np.longdouble(kappa) * r)
    np.fill_diagonal(e, 0.0)
    return d, r, e


def check(got, terms_):
    err = np.abs(got - terms_.sum(1))
    assert np.all(np.isfinite(got))
    assert np.all(err <= 1e-12 * np.abs(terms_).sum(1) + 1e-300)


@pytest.mark.parametrize("kappa", [150.0, 709.4, 2129.0, 1e5])
@pytest.mark.parametrize("extent", [690.0, 715.0])
def test_potentials_at_the_limit_of_the_unchecked_exponential(ctx, kappa, extent):
    import bit_b200 as B
    p, q = cloud(300, kappa, extent, 1)
    t = ctx.treemake(*p, 40)
    t.treemoments(q, 2)
    d, r, e = terms(p, q, kappa)
    check(t.evaluate(B.params(B.SCREENED, B.CONSISTENT, B.FP64, kappa=kappa, acc=0.0)), -e / r)
    delta = (3.0 / kappa) ** 2
    d, r, e = terms(p, q, kappa, delta)
    check(t.evaluate(B.params(B.SCREENED_REG, B.CONSISTENT, B.FP64, kappa=kappa, del_=delta, acc=0.0)), e / r)
    t.treeempty()


@pytest.mark.parametrize("kappa", [150.0, 709.4, 2129.0, 1e5])
@pytest.mark.parametrize("extent", [690.0, 715.0])
def test_field_at_the_limit_of_the_unchecked_exponential(ctx, kappa, extent):
    import bit_b200 as B
    p, q = cloud(300, kappa, extent, 2)
    t = ctx.treemake(*p, 40)
    t.treemoments(q, 2)
    d, r, e = terms(p, q, kappa)
    w = e / (r * r) * (kappa + 1 / r)
    fx, fy, fz = t.field(B.FIELD_SCREENED, acc=0.0, kappa=kappa)
    check(fx, -d[1] * w)
    check(fy, d[0] * w)
    assert not np.any(fz)
    t.treeempty()


@pytest.mark.parametrize("nterms", [3, 9, 10])
@pytest.mark.parametrize("kappa", [3e3, 1e5, 1e7, 1e12, 1e25])
def test_far_field_of_clusters_many_screening_lengths_wide(ctx, nterms, kappa):
    """Accepted clusters lie so many screening lengths away that their potential is 0; powers of
    kappa times their size, up to the eighth, and of kappa times the distance leave FP32's range."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(4000, seed=3)
    far = np.random.default_rng(4).uniform(-1, 1, (100, 3)) * 10.0 ** np.arange(1, 11).repeat(10)[:, None] + 50.0
    t = ctx.treemake(x, y, z, 60)
    t.treemoments(q, nterms)
    for kernel, delta in ((B.SCREENED, 0.0), (B.SCREENED_REG, 1e-4)):
        got = {}
        for prec in (B.FP64, B.MIXED):
            p = B.params(kernel, B.CONSISTENT, prec, kappa=kappa, del_=delta, acc=0.5)
            got[prec] = t.evaluate(p)
            assert not np.any(t.evaluate(p, points=far))
        assert np.all(np.isfinite(got[B.FP64]))
        # (FP32 holds nothing below 1e-45; kappa R rounds to 6e-8 of at most 100)
        assert np.max(np.abs(got[B.MIXED] - got[B.FP64])) <= 1e-5 * np.max(np.abs(got[B.FP64])) + 1e-40
    t.treeempty()
