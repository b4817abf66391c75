"""The fields' near kernel and the direct sums at the edges of their work division: every
remainder of a block of targets, one source, groups in several parts, few targets; against
sums in numpy (FP64, 1e-12 of the largest value: at most 5,000 pairs of either sign, each
within a few roundings of 1.1e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pairs(x, y, z):
    d = np.stack([a[:, None] - a[None, :] for a in (x, y, z)])
    return d, (d * d).sum(0)


def coulomb_field(x, y, z, q, delta):
    d, r2 = pairs(x, y, z)
    r2 = r2 + delta
    np.fill_diagonal(r2, np.inf)
    return (d * (q * r2 ** -1.5)).sum(2)


def curl_field(x, y, z, q, kappa):
    d, r2 = pairs(x, y, z)
    np.fill_diagonal(r2, 1.0)
    r = np.sqrt(r2)
    w = np.exp(-kappa * r) / r2 * (kappa + 1 / r) * q
    np.fill_diagonal(w, 0.0)
    return np.stack([-(d[1] * w).sum(1), (d[0] * w).sum(1), np.zeros(len(x))])


def check(got, want, tol):
    assert np.max(np.abs(got - want)) <= tol * max(np.max(np.abs(want)), 1e-300)


@pytest.mark.parametrize("n,maxmemb", [(1, 1), (2, 2), (31, 31), (33, 33), (49, 49), (64, 64), (65, 65),
                                       (113, 113), (600, 50), (1025, 1025), (3000, 1500)])
def test_fields_of_every_list_length(ctx, n, maxmemb):
    import bit_b200 as B
    rng = np.random.default_rng(n)
    x, y, z, q = rng.uniform(-1, 1, (4, n))
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, 2)
    want = coulomb_field(x, y, z, q, 1e-3)
    for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
        got = np.stack(t.treeforce(0.0, 1e-3, prec))
        check(got, want, tol)
        np.testing.assert_array_equal(got, np.stack(t.treeforce(0.0, 1e-3, prec)))
    for kappa in (1.5, 5000.0):  # the second underflows for most pairs
        got = np.stack(t.field(B.FIELD_SCREENED, acc=0.0, kappa=kappa))
        check(got, curl_field(x, y, z, q, kappa), 1e-12)
    order = np.stack(t.field(B.FIELD_COULOMB, acc=0.0, del_=1e-3, kernel_order=0))
    check(order, want, 1e-12)
    t.treeempty()


@pytest.mark.parametrize("kappa,del_", [(1.0, 0.0), (0.5, 1e-3)])
@pytest.mark.parametrize("m", [1, 2, 63, 64, 65, 129, 513])
@pytest.mark.parametrize("n", [1, 511, 513, 4000])
def test_direct_sums_of_every_shape(ctx, orc, n, m, kappa, del_):
    import bit_b200 as B
    rng = np.random.default_rng(n + m)
    x, y, z, q = rng.uniform(-1, 1, (4, n))
    tg = np.sort(rng.integers(0, n, m)).astype(np.int32)
    for kb, ko in ((B.COULOMB, orc.COULOMB), (B.SCREENED, orc.SCREENED), (B.SCREENED_REG, orc.SCREENED_REG)):
        want = orc.direct(x, y, z, q, orc.params(ko, orc.MODE_CONSISTENT, kappa=kappa, del_=del_), tg)
        got = ctx.direct(x, y, z, q, B.params(kb, B.CONSISTENT, B.FP64, kappa=kappa, del_=del_), tg)
        check(got, want, 1e-12)


def test_direct_sums_of_coincident_particles(ctx, orc):
    """Coulomb skips a pair at distance 0; the screened sum is infinite, as the plain formula."""
    import bit_b200 as B
    rng = np.random.default_rng(4)
    x, y, z = rng.uniform(-1, 1, (3, 700))
    q = rng.uniform(0.1, 1, 700)
    x[650], y[650], z[650] = x[3], y[3], z[3]
    tg = np.array([0, 3, 5, 650], np.int32)
    for kb, ko in ((B.COULOMB, orc.COULOMB), (B.SCREENED, orc.SCREENED)):
        want = orc.direct(x, y, z, q, orc.params(ko, orc.MODE_CONSISTENT, kappa=1.0), tg)
        got = ctx.direct(x, y, z, q, B.params(kb, B.CONSISTENT, B.FP64, kappa=1.0), tg)
        fine = np.isfinite(want)
        np.testing.assert_array_equal(got[~fine], want[~fine])
        np.testing.assert_allclose(got[fine], want[fine], rtol=1e-12)
