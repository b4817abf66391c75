"""The near field where its work division can go wrong: lists of every remainder of a block of
64 targets, leaves that end inside a source tile, one source, groups cut into several parts,
and exponentials that underflow.  FP64 against the oracle's direct sum to 1e-12 of the largest
value (one rounding of 1.1e-16 per pair, at most 5,000 pairs of either sign); mixed to 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 97, 112, 113, 129, 200, 1025]


def kernels(B, orc):
    return [(B.COULOMB, orc.COULOMB, dict(del_=0.0)), (B.COULOMB, orc.COULOMB, dict(del_=1e-3)),
            (B.SCREENED, orc.SCREENED, dict(kappa=1.5)),
            (B.SCREENED_REG, orc.SCREENED_REG, dict(kappa=0.7, del_=1e-3))]


def check(got, want, tol):
    assert np.max(np.abs(got - want)) <= tol * max(np.max(np.abs(want)), 1e-300)


@pytest.mark.parametrize("n", SIZES)
def test_single_leaf_of_every_size(ctx, orc, n):
    import bit_b200 as B
    rng = np.random.default_rng(n)
    x, y, z, q = rng.uniform(-1, 1, (4, n))
    t = ctx.treemake(x, y, z, n)
    t.treemoments(q, 2)
    tg = np.arange(n, dtype=np.int32)
    for kb, ko, kw in kernels(B, orc):
        want = orc.direct(x, y, z, q, orc.params(ko, orc.MODE_CONSISTENT, acc=0.0, **kw), tg)
        for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
            check(t.evaluate(B.params(kb, B.CONSISTENT, prec, acc=0.0, **kw)), want, tol)
    t.treeempty()


@pytest.mark.parametrize("m", [1, 31, 33, 50, 64, 255, 256, 257])
def test_points_of_every_list_length(ctx, orc, m):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(1500, seed=m)
    pts = np.random.default_rng(m).uniform(-1.5, 1.5, (m, 3))
    t = ctx.treemake(x, y, z, 70)
    t.treemoments(q, 6)
    T = orc.Tree(x, y, z, 70)
    T.compute_moments(q, 6)
    for kb, ko, kw in kernels(B, orc):
        want = T.evaluate(orc.params(ko, orc.MODE_CONSISTENT, acc=0.4, **kw), points=pts)
        for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
            check(t.evaluate(B.params(kb, B.CONSISTENT, prec, acc=0.4, **kw), points=pts), want, tol)
    t.treeempty()


@pytest.mark.parametrize("n,maxmemb", [(4000, 900), (5000, 60), (3000, 3000)])
def test_groups_in_several_parts(ctx, orc, n, maxmemb):
    """acc = 0: every pair is a near pair, so groups of 900 hold millions and are cut into
    parts whose sums meet in scratch; the result is the same on every call."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(n, seed=3)
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, 2)
    tg = np.arange(n, dtype=np.int32)
    for kb, ko, kw in kernels(B, orc):
        want = orc.direct(x, y, z, q, orc.params(ko, orc.MODE_CONSISTENT, acc=0.0, **kw), tg)
        for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
            p = B.params(kb, B.CONSISTENT, prec, acc=0.0, **kw)
            a = t.evaluate(p)
            check(a, want, tol)
            np.testing.assert_array_equal(a, t.evaluate(p))
    t.treeempty()


@pytest.mark.parametrize("kappa", [300.0, 2000.0, 1e5, 1e9])
def test_strong_screening_underflows_to_zero(ctx, orc, kappa):
    """kappa R from below the limit of the check-free exponential to past 32-bit exponents."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(600, seed=5)
    t = ctx.treemake(x, y, z, 50)
    t.treemoments(q, 2)
    tg = np.arange(600, dtype=np.int32)
    want = orc.direct(x, y, z, q, orc.params(orc.SCREENED, orc.MODE_CONSISTENT, acc=0.0, kappa=kappa), tg)
    got = t.evaluate(B.params(B.SCREENED, B.CONSISTENT, B.FP64, acc=0.0, kappa=kappa))
    assert np.all(np.abs(got - want) <= 1e-12 * np.abs(want) + 1e-300)
    t.treeempty()


@pytest.mark.parametrize("m", [1, 40, 300])
def test_points_with_no_near_entries(ctx, orc, m):
    """Points far outside: every cluster is accepted at the root, the near lists are empty."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(1500, seed=9)
    pts = np.random.default_rng(m).uniform(-1, 1, (m, 3)) + 40.0
    t = ctx.treemake(x, y, z, 70)
    t.treemoments(q, 6)
    T = orc.Tree(x, y, z, 70)
    T.compute_moments(q, 6)
    for kb, ko, kw in kernels(B, orc)[:2]:
        want = T.evaluate(orc.params(ko, orc.MODE_CONSISTENT, acc=0.4, **kw), points=pts)
        for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
            check(t.evaluate(B.params(kb, B.CONSISTENT, prec, acc=0.4, **kw), points=pts), want, tol)
    t.treeempty()


@pytest.mark.parametrize("n,maxmemb", [(3000, 100), (9000, 700)])
def test_close_pairs_across_leaves(ctx, orc, n, maxmemb):
    """Partners on either side of the tree's first cuts, 1e-7 to 1e-3 apart: the loop that watches
    for close pairs meets them in other leaves than the target's own, and is done again."""
    import bit_b200 as B
    rng = np.random.default_rng(n)
    p = rng.uniform(-1, 1, (3, n))
    for a in range(3):
        i = rng.choice(n, 60, replace=False)
        gap = 10.0 ** rng.uniform(-7, -3, 30)
        p[:, i[30:]] = p[:, i[:30]]
        p[a, i[:30]], p[a, i[30:]] = gap / 2, -gap / 2
    p[:, 0], p[:, 1] = 1.0, -1.0  # the box is symmetric: cuts through 0
    q = rng.uniform(-1, 1, n)
    t = ctx.treemake(*p, maxmemb)
    t.treemoments(q, 2)
    tg = np.arange(n, dtype=np.int32)
    for kb, ko, kw in kernels(B, orc):
        want = orc.direct(*p, q, orc.params(ko, orc.MODE_CONSISTENT, acc=0.0, **kw), tg)
        for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 1e-6)):
            check(t.evaluate(B.params(kb, B.CONSISTENT, prec, acc=0.0, **kw)), want, tol)
    t.treeempty()
