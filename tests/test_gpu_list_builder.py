"""The list builder where its work division can go wrong: groups of one mask word to 32, trees
whose levels hold more nodes than one round of visits, groups that overrun the first build's
regions, and arrays that overflow.  Pair counts equal the oracle traversal's; values agree to
1e-12 of the largest (one rounding of 1.1e-16 per pair, at most 5,000 pairs); a build that was run
again gives the same bits as one that was not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 32, 33, 65, 97, 128, 129, 160, 225, 256, 289, 513])
def test_points_of_every_remainder(ctx, orc, m):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(4000, seed=m)
    pts = np.random.default_rng(m).uniform(-1.2, 1.2, (m, 3))
    t = ctx.treemake(x, y, z, 9)
    t.treemoments(q, 2)
    T = orc.Tree(x, y, z, 9)
    T.compute_moments(q, 2)
    for acc in (0.02, 0.3, 0.9):
        want = T.evaluate(orc.params(orc.COULOMB, orc.MODE_CONSISTENT, acc=acc, del_=1e-3), points=pts)
        got = t.evaluate(B.params(B.COULOMB, B.CONSISTENT, B.FP64, acc=acc, del_=1e-3), points=pts)
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    t.treeempty()


@pytest.mark.parametrize("size", [32, 33, 64, 65, 96, 128, 129, 160, 256, 288, 992, 1024])
def test_packed_leaves_of_every_mask_width(orc, size):
    """Runs of small leaves packed to groups of up to `size` targets: 1 to 32 mask words."""
    import bit_b200 as B
    from bit_b200 import workloads
    ctx = B.Context()
    ctx.set_group_size(size)
    n = 4000
    x, y, z, q = workloads.clustered_blobs(n, seed=size)
    t = ctx.treemake(x, y, z, 9)
    t.treemoments(q, 2)
    T = orc.Tree(x, y, z, 9)
    T.compute_moments(q, 2)
    for acc in (0.02, 0.3, 0.9):
        nf, nn, _ = T.count(orc.params(orc.COULOMB, acc=acc, del_=1e-3))
        want = T.evaluate(orc.params(orc.COULOMB, orc.MODE_CONSISTENT, acc=acc, del_=1e-3))
        got = t.evaluate(B.params(B.COULOMB, B.CONSISTENT, B.FP64, acc=acc, del_=1e-3))
        st = t.stats()
        assert st["far_pairs"] == nf and st["near_pairs"] - n == nn
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    t.treeempty()


@pytest.mark.parametrize("n,maxmemb,acc", [
    (300, 300, 0.5), (3000, 2, 0.02), (6000, 3, 0.3), (20000, 40, 0.05), (9000, 1000, 0.6),
])
def test_same_lists_when_the_build_is_run_again(orc, n, maxmemb, acc):
    import bit_b200 as B
    from bit_b200 import workloads
    ctx = B.Context()
    x, y, z, q = workloads.clustered_blobs(n, seed=n)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, 3)
    nf, nn, _ = T.count(orc.params(orc.COULOMB, acc=acc, del_=1e-3))
    p = B.params(B.COULOMB, B.CONSISTENT, B.FP64, acc=acc, del_=1e-3)
    got, again = [], []
    for _ in range(2):
        t = ctx.treemake(x, y, z, maxmemb)
        t.treemoments(q, 3)
        got.append(t.evaluate(p))
        st = t.stats()
        again.append(st["list_fallback"])
        assert st["far_pairs"] == nf and st["near_pairs"] - n == nn
        t.treeempty()
    assert again[1] == 0
    if maxmemb == 2 and acc == 0.02:  # visits nearly every node: past the first allowance
        assert again[0] == 1
    assert np.array_equal(got[0], got[1])
    want = T.evaluate(orc.params(orc.COULOMB, orc.MODE_CONSISTENT, acc=acc, del_=1e-3))
    assert np.max(np.abs(got[0] - want)) <= 1e-12 * np.max(np.abs(want))
