"""The fields' far kernel at the edges of its work division: groups around a chunk of 256 targets
and its multiples, every order, delta positive, zero and negative.  FP64 against the oracle's
force to 1e-12 of the largest value (a few hundred roundings of 1.1e-16 a cluster); mixed to
2e-6 (a few tens of roundings of 6e-8 a cluster, of either sign).  The screened field against the
direct sum: with cluster ratios below sqrt(0.05), order 10 leaves at most 11 * 0.05^5 / (1 - 0.23) =
5e-6 of each pair's size."""
import numpy as np
import pytest

from test_gpu_field_direct_edges import curl_field, pairs

pytestmark = pytest.mark.gpu


def compare(ctx, orc, x, y, z, q, maxmemb, nterms, acc, delta, tol32=2e-6):
    import bit_b200 as B
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, nterms)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, nterms)
    want = np.stack(T.evaluate_force(delta, acc))
    size = np.max(np.abs(want))
    for prec, tol in ((B.FP64, 1e-12), (B.MIXED, tol32)):
        got = np.stack(t.treeforce(acc, delta, prec))
        assert np.max(np.abs(got - want)) <= tol * size
        again = np.stack(t.treeforce(acc, delta, prec))
        assert np.array_equal(got, again)
    t.treeempty()


@pytest.mark.parametrize("maxmemb", [31, 33, 255, 256, 257, 511, 513, 1000, 1024])
def test_groups_around_the_chunks(ctx, orc, maxmemb):
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(9 * maxmemb + 300, seed=maxmemb)
    compare(ctx, orc, x, y, z, q, maxmemb, 5, 0.8, 1e-3)


@pytest.mark.parametrize("n,maxmemb", [(20000, 200), (50000, 300), (100000, 300), (150000, 1000)])
def test_larger_systems_take_larger_chunks(ctx, orc, n, maxmemb):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(n, seed=n)
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, 4)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, 4)
    tg = workloads.sample_targets(n, 400, seed=1)
    want = np.stack(T.evaluate_force(1e-3, 0.7, targets=tg))
    for prec, tol in ((B.FP64, 1e-12), (B.MIXED, 2e-6)):
        got = np.stack(t.treeforce(0.7, 1e-3, prec))[:, tg]
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
    t.treeempty()


@pytest.mark.parametrize("nterms", range(1, 11))
@pytest.mark.parametrize("delta", [1e-2, 0.0, -1e-9])
def test_every_order_and_sign_of_delta(ctx, orc, nterms, delta):
    from bit_b200 import workloads
    x, y, z, q = workloads.uniform_cube(4000, seed=nterms)
    compare(ctx, orc, x, y, z, q, 60, nterms, 0.6, delta)


@pytest.mark.parametrize("maxmemb", [40, 300])
def test_screened_field_tends_to_the_direct_sum(ctx, orc, maxmemb):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(3000, seed=maxmemb)
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, 10)
    got = np.stack(t.field(B.FIELD_SCREENED, acc=0.05, kappa=1.3))
    want = curl_field(x, y, z, q, 1.3)
    _, r2 = pairs(x, y, z)
    np.fill_diagonal(r2, 1.0)
    r = np.sqrt(r2)
    w = np.exp(-1.3 * r) / r * (1.3 + 1 / r) * np.abs(q)
    np.fill_diagonal(w, 0.0)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, 10)
    assert T.count(orc.params(orc.SCREENED, acc=0.05, kappa=1.3))[0] > 0
    assert np.max(np.abs(got - want) / w.sum(1)) <= 5e-6
    t.treeempty()
