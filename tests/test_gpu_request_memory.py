"""Device memory of a served request.  A request runs within its own reservation (64 MB and 448
bytes a particle, or what its slot holds), at leaf sizes and theta where its interaction lists
are most of its memory, and with the same bits as without a limit.  A request that does need more
fails by itself: what the slot's context has freed serves the next ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,maxmemb,nterms,acc", [(20000, 20, 5, 0.015), (20000, 20, 9, 0.05), (60000, 60, 5, 0.015),
                                                  (60000, 60, 9, 0.05), (200000, 200, 9, 0.05)])
def test_long_lists_within_a_requests_reservation(ctx, n, maxmemb, nterms, acc):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(n, seed=n)
    srv = B.Server(slots=1)
    for prec in (B.FP64, B.MIXED):
        p = B.params(B.SCREENED, B.CONSISTENT, prec, kappa=1.0, acc=acc)
        got, info, st = srv.wait(srv.submit_eval(x, y, z, q, nterms, maxmemb, p))
        assert st == 0, info
        assert info["peak_bytes"] <= info["bytes_reserved"]
        np.testing.assert_array_equal(got, ctx.treecode_potential(x, y, z, q, nterms, maxmemb, p))
    srv.close()


def test_requests_after_one_that_failed(ctx):
    """Lists of some 40 million entries do not fit 149 MB; what follows in the slot does."""
    import bit_b200 as B
    from bit_b200 import workloads
    srv = B.Server(slots=1)
    x, y, z, q = workloads.clustered_blobs(200000, seed=1)
    p = B.params(B.COULOMB, B.CONSISTENT, B.MIXED, del_=1e-6, acc=0.015)
    assert srv.wait(srv.submit_eval(x, y, z, q, 9, 20, p))[2] == 9  # over its reservation
    for k, (n, maxmemb) in enumerate([(1000, 50), (30000, 300), (5000, 20), (100000, 500), (2000, 2000)]):
        x, y, z, q = workloads.clustered_blobs(n, seed=k)
        p = B.params(B.COULOMB, B.CONSISTENT, B.MIXED, del_=1e-6, acc=0.5)
        got, info, st = srv.wait(srv.submit_eval(x, y, z, q, 7, maxmemb, p))
        assert st == 0, (n, info)
        np.testing.assert_array_equal(got, ctx.treecode_potential(x, y, z, q, 7, maxmemb, p))
    srv.close()


def test_a_context_of_any_budget(ctx):
    """A context is made whatever its budget; the calls that need memory fail, by themselves."""
    import bit_b200 as B
    x, y, z, q = np.random.default_rng(1).uniform(-1, 1, (4, 1000))
    for budget in (1, 1000, 5000):
        c = B.Context(hbm_budget=budget)
        for _ in range(2):
            with pytest.raises(B.BitError) as e:
                c.treemake(x, y, z, 50)
            assert e.value.status == 9
        c.close()
