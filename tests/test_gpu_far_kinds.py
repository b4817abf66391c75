"""The far field's four kinds (delta = 0 or not, screened or not) against the oracle's
Taylor recurrences at the edges of their ranges: no regularisation, one above the cluster
size, no and strong screening, clusters of one particle, groups that end inside a mask word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [("coulomb", dict(del_=0.0)), ("coulomb", dict(del_=0.3)),
         ("screened", dict(kappa=0.0)), ("screened", dict(kappa=20.0)),
         ("reg", dict(kappa=0.7, del_=0.0)), ("reg", dict(kappa=5.0, del_=0.3)),
         ("reg", dict(kappa=0.0, del_=1e-4))]


@pytest.mark.parametrize("nterms", [1, 2, 6, 7, 9, 10])
@pytest.mark.parametrize("n,maxmemb", [(300, 1), (3000, 33), (5001, 700)])
def test_far_kinds_match_oracle(ctx, orc, nterms, n, maxmemb):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(n, seed=nterms)
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, nterms)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, nterms)
    ids = {"coulomb": (B.COULOMB, orc.COULOMB), "screened": (B.SCREENED, orc.SCREENED),
           "reg": (B.SCREENED_REG, orc.SCREENED_REG)}
    for kern, kw in KINDS:
        kb, ko = ids[kern]
        want = T.evaluate(orc.params(ko, orc.MODE_CONSISTENT, acc=0.6, **kw))
        got = t.evaluate(B.params(kb, B.CONSISTENT, B.FP64, acc=0.6, **kw))
        assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want), (kern, kw)
        mixed = t.evaluate(B.params(kb, B.CONSISTENT, B.MIXED, acc=0.6, **kw))
        assert np.linalg.norm(mixed - want) < 1e-6 * np.linalg.norm(want), (kern, kw)
    t.treeempty()


@pytest.mark.parametrize("n,maxmemb", [(2500, 1000), (12000, 900), (30000, 1000), (60000, 1000), (200000, 1000)])
def test_every_chunk_of_a_group(ctx, orc, n, maxmemb):
    """Few large groups are cut into chunks of 32 targets and up, many are taken whole; a target's
    result does not depend on it: alone and beside a larger system it is the same."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(n, seed=n)
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, 4)
    T = orc.Tree(x, y, z, maxmemb)
    T.compute_moments(q, 4)
    tg = workloads.sample_targets(n, 400, seed=2)
    want = T.evaluate(orc.params(orc.SCREENED, orc.MODE_CONSISTENT, acc=0.8, kappa=1.0), targets=tg)
    p = B.params(B.SCREENED, B.CONSISTENT, B.FP64, acc=0.8, kappa=1.0)
    got = t.evaluate(p)
    assert np.linalg.norm(got[tg] - want) < 1e-12 * np.linalg.norm(want)
    t.treeempty()
    X, Y, Z, Q = workloads.uniform_cube(250000, seed=1)
    f = ctx.forest(np.concatenate([x, X]), np.concatenate([y, Y]), np.concatenate([z, Z]), [n, 250000], maxmemb)
    f.set_charges(np.concatenate([q, Q]))
    f.moments([4, 4])
    assert np.array_equal(f.evaluate([p, p])[:n], got)
    f.treeempty()
