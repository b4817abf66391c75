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
