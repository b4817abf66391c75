"""The order of external points, where its runs and merges can go wrong: one run, a remainder of
one, one, two and three merges, every group size; equal points, points on a line, one far away.  Each point's value agrees
with the oracle's to 1e-12 of the largest (one rounding of 1.1e-16 per pair, 3,000 pairs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(kind, m):
    r = np.random.default_rng(m)
    p = r.uniform(-1, 1, (m, 3))
    if kind == "equal":
        p[:] = 0.3, -0.2, 1.1
    elif kind == "line":
        p[:, 1:] = 0.25
    elif kind == "pairs":  # half the points twice, and one far from the rest
        p[m // 2:] = p[:m - m // 2][::-1]
        p[0] = 1e6, -1e6, 3.0
    return p


@pytest.mark.parametrize("kind,m", [(k, m) for k in ("cube", "equal", "line", "pairs")
                                    for m in (1, 511, 512, 513, 4095, 4097, 33001)]
                         + [("cube", 28416), ("cube", 28417), ("pairs", 70001), ("cube", 120001)])
def test_each_point_gets_its_own_value(ctx, orc, kind, m):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.uniform_cube(3000, seed=5)
    t = ctx.treemake(x, y, z, 100)
    t.treemoments(q, 4)
    T = orc.Tree(x, y, z, 100)
    T.compute_moments(q, 4)
    pts = points(kind, m)
    got = t.evaluate(B.params(B.COULOMB, B.CONSISTENT, B.FP64, acc=0.5, del_=1e-3), points=pts)
    want = T.evaluate(orc.params(orc.COULOMB, orc.MODE_CONSISTENT, acc=0.5, del_=1e-3), points=pts)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    t.treeempty()


def test_nan_is_refused_anywhere_and_infinity_is_not(ctx):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.uniform_cube(2000, seed=6)
    t = ctx.treemake(x, y, z, 100)
    t.treemoments(q, 3)
    p = B.params(B.COULOMB, B.CONSISTENT, B.FP64, acc=0.5, del_=1e-3)
    pts = points("cube", 1500)
    ref = t.evaluate(p, points=pts)
    for i, a in ((0, 0), (700, 1), (1499, 2)):
        bad = pts.copy()
        bad[i, a] = np.nan
        with pytest.raises(Exception):
            t.evaluate(p, points=bad)
    far = pts.copy()
    far[3, 1] = -np.inf
    got = t.evaluate(p, points=far)
    keep = np.arange(1500) != 3
    assert np.max(np.abs(got - ref)[keep]) <= 1e-12 * np.max(np.abs(ref))
    t.treeempty()
