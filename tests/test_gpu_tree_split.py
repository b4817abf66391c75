"""The tree build where nodes change from one CTA's work to a cluster's (3,584 and 14,336
members; 57,344 and 114,688 to all SMs'), on shapes that exercise every branch of the split program:
bit for bit the oracle's tree."""
import numpy as np
import pytest

from test_gpu_tree import assert_same_bits

pytestmark = pytest.mark.gpu


def shape(kind, n, seed):
    from bit_b200 import workloads
    rng = np.random.default_rng(seed)
    if kind == "blobs":
        return workloads.clustered_blobs(n, seed=seed)[:3]
    p = rng.uniform(-1, 1, (3, n))
    if kind == "slab":            # thin in z: x and y splits only
        p[2] *= 1e-3
    elif kind == "rod":           # long in y
        p[0] *= 0.01
        p[2] *= 0.01
    elif kind == "plane":         # zero extent: NaN and infinite aspect ratios
        p[2] = 0.25
    elif kind == "line":
        p[1] = -0.5
        p[2] = 0.0
    elif kind == "graded":        # deep: geometric spacing towards the origin
        p *= 2.0 ** -rng.uniform(0, 40, n)
    elif kind == "lattice":       # many coordinates on the midpoints, -0.0 among them
        p = np.round(p * 8) / 8 + 0.0 * p
        p = p + rng.choice([0.0, 1e-9], (3, n)) * np.arange(n)
    return p[0].copy(), p[1].copy(), p[2].copy()


@pytest.mark.parametrize("n,maxmemb", [(1, 1), (2, 1), (700, 1), (3584, 60), (3585, 60), (14336, 500),
                                       (14337, 64), (57344, 800), (57345, 800), (90001, 30000), (114688, 900),
                                       (114689, 900), (150001, 60000)])
@pytest.mark.parametrize("kind", ["cube", "blobs", "slab", "rod", "plane", "line", "graded", "lattice"])
def test_tree_matches_oracle_around_the_limits(ctx, orc, kind, n, maxmemb):
    import bit_b200
    x, y, z = shape(kind, n, seed=n % 97 + len(kind))
    try:
        T = orc.Tree(x, y, z, maxmemb)
    except RuntimeError:  # coincident points: the reference would not terminate
        with pytest.raises(bit_b200.BitError) as e:
            ctx.treemake(x, y, z, maxmemb)
        assert e.value.status == 5
        return
    t = ctx.treemake(x, y, z, maxmemb)
    nm, ch, f, mem = t.export()
    assert t.numtree == T.numtree and t.depth == int(T.level.max()) + 1
    np.testing.assert_array_equal(nm, T.nummemb)
    np.testing.assert_array_equal(ch, T.children)
    assert_same_bits(f, T.fields)
    off = np.concatenate([[0], np.cumsum(nm)])
    for i in range(0, t.numtree, max(1, t.numtree // 200)):
        np.testing.assert_array_equal(mem[off[i]:off[i + 1]], T.members(i))
    t.treeempty()


def test_node_arrays_grow(ctx, orc):
    """Every split of 2^-i peels one point off: 500 levels, and ten times the nodes that the
    first estimate holds."""
    n, maxmemb = 1000, 500
    x, z = 2.0 ** -np.arange(n), np.zeros(n)
    T = orc.Tree(x, z, z, maxmemb, cap=4 * n)
    assert T.numtree > 2 * (64 + 16 * (n // maxmemb + 1) + 8)
    t = ctx.treemake(x, z, z, maxmemb)
    assert t.numtree == T.numtree
    nm, ch, f, _ = t.export()
    np.testing.assert_array_equal(nm, T.nummemb)
    np.testing.assert_array_equal(ch, T.children)
    assert_same_bits(f, T.fields)
    t.treeempty()
