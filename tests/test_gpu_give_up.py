"""After a device-side wait gave up, the context's trees evaluate as before: the diagnostic's give-up
leaves every group with a part counted as done, as a near-field work queue whose CTAs all gave up
would, and the host's report of the error sets the counts back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queue", [1, 0])
def test_trees_evaluate_as_before_after_a_wait_gave_up(ctx, queue):
    import bit_b200 as B
    from bit_b200 import workloads
    sizes = [9000, 14000, 2500]
    parts = [workloads.clustered_blobs(n, seed=n) for n in sizes]
    x, y, z, q = (np.concatenate([p[i] for p in parts]) for i in range(4))
    f = ctx.forest(x, y, z, sizes, 700)  # groups of several parts
    f.set_charges(q)
    f.moments(4)
    t = ctx.treemake(*parts[1][:3], 700)
    t.treemoments(parts[1][3], 4)
    ctx.set_work_queue(queue)
    for prec in (B.FP64, B.MIXED):
        prm = [B.params((B.SCREENED, B.COULOMB)[i % 2], B.CONSISTENT, prec, kappa=1.0, acc=0.3) for i in range(3)]
        want = f.evaluate(prm), t.evaluate(prm[0]), np.stack(t.treeforce(0.3, 1e-4, prec))
        t.evaluate(prm[0])
        assert ctx.wait_check(1000) == 2  # BIT_ERR_CUDA
        got = f.evaluate(prm), t.evaluate(prm[0]), np.stack(t.treeforce(0.3, 1e-4, prec))
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
    ctx.set_work_queue(1)
    f.treeempty()
    t.treeempty()
