"""A result's bits do not depend on the memory budget.  Contexts of less and less memory, from what
the evaluation takes without a limit downwards: every call either fails with the budget's own
status or gives the result of the unlimited context, bit for bit.  (The near field cuts heavy groups
into parts that meet in scratch; without room for it a group takes its parts in turn.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
BUDGET = 9  # BIT_ERR_BUDGET


def shrinking(peak, step, run):
    """run(budget) for budgets from `peak` down; how many gave a result."""
    import bit_b200 as B
    done = 0
    for k in range(60):
        budget = peak - k * step
        if budget <= 0:
            break
        ctx = B.Context(hbm_budget=budget)
        try:
            run(ctx)
            done += 1
        except B.BitError as e:
            assert e.status == BUDGET, e
        ctx.close()
    return done


def evaluate(ctx, calls, x, y, z, q, maxmemb, nterms):
    t = ctx.treemake(x, y, z, maxmemb)
    t.treemoments(q, nterms)
    out = [f(t) for f in calls]
    t.treeempty()
    return out


def calls(B):
    p = lambda *a, **k: B.params(*a, **k)
    return {
        "screened": lambda t: t.evaluate(p(B.SCREENED, B.CONSISTENT, B.FP64, kappa=1.0, acc=0.3)),
        "coulomb reference": lambda t: t.evaluate(p(B.COULOMB, B.REFERENCE, B.FP64, del_=1e-4, acc=0.3)),
        "mixed": lambda t: t.evaluate(p(B.SCREENED_REG, B.CONSISTENT, B.MIXED, kappa=1.0, del_=1e-6, acc=0.3)),
        "force": lambda t: np.stack(t.treeforce(0.3, 1e-4)),
        "force mixed": lambda t: np.stack(t.treeforce(0.3, 1e-4, B.MIXED)),
        "curl": lambda t: np.stack(t.field(B.FIELD_SCREENED, acc=0.3, kappa=1.0)),
        "kernel order": lambda t: np.stack(t.field(B.FIELD_COULOMB, acc=0.3, del_=1e-2, kernel_order=2)),
    }


@pytest.mark.parametrize("name", ["screened", "coulomb reference", "mixed", "force", "force mixed", "curl",
                                  "kernel order"])
def test_particles_within_less_and_less_memory(name):
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(60000, seed=1)
    args = (x, y, z, q, 700, 5)
    f = calls(B)[name]
    free = B.Context()
    want, = evaluate(free, [f], *args)
    peak = free.memory()[1]
    free.close()

    def run(ctx):
        np.testing.assert_array_equal(evaluate(ctx, [f], *args)[0], want)
    assert shrinking(peak + 2 * MB, MB // 2, run) > 3


@pytest.mark.parametrize("queue", [1, 0])
def test_forest_within_less_and_less_memory(queue):
    import bit_b200 as B
    from bit_b200 import workloads
    sizes = [9000, 14000, 2500, 20000]
    parts = [workloads.clustered_blobs(n, seed=n) for n in sizes]
    x, y, z, q = (np.concatenate([p[i] for p in parts]) for i in range(4))
    prm = [B.params((B.SCREENED, B.COULOMB)[i % 2], B.CONSISTENT, (B.FP64, B.FP64)[i % 2], kappa=1.0, del_=1e-4 * (i % 2),
                    acc=0.3) for i in range(4)]

    def run_on(ctx):
        ctx.set_work_queue(queue)
        f = ctx.forest(x, y, z, sizes, 700)
        f.set_charges(q)
        f.moments([5, 3, 4, 5])
        got = f.evaluate(prm)
        f.treeempty()
        return got
    free = B.Context()
    want = run_on(free)
    peak = free.memory()[1]
    free.close()

    def run(ctx):
        np.testing.assert_array_equal(run_on(ctx), want)
    assert shrinking(peak + 2 * MB, MB // 2, run) > 3


@pytest.mark.parametrize("m", [1, 70, 3000])
def test_direct_sums_within_less_and_less_memory(m):
    """The chunks of sources go a few at a time, to one, where the budget has no room for all sums."""
    import bit_b200 as B
    from bit_b200 import workloads
    x, y, z, q = workloads.clustered_blobs(60000, seed=2)
    tg = np.random.default_rng(m).choice(60000, m, replace=False).astype(np.int32)
    prm = [B.params(B.COULOMB, B.CONSISTENT, B.FP64, del_=1e-4), B.params(B.SCREENED, B.CONSISTENT, B.FP64, kappa=1.0)]
    free = B.Context()
    want = [free.direct(x, y, z, q, p, tg) for p in prm]
    peak = free.memory()[1]
    free.close()
    inputs = 4 * (60000 * 8 + 511) // 512 * 512 + (1 << 14)  # the least that a sum takes

    def run(ctx):
        for p, w in zip(prm, want):
            np.testing.assert_array_equal(ctx.direct(x, y, z, q, p, tg), w)
    done = shrinking(peak + (1 << 14), 1 << 14, run)
    assert done >= min(60, (peak - inputs - 3 * 8 * m) // (1 << 14) - 2)
