"""The performance cases of the treecode: what its users have it do, one pass each.

listed() names the cases, draw(rng) gives more of the same ranges, prepare(case, seed) makes a
program's inputs and handles, run(state) is one pass through the public entry points of
bit_b200, work(case) is what a pass cannot do without, exact(case, seed) the direct sums (and
the dense solve) it approximates, in 64 bits.  Every random number comes from the seed.

Kinds of pass (case["kind"]):

step      a new particle system in device memory: treemake, charges, moments, potentials of
          one or two kernels at every particle, treeempty: the time-stepping and headline use
recharge  the tree is kept, the charges are new: moments and the potential (an iterative
          method's matrix-vector product)
pipeline  one potential from host arrays in one call (treecode_potential), reference mode
force     treemake, treemoments and a field from host arrays, as the reference's drivers do
points    the potential at external points (host arrays) of a tree that is kept
forest    many independent systems of mixed orders and kernels in one tree
solve     a boundary-integral equation on a sphere by GMRES over the treecode
pic       device-resident particle-in-cell steps (tree, moments, field, update per step)
direct    FP64 direct sums at some particles (what errors are measured against)

A mixed-precision result is held to about 1e-7, so those passes keep it in a float32 array.
"""
import functools
import math
import random

import numpy as np
import torch

import bit_b200 as B
from bit_b200 import workloads

DEV = "cuda"


# ------------------------------------------------------------------------------- the cases
def _step(name, n, dist, maxmemb, nterms, acc, kernels, prec, kappa=1.0, delta=0.005):
    return dict(name=name, kind="step", n=n, dist=dist, maxmemb=maxmemb, nterms=nterms, acc=acc,
                kernels=kernels, prec=prec, kappa=kappa, delta=delta)


def listed():
    return [
        # the smallest call: a caller of the reference's serial interface, a few thousand
        # particles in host memory, once per call; launches and latency are all of it
        dict(name="pipeline_2k_fp64", kind="pipeline", n=2000, dist="cube", maxmemb=100, nterms=5,
             acc=0.5, kernel="coulomb", prec="fp64", kappa=0.0, delta=0.01),
        # a small system of an odd size, new at every time step
        _step("step_10k_screened_mixed", 10007, "cube", 200, 7, 0.6, "screened", "mixed", kappa=2.0),
        # the headline evaluation in the reference's arithmetic: 2M clustered particles, p = 8,
        # theta = 0.7, leaves of 1000, screened and Coulomb potentials
        _step("step_2M_both_fp64", 2000000, "blobs", 1000, 9, 0.7, "both", "fp64"),
        # the same in mixed precision
        _step("step_2M_both_mixed", 2000000, "blobs", 1000, 9, 0.7, "both", "mixed"),
        # mixed precision where the truncation error is about 1e-6 (theta = 0.15): the
        # accuracy-matched setting, long interaction lists
        _step("step_100k_tight_mixed", 100000, "blobs", 500, 9, 0.15, "both", "mixed"),
        # new charges on a tree that is kept, the regularised screened kernel, a middling size
        dict(name="recharge_200k_reg_fp64", kind="recharge", n=200003, dist="blobs", maxmemb=500,
             nterms=7, acc=0.6, kernel="reg", prec="fp64", kappa=0.7, delta=1e-4),
        # treeforce at every particle, as the reference's free-space driver calls it
        dict(name="force_50k_fp64", kind="force", n=50000, dist="blobs", maxmemb=300, nterms=7,
             acc=0.6, field="coulomb", prec="fp64", kappa=0.0, delta=1e-4),
        # probes of the potential away from the particles (a plot, a surface)
        dict(name="points_30k_screened_fp64", kind="points", n=200000, m=30011, dist="blobs",
             maxmemb=1000, nterms=9, acc=0.7, kernel="screened", prec="fp64", kappa=1.0, delta=0.0),
        # a batch of independent systems of 1e3..1e5 particles, p in {4, 6, 8}, both kernels
        dict(name="forest_48_mixed", kind="forest", systems=48, nmin=1000, nmax=100000,
             maxmemb=512, acc=0.6, prec="mixed"),
        # a boundary-integral solve on an icosphere of 20,480 faces, p = 6, theta = 0.5
        dict(name="solve_20k_fp64", kind="solve", level=5, maxmemb=500, nterms=7, acc=0.5,
             kappa=1.0, tol=1e-8, prec="fp64"),
        # three steps of a particle-in-cell loop that stays on the device
        dict(name="pic_20k_fp64", kind="pic", n=20000, dist="cube", steps=3, maxmemb=200,
             nterms=6, acc=0.6, prec="fp64", delta=1e-3),
        # the direct sum at 10,000 of 200,000 particles: an error check
        dict(name="direct_200k_fp64", kind="direct", n=200000, m=10000, dist="blobs",
             kernel="screened", kappa=1.0, delta=0.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges, no costlier than the largest listed one."""
    kind = rng.choice(["step", "step", "step", "recharge", "pipeline", "force", "points",
                       "forest", "solve", "pic", "direct"])
    dist = rng.choice(["blobs", "cube"])
    prec = rng.choice(["fp64", "mixed"])
    nterms = rng.randint(3, 10)
    kernel = rng.choice(["coulomb", "screened", "reg"])
    kappa = round(rng.uniform(0.3, 4.0), 3)
    delta = rng.choice([0.0, 1e-4, 0.005, 0.01])
    acc = round(rng.uniform(0.4, 0.75), 3)
    if kind == "step":
        n = _logint(rng, 2000, 800000)
        if n <= 60000 and rng.random() < 0.3:
            acc = round(rng.uniform(0.1, 0.3), 3)
        return dict(kind=kind, n=n, dist=dist, maxmemb=_logint(rng, max(40, min(n // 1000, 200)), 1000),
                    nterms=nterms, acc=acc, kernels=rng.choice(["both", "screened", "coulomb", "reg"]),
                    prec=prec, kappa=kappa, delta=delta)
    if kind in ("recharge", "pipeline"):
        n = _logint(rng, 2000, 300000) if kind == "recharge" else _logint(rng, 1000, 100000)
        return dict(kind=kind, n=n, dist=dist, maxmemb=_logint(rng, 50, 800), nterms=nterms, acc=acc,
                    kernel=kernel, prec=prec, kappa=kappa, delta=delta)
    if kind == "force":
        field = rng.choice(["coulomb", "coulomb", "curl"])
        return dict(kind=kind, n=_logint(rng, 2000, 150000), dist=dist, maxmemb=_logint(rng, 50, 600),
                    nterms=rng.randint(3, 9), acc=acc, field=field,
                    prec="fp64" if field == "curl" else prec, kappa=kappa,
                    delta=rng.choice([1e-4, 0.005, 0.01]))
    if kind == "points":
        return dict(kind=kind, n=_logint(rng, 5000, 300000), m=_logint(rng, 50, 100000), dist=dist,
                    maxmemb=_logint(rng, 100, 1000), nterms=nterms, acc=acc, kernel=kernel,
                    prec=prec, kappa=kappa, delta=delta)
    if kind == "forest":
        return dict(kind=kind, systems=_logint(rng, 3, 100), nmin=500, nmax=_logint(rng, 5000, 100000),
                    maxmemb=_logint(rng, 100, 512), acc=acc, prec=prec)
    if kind == "solve":
        return dict(kind=kind, level=rng.randint(3, 5), maxmemb=_logint(rng, 100, 600),
                    nterms=rng.randint(5, 9), acc=round(rng.uniform(0.15, 0.5), 3), kappa=kappa,
                    tol=1e-8, prec="fp64")
    if kind == "pic":
        return dict(kind=kind, n=_logint(rng, 2000, 60000), dist=dist, steps=rng.randint(1, 4),
                    maxmemb=_logint(rng, 50, 400), nterms=rng.randint(3, 8), acc=acc, prec="fp64",
                    delta=rng.choice([1e-3, 0.01]))
    return dict(kind="direct", n=_logint(rng, 2000, 400000), m=_logint(rng, 100, 10000), dist=dist,
                kernel=kernel, kappa=kappa, delta=delta)


# --------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _context(group):
    """A program has one context for all its calls (leaf packing is set on it)."""
    ctx = B.Context()
    ctx.set_group_size(group)
    return ctx


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _particles(dist, n, seed):
    """x, y, z, q on the device: uniform in [-1, 1]^3, or 80% in eight Gaussian blobs of
    sigma 0.1 (workloads.clustered_blobs); charges uniform in [-1, 1]."""
    g = _generator(seed)
    u = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    if dist == "cube":
        p = u(3, n)
    else:
        nb = int(round(0.8 * n))
        centres = u(3, 8)
        which = torch.randint(0, 8, (nb,), generator=g, device=DEV)
        blobs = centres[:, which] + 0.1 * torch.randn(3, nb, generator=g, device=DEV,
                                                      dtype=torch.float64)
        p = torch.cat([blobs, u(3, n - nb)], dim=1)
        p = p[:, torch.randperm(n, generator=g, device=DEV)].contiguous()
    return p, u(n)


def _charges(n, seed):
    g = _generator(seed + 7919)
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1


def _prec(case):
    return B.MIXED if case["prec"] == "mixed" else B.FP64


def _params(kernel, case, mode=B.CONSISTENT):
    if kernel == "coulomb":
        return B.params(B.COULOMB, mode, _prec(case), del_=case["delta"], acc=case["acc"])
    if kernel == "screened":
        return B.params(B.SCREENED, mode, _prec(case), kappa=case["kappa"], acc=case["acc"])
    return B.params(B.SCREENED_REG, mode, _prec(case), kappa=case["kappa"], del_=case["delta"],
                    acc=case["acc"])


def _kernels(case):
    return ["screened", "coulomb"] if case["kernels"] == "both" else [case["kernels"]]


def _forest_systems(case, seed):
    """Sizes log-uniform, kernels alternating, p in {4, 6, 8}: workloads.batched_systems."""
    r = random.Random(seed)
    out = []
    # the sizes belong to the case, so that passes on several seeds cost the same
    sizes = random.Random(case["systems"] * 1000003 + case["nmax"])
    for i in range(case["systems"]):
        n = _logint(sizes, case["nmin"], case["nmax"])
        nterms = sizes.choice([4, 6, 8]) + 1
        coul = i % 2 == 0
        out.append((n, "coulomb" if coul else "screened", 0.0 if coul else r.uniform(0.5, 4.0),
                    1e-4 if coul else 0.0, nterms))
    return out


def _host(*tensors):
    return [t.cpu().numpy() for t in tensors]


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, ctx=_context(1024 if kind == "forest" else 0))
    if kind == "forest":
        sysm = _forest_systems(case, seed)
        st["sizes"] = [s[0] for s in sysm]
        n = sum(st["sizes"])
        g = _generator(seed)
        st["p"] = torch.rand(3, n, generator=g, device=DEV, dtype=torch.float64)
        st["q"] = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
        st["nterms"] = [s[4] for s in sysm]
        st["prm"] = [_params(k, dict(case, kappa=kap, delta=d)) for _, k, kap, d, _ in sysm]
        _outputs(st, 1, n)
    elif kind == "solve":
        cen, area, edge = workloads.icosphere(case["level"])
        st["f"] = workloads.sh_rhs(cen, seed=seed)
        st["area"] = area
        st["edge"] = edge
        st["prm"] = B.params(B.SCREENED_REG, B.CONSISTENT, _prec(case), kappa=case["kappa"],
                             del_=edge * edge, acc=case["acc"])
        st["tree"] = st["ctx"].treemake(cen[:, 0], cen[:, 1], cen[:, 2], case["maxmemb"])
    else:
        n = case["n"]
        p, q = _particles(case["dist"], n, seed)
        if kind == "step":
            st.update(p=p, q=q, prm=[_params(k, case) for k in _kernels(case)])
            _outputs(st, len(st["prm"]), n)
        elif kind == "recharge":
            st["tree"] = st["ctx"].treemake(*_host(*p), case["maxmemb"])
            st.update(q=_charges(n, seed), prm=_params(case["kernel"], case))
            _outputs(st, 1, n)
        elif kind == "pipeline":
            st["host"] = _host(*p, q)
            st["prm"] = _params(case["kernel"], case, B.REFERENCE if case["kernel"] == "coulomb"
                                else B.CONSISTENT)
        elif kind == "force":
            st["host"] = _host(*p, q)
        elif kind == "points":
            st["tree"] = st["ctx"].treemake(*_host(*p), case["maxmemb"])
            st["tree"].treemoments(_host(q)[0], case["nterms"])
            st["prm"] = _params(case["kernel"], case)
            st["points"] = _points(case, seed)
        elif kind == "pic":
            st.update(p0=p, q=q, opts=B.PicOpts(case["steps"], case["nterms"], case["maxmemb"], 1e-4,
                                                case["delta"], case["acc"], 1.0, 1.0, _prec(case)))
            st.update(p=p.clone(), v=torch.zeros_like(p), f=torch.zeros_like(p))
            st["stream"] = torch.cuda.ExternalStream(st["ctx"].stream)
        else:
            st["host"] = _host(*p, q)
            st["prm"] = B.params({"coulomb": B.COULOMB, "screened": B.SCREENED,
                                  "reg": B.SCREENED_REG}[case["kernel"]], B.CONSISTENT, B.FP64,
                                 del_=case["delta"], kappa=case["kappa"])
            st["targets"] = _targets(case, seed)
    return st


def _points(case, seed):
    return np.random.default_rng(seed + 31).uniform(-1.2, 1.2, (case["m"], 3))


def _targets(case, seed):
    return workloads.sample_targets(case["n"], case["m"], seed=seed + 17)


def _outputs(st, count, n):
    st["stream"] = torch.cuda.ExternalStream(st["ctx"].stream)
    st["out"] = [torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(count)]
    if st["case"]["prec"] == "mixed":
        st["out32"] = [torch.zeros(n, dtype=torch.float32, device=DEV) for _ in range(count)]


def _result(st):
    """The potentials; a mixed result is held in float32."""
    if "out32" not in st:
        return st["out"]
    with torch.cuda.stream(st["stream"]):
        for a, b in zip(st["out32"], st["out"]):
            a.copy_(b)
    return st["out32"]


# ------------------------------------------------------------------------------- one pass
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "step":
        p = st["p"]
        t = ctx.treemake_device(case["n"], p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(),
                                case["maxmemb"])
        t.set_charges_device(st["q"].data_ptr())
        t.moments(case["nterms"])
        for prm, out in zip(st["prm"], st["out"]):
            t.evaluate_device(prm, out.data_ptr())
        r = _result(st)
        t.treeempty()
        return r
    if kind == "recharge":
        t = st["tree"]
        t.set_charges_device(st["q"].data_ptr())
        t.moments(case["nterms"])
        t.evaluate_device(st["prm"], st["out"][0].data_ptr())
        return _result(st)
    if kind == "pipeline":
        return _as_held(case, ctx.treecode_potential(*st["host"], case["nterms"], case["maxmemb"],
                                                     st["prm"]))
    if kind == "force":
        x, y, z, q = st["host"]
        t = ctx.treemake(x, y, z, case["maxmemb"])
        t.treemoments(q, case["nterms"])
        if case["field"] == "curl":
            f = t.field(B.FIELD_SCREENED, acc=case["acc"], kappa=case["kappa"])
        else:
            f = t.treeforce(case["acc"], case["delta"], _prec(case))
        t.treeempty()
        return [_as_held(case, a) for a in f]
    if kind == "points":
        return _as_held(case, st["tree"].evaluate(st["prm"], points=st["points"]))
    if kind == "forest":
        p = st["p"]
        t = ctx.forest_device(st["sizes"], case["maxmemb"], p[0].data_ptr(), p[1].data_ptr(),
                              p[2].data_ptr())
        t.set_charges_device(st["q"].data_ptr())
        t.moments(st["nterms"])
        t.evaluate_device(st["prm"], st["out"][0].data_ptr())
        r = _result(st)
        t.treeempty()
        return r
    if kind == "solve":
        return st["tree"].bie_solve(st["prm"], case["nterms"], 0.5, st["area"], st["f"],
                                    tol=case["tol"], precision=_prec(case))[0]
    if kind == "pic":
        p, v, f = st["p"], st["v"], st["f"]
        with torch.cuda.stream(st["stream"]):  # every pass starts from the same state
            p.copy_(st["p0"])
            v.zero_()
        ptr = lambda a: tuple(r.data_ptr() for r in a)
        ctx.pic_steps_device(case["n"], ptr(p) + ptr(v), st["q"].data_ptr(), st["opts"], ptr(f))
        return dict(position=p, velocity=v, force=f)
    return ctx.direct(*st["host"], st["prm"], st["targets"])


def _as_held(case, a):
    return a.astype(np.float32) if case["prec"] == "mixed" else a


# ----------------------------------------------------------------------------- what it takes
# Flops of one near pair (a distance, a reciprocal square root, for the screened kernels an
# exponential, a product) and of one far pair per expansion coefficient; a tree's near and
# far pairs per target, as counts over these distributions run: about eight half-full leaves
# of sources at theta = 0.7, growing as theta falls, and 24 clusters per octave of size.
NEAR = dict(coulomb=11, screened=14, reg=15, force=18, curl=20)


def _pairs(n, maxmemb, acc):
    leaf = 0.55 * min(maxmemb, n)  # leaves come out about half full
    near = min(n, leaf * 8.0 * (0.7 / max(acc, 1e-3)) ** 1.2)
    levels = max(0.0, math.log2(max(1.0, n / maxmemb)) / 3)
    far = min(n / leaf, 24.0 * levels)
    return near, far


def _tree_flops(n, maxmemb, acc, nterms, near_flops, evals=1):
    near, far = _pairs(n, maxmemb, acc)
    coefs = nterms * (nterms + 1) * (nterms + 2) // 6
    levels = 1 + max(0.0, math.log2(max(1.0, n / maxmemb)) / 2)
    return n * (evals * (near * near_flops + far * 2 * coefs) + 2 * coefs * levels)


def work(case):
    kind = case["kind"]
    if kind == "step":
        ks = _kernels(case)
        fl = sum(_tree_flops(case["n"], case["maxmemb"], case["acc"], case["nterms"], NEAR[k]) for k in ks)
        return dict(bytes=case["n"] * (32 + 8 * len(ks)), flops=fl)
    if kind in ("recharge", "pipeline"):
        return dict(bytes=case["n"] * 40, flops=_tree_flops(
            case["n"], case["maxmemb"], case["acc"], case["nterms"], NEAR[case["kernel"]]))
    if kind == "force":
        return dict(bytes=case["n"] * 56, flops=_tree_flops(
            case["n"], case["maxmemb"], case["acc"], case["nterms"] + 1,
            NEAR["curl" if case["field"] == "curl" else "force"], 3))
    if kind == "points":
        near, far = _pairs(case["n"], case["maxmemb"], case["acc"])
        coefs = case["nterms"] * (case["nterms"] + 1) * (case["nterms"] + 2) // 6
        return dict(bytes=case["n"] * 32 + case["m"] * 32,
                    flops=case["m"] * (near * NEAR[case["kernel"]] + far * 2 * coefs))
    if kind == "forest":
        sysm = _forest_systems(case, 0)
        return dict(bytes=40 * sum(s[0] for s in sysm),
                    flops=sum(_tree_flops(s[0], case["maxmemb"], case["acc"], s[4], NEAR[s[1]])
                              for s in sysm))
    if kind == "solve":
        n = 20 * 4 ** case["level"]
        return dict(bytes=48 * n, flops=10 * _tree_flops(n, case["maxmemb"], case["acc"],
                                                         case["nterms"], NEAR["reg"]))
    if kind == "pic":
        return dict(bytes=case["n"] * 104 * case["steps"], flops=case["steps"] * _tree_flops(
            case["n"], case["maxmemb"], case["acc"], case["nterms"] + 1, NEAR["force"], 3))
    return dict(bytes=32 * case["n"] + 12 * case["m"],
                flops=float(case["n"]) * case["m"] * NEAR[case["kernel"]])


# ------------------------------------------------------------------------- direct sums, FP64
EPS = 1e-14  # a regularised pair with r^2 + delta below this adds nothing


def _direct(kernel, src, q, tgt, self_index, kappa, delta):
    """sum_j q_j G(r_ij) over j != i; src (3, n), tgt (3, m); self_index: the particle each
    target is, or None.  Screened potentials carry the reference's minus sign."""
    n, m = src.shape[1], tgt.shape[1]
    out = torch.empty(m, dtype=torch.float64, device=src.device)
    rows = max(1, int(1.6e8 // n))
    for i in range(0, m, rows):
        t = tgt[:, i:i + rows]
        r2 = (t[0, :, None] - src[0]).square_()
        for a in (1, 2):
            r2 += (t[a, :, None] - src[a]).square_()
        if kernel != "screened":
            r2 += delta
        skip = r2 <= EPS if kernel != "screened" else None
        if self_index is not None:
            k = self_index[i:i + rows]
            r2[torch.arange(len(k), device=src.device), k] = math.inf
        if skip is not None:
            r2[skip] = math.inf
        if kernel == "coulomb":
            g = r2.rsqrt_()
        else:
            r = r2.sqrt_()
            g = torch.exp(-kappa * r) / r
            g[torch.isinf(r)] = 0.0
        out[i:i + rows] = g @ q
    return -out if kernel == "screened" else out


def _direct_field(src, q, delta):
    """sum_j q_j (x_i - x_j) / (r^2 + delta)^(3/2), (3, n)."""
    n = src.shape[1]
    out = torch.empty_like(src)
    rows = max(1, int(8e7 // n))
    for i in range(0, n, rows):
        d = src[:, i:i + rows, None] - src[:, None, :]
        w = (d.square().sum(0) + delta).pow_(-1.5) * q
        out[:, i:i + rows] = torch.einsum("aij,ij->ai", d, w)
    return out


def _direct_curl(src, q, kappa):
    """The screened 2-D field: sum_j q_j e^{-kappa r} / r^2 (kappa + 1/r) (-dy, dx, 0)."""
    n = src.shape[1]
    out = torch.zeros_like(src)
    rows = max(1, int(8e7 // n))
    for i in range(0, n, rows):
        d = src[:, i:i + rows, None] - src[:, None, :]
        r = d.square().sum(0).sqrt_()
        r[torch.arange(r.shape[0], device=r.device), torch.arange(i, i + r.shape[0], device=r.device)] = math.inf
        w = torch.exp(-kappa * r) / r.square() * (kappa + 1 / r)
        w[torch.isinf(r)] = 0.0
        w *= q
        out[0, i:i + rows] = -(d[1] * w).sum(1)
        out[1, i:i + rows] = (d[0] * w).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        n = 20 * 4 ** case["level"]
        cen, area, edge = workloads.icosphere(case["level"])
        p = torch.tensor(cen.T.copy(), device=DEV)
        r = (torch.cdist(p.T, p.T, compute_mode="donot_use_mm_for_euclid_dist").square()
             + edge * edge).sqrt_()
        a = torch.exp(-case["kappa"] * r) / r * torch.tensor(area, device=DEV)
        i = torch.arange(n, device=DEV)
        a[i, i] = 0.5
        f = torch.tensor(workloads.sh_rhs(cen, seed=seed), device=DEV)
        return torch.linalg.solve(a, f).cpu().numpy()
    if kind == "forest":
        sysm = _forest_systems(case, seed)
        if sum(float(s[0]) ** 2 for s in sysm) > 1.5e11:
            return None
        n = sum(s[0] for s in sysm)
        g = _generator(seed)
        p = torch.rand(3, n, generator=g, device=DEV, dtype=torch.float64)
        q = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
        out, o = [], 0
        for m, k, kappa, delta, _ in sysm:
            s = p[:, o:o + m]
            out.append(_direct(k, s, q[o:o + m], s, torch.arange(m, device=DEV), kappa, delta))
            o += m
        return [torch.cat(out)]
    n = case["n"]
    m = case.get("m", n)
    if float(n) * m > 1.2e11:
        return None
    p, q = _particles(case["dist"], n, seed)
    if kind == "step":
        i = torch.arange(n, device=DEV)
        return [_direct(k, p, q, p, i, case["kappa"], case["delta"]) for k in _kernels(case)]
    if kind == "recharge":
        return [_direct(case["kernel"], p, _charges(n, seed), p, torch.arange(n, device=DEV),
                        case["kappa"], case["delta"])]
    if kind == "pipeline":
        if case["kernel"] == "coulomb" and case["delta"]:
            return None  # reference mode: delta in the far field only, no one direct sum
        return _direct(case["kernel"], p, q, p, torch.arange(n, device=DEV), case["kappa"],
                       case["delta"]).cpu().numpy()
    if kind == "force":
        f = (_direct_curl(p, q, case["kappa"]) if case["field"] == "curl"
             else _direct_field(p, q, case["delta"]))
        return _host(*f)
    if kind == "points":
        t = torch.tensor(_points(case, seed).T.copy(), device=DEV)
        return _direct(case["kernel"], p, q, t, None, case["kappa"], case["delta"]).cpu().numpy()
    if kind == "pic":
        v = torch.zeros_like(p)
        for _ in range(case["steps"]):
            f = _direct_field(p, q, case["delta"]) * q
            v = v + 1e-4 * f
            p = p + 1e-4 * v
        return dict(position=p, velocity=v, force=f)
    tg = torch.tensor(_targets(case, seed).astype(np.int64), device=DEV)
    return _direct(case["kernel"], p, q, p[:, tg], tg, case["kappa"], case["delta"]).cpu().numpy()
