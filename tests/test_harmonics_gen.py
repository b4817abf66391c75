"""The generated solid-harmonic far field (bit_b200/csrc/gen_harmonics.py), run in FP64 on
the CPU: coefficients formed as k_far_coefs forms them, evaluated by the generated code,
equal the literal form of the reference's Taylor recurrence for every order and kernel.

Tolerance: both sides sum a few hundred products of size at most eta^n (eta = 0.87, the
largest cluster-radius ratio here) times sum |q| e^(-kappa R) / R, so each side's rounding
is below about 500 * 1.1e-16 * sum_n eta^n = 4e-13 of that scale."""
import math
import re

import numpy as np
import pytest

from test_farfield_gen import compile_lines, gen as gen_taylor

TOL = 5e-13
ARGS = ["dx", "dy", "dz", "r2", "add", "kappa", "H", "M"]


def gen():
    import importlib.util
    import os
    from conftest import ROOT
    spec = importlib.util.spec_from_file_location(
        "gen_harmonics", os.path.join(ROOT, "bit_b200", "csrc", "gen_harmonics.py"))
    g = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(g)
    return g


def coefficients(g, nt, reg, moments, kappa, delta, H):
    """k_far_coefs: shell-order moments to the coefficients of one kernel."""
    hl = g.harmonic_list(nt)
    pos = {h: i for i, h in enumerate(hl)}
    A = [sum(f * moments[p] for p, f in row) / H ** (h[0] + 2 * h[3])
         for h, row in zip(hl, g.harmonic_table(nt))]
    kmax = (nt - 1) // 2
    e = np.zeros((kmax + 2, 2 * kmax + 4))
    e[0, 0] = 1.0
    for k in range(kmax):
        for s in range(2 * k + 1):
            e[k + 1, s] += (kappa * H) ** 2 * e[k, s]
            e[k + 1, s + 1] += 2 * s * e[k, s]
            e[k + 1, s + 2] -= delta / H ** 2 * e[k, s]
    out = [g.dfact(2 * (l + s) - 1) * sum(e[k, s] * A[pos[(l, m, p, k)]]
                                          for k in range((nt - 1 - l) // 2 + 1))
           for l, m, p, s in g.coefficient_list(nt, reg)]
    return np.array(out + [0.0] * (-len(out) % 4))


@pytest.mark.parametrize("nt", range(1, 11))
def test_harmonic_form_equals_the_taylor_recurrence(nt):
    g, t = gen(), gen_taylor()
    coulomb = compile_lines(t.gen_coulomb(nt), ["dx", "dy", "dz", "rs", "M"])
    screened = compile_lines(t.gen_screened(nt), ["dx", "dy", "dz", "dist2", "kappa", "M"])
    shells = list(t.shells(nt - 1))
    rng = np.random.default_rng(nt)
    for name, reg, scr in g.VARIANTS:
        f = compile_lines(g.gen_eval(nt, reg, scr), ARGS)
        for trial in range(12):
            radius = 10.0 ** rng.uniform(-5, 1)
            y = rng.uniform(-1, 1, (30, 3)) * radius / math.sqrt(3.0)
            q = rng.uniform(-1, 1, 30)
            M = np.array([np.sum(q * y[:, 0] ** v[0] * y[:, 1] ** v[1] * y[:, 2] ** v[2])
                          for v in shells])
            d = rng.standard_normal(3)
            d *= radius / math.sqrt(rng.uniform(0.05, 0.75)) / np.linalg.norm(d)
            # delta far below, near and far above the squared distance
            delta = radius ** 2 * 10.0 ** rng.uniform(-6, 3) if reg else 0.0
            kappa = rng.uniform(0.0, 4.0) / radius if scr else 0.0
            R2 = float(d @ d) + delta
            H = 2.0 ** (math.floor(math.log2(max(radius, math.sqrt(delta)))) + 1)
            pad = np.concatenate([M, np.zeros(-len(M) % 4)])
            want = screened(*d, R2, kappa, pad) if scr else coulomb(*d, R2, pad)
            got = f(*d, float(d @ d), delta, kappa, H, coefficients(g, nt, reg, M, kappa, delta, H))
            scale = np.abs(q).sum() * math.exp(-kappa * math.sqrt(R2)) / math.sqrt(R2)
            # the reference's screened recurrence has terms of size (kappa radius)^n
            scale *= 1.0 + (kappa * radius) ** (nt - 1) / math.factorial(nt - 1)
            assert abs(got - want) <= TOL * scale, (name, trial, got, want)


def test_harmonic_moments_keep_every_cartesian_moment():
    """The table is a change of basis: as many harmonic moments as Cartesian ones, of full
    rank for every degree, and each a combination of its own degree's moments only."""
    g = gen()
    nt = g.NTMAX
    rows, hl = g.harmonic_table(nt), g.harmonic_list(nt)
    n = nt * (nt + 1) * (nt + 2) // 6
    A = np.zeros((n, n))
    for i, row in enumerate(rows):
        deg = hl[i][0] + 2 * hl[i][3]
        for p, f in row:
            assert deg * (deg + 1) * (deg + 2) // 6 <= p < (deg + 1) * (deg + 2) * (deg + 3) // 6
            A[i, p] = f
    assert np.linalg.matrix_rank(A / np.abs(A).max(axis=1, keepdims=True)) == n


@pytest.mark.parametrize("nt", range(1, 11))
def test_gradients_equal_the_taylor_recurrences(nt):
    """The generated gradients against the literal field sums: Coulomb with and without delta,
    and the screened curl (d phi/dy, -d phi/dx).  A field term is at most (n + 1) / R times its
    potential's, so the scale is that of the potential times nterms / R."""
    g, t = gen(), gen_taylor()
    args = ["dx", "dy", "dz", "rs", "M", "fx", "fy", "fz"]

    def fields(lines, names):
        out = lines + ["  return fx, fy, fz;"]
        return compile_lines([re.sub(r"f([xyz]) \+= (\w+)", r"f\1 = \2", ln) for ln in out], names)

    coulomb = fields(t.gen_force(nt), args)
    curl = fields(t.gen_screened_curl(nt), ["dx", "dy", "dz", "dist2", "kappa", "M", "fx", "fy", "fz"])
    shells = list(t.shells(nt - 1))
    rng = np.random.default_rng(nt)
    for name, reg, scr in g.GRADIENTS:
        f = fields(g.gen_grad(nt, reg, scr), ARGS)
        for trial in range(12):
            radius = 10.0 ** rng.uniform(-5, 1)
            y = rng.uniform(-1, 1, (30, 3)) * radius / math.sqrt(3.0)
            q = rng.uniform(-1, 1, 30)
            M = np.array([np.sum(q * y[:, 0] ** v[0] * y[:, 1] ** v[1] * y[:, 2] ** v[2])
                          for v in shells])
            d = rng.standard_normal(3)
            d *= radius / math.sqrt(rng.uniform(0.05, 0.75)) / np.linalg.norm(d)
            delta = radius ** 2 * 10.0 ** rng.uniform(-6, 3) if reg else 0.0
            kappa = rng.uniform(0.0, 4.0) / radius if scr else 0.0
            r2 = float(d @ d)
            R2 = r2 + delta
            H = 2.0 ** (math.floor(math.log2(max(radius, math.sqrt(delta)))) + 1)
            pad = np.concatenate([M, np.zeros(-len(M) % 4)])
            got = f(*d, r2, delta, kappa, H, coefficients(g, nt, reg, M, kappa, delta, H))
            if scr:
                want = curl(*d, R2, kappa, pad, 0.0, 0.0, 0.0)
                got = (-got[1], got[0], 0.0)
            else:
                want = coulomb(*d, R2, pad, 0.0, 0.0, 0.0)
            scale = np.abs(q).sum() * math.exp(-kappa * math.sqrt(R2)) / R2 * (nt + kappa * math.sqrt(R2))
            scale *= 1.0 + (kappa * radius) ** (nt - 1) / math.factorial(nt - 1)
            assert np.max(np.abs(np.subtract(got, want))) <= TOL * scale, (name, trial, got, want)
