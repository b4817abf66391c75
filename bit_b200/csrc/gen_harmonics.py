"""Generate harmonics_gen.cuh: the far-field potentials in solid harmonics, nterms = 1..10.

The reference evaluates, per (target, cluster), the Taylor polynomial of the kernel about
the cluster centre to degree nterms - 1 (treetaylorpotential, src/tree3d.cpp:4468-4640;
shielded_treetaylorpot, :3004-3227).  For a kernel f(|d|) that depends on the distance only,
its degree-n term is (Hobson's theorem on a harmonic polynomial of the gradient)

  (-y.grad)^n f / n! = sum over l + 2k = n of  (-1)^l (2l + 1) / (2^k k! (2l + 2k + 1)!!)
                       |y|^2k  sum_m w_lm B_lm(y) B_lm(d)  D^l lap^k f,   D = (1/r) d/dr,

with B_lm the real solid harmonics.  Summed over a cluster's particles, the Taylor
polynomial is therefore, exactly and term by term,

  sum_(l,m,k)  A_lmk B_lm(d) (-1)^l D^l lap^k f,   A_lmk = const sum_i q_i |y_i|^2k B_lm(y_i),

and each A_lmk is a fixed combination of the Cartesian moments of degree l + 2k.  It is the
reference's polynomial regrouped, so the values agree to rounding; but lap^k f collapses:

  f = e^(-kappa r)/r:  lap^k f = kappa^2k f, so every k of one (l, m) shares one coefficient
      and nterms^2 = 81 of them (nterms 9) take the place of 165 (Coulomb: kappa = 0, k = 0);
  f = e^(-kappa rho)/rho, rho^2 = r^2 + delta:  with E_s = (-D)^s f,
      lap E_s = kappa^2 E_s + 2 s E_(s+1) - delta E_(s+2), so lap^k f is a combination of
      E_0, E_2 .. E_2k whose factors depend on the system only: nterms 9 has 200 coefficients.

E_s = (2s - 1)!! beta_s rho^-(2s+1) with beta_0 = e^-x, beta_1 = (1 + x) e^-x,
beta_(s+1) = beta_s + x^2 beta_(s-1) / ((2s + 1)(2s - 1)), x = kappa rho: every term positive.

B_lm = Q_lm(z) Re / Im (x + i y)^m, Q_mm = 1, Q_(l+1)m = z Q_lm - c_lm |.|^2 Q_(l-1)m,
c_lm = (l^2 - m^2)/(4 l^2 - 1): the associated Legendre function, scaled to a leading 1.

The gradient of the same polynomial (treetaylorforce, :456-810; shielded_treetaylorforce,
:2745-2973) reads the same coefficients.  With U_lm the coefficient times its radial factor,
S = sum U_lm B_lm(v) and the derivative of the radial factors by Euler's theorem,

  grad phi = c (S_v - d' (S + 2 v.S_v + sum U'_lm B_lm(v))),   S_v = grad_v S at fixed U,

where U' is 2 s per term of E_(l+s) (delta > 0), and kappa^2 H r g_(l-1) / (2l - 1) in the place
of g_l (screened, delta = 0).  S_v needs no further harmonics: d/dz B_lm = k_lm B_(l-1)m, and
as a function of z and |v|^2, d/d|v|^2 Q_lm = n_lm Q_(l-1)(m+1).

Written per nterms: four evaluation functions (delta = 0 or not, kappa = 0 or not), three of
the gradient, the order in which they read a cluster's coefficients, and, once for all orders,
the table of the harmonic moments A in terms of the shell-order Cartesian moments.

Usage: python gen_harmonics.py <out.cuh>
"""
import sys
from fractions import Fraction
from math import factorial

NTMAX = 10
# evaluation variants: (name, regularised, screened)
VARIANTS = [("hc", False, False), ("hs", False, True), ("rc", True, False), ("rs", True, True)]


def dfact(n):
    r = 1
    while n > 1:
        r *= n
        n -= 2
    return r


# -------------------------------------------------- polynomials {(i, j, k): Fraction}
def pmul(a, b):
    r = {}
    for (i, j, k), u in a.items():
        for (p, q, s), v in b.items():
            w = (i + p, j + q, k + s)
            r[w] = r.get(w, 0) + u * v
    return {w: c for w, c in r.items() if c}


def padd(a, b, f=1):
    r = dict(a)
    for w, c in b.items():
        r[w] = r.get(w, 0) + f * c
    return {w: c for w, c in r.items() if c}


X, Y, Z = {(1, 0, 0): Fraction(1)}, {(0, 1, 0): Fraction(1)}, {(0, 0, 1): Fraction(1)}
R2 = {(2, 0, 0): Fraction(1), (0, 2, 0): Fraction(1), (0, 0, 2): Fraction(1)}
ONE = {(0, 0, 0): Fraction(1)}


def rec_c(l, m):
    return Fraction(l * l - m * m, 4 * l * l - 1)


def solid_harmonics(lmax):
    """{(l, m, part)}: B_lm as a polynomial; part 0: Re, 1: Im (m >= 1)."""
    out = {}
    cm, sm = ONE, {}
    for m in range(lmax + 1):
        q0, q1 = {}, ONE  # Q_(l-1)m, Q_lm
        for l in range(m, lmax + 1):
            out[(l, m, 0)] = pmul(q1, cm)
            if m:
                out[(l, m, 1)] = pmul(q1, sm)
            q2 = pmul(Z, q1)
            if q0:
                q2 = padd(q2, pmul(R2, q0), -rec_c(l, m))
            q0, q1 = q1, q2
        cm, sm = padd(pmul(X, cm), pmul(Y, sm), -1), padd(pmul(X, sm), pmul(Y, cm))
    return out


def weight(l, m):
    """w_lm: |y|^l |d|^l P_l(cos) = sum_m w_lm B_lm(y) B_lm(d) (the addition theorem)."""
    lead = Fraction(factorial(2 * l), 2 ** l * factorial(l) * factorial(l - m))
    return (2 if m else 1) * Fraction(factorial(l - m), factorial(l + m)) * lead * lead


def shell_pos(v):
    """Position of moment (i, j, k) in shell order (degree, then i, then j descending)."""
    i, j, k = v
    d = i + j + k
    return d * (d + 1) * (d + 2) // 6 + (d - i) * (d - i + 1) // 2 + (d - i - j)


def harmonic_list(nt):
    """(l, m, part, k) of the harmonic moments, by degree l + 2k: a prefix for every order."""
    out = []
    for n in range(nt):
        for k in range(n // 2 + 1):
            l = n - 2 * k
            for m in range(l + 1):
                for part in range(2 if m else 1):
                    out.append((l, m, part, k))
    return out


def harmonic_table(nt):
    """Per harmonic moment: [(shell position, factor)], the constants of the header included."""
    B = solid_harmonics(nt - 1)
    r2k = [ONE]
    for _ in range(nt // 2):
        r2k.append(pmul(r2k[-1], R2))
    rows = []
    for l, m, part, k in harmonic_list(nt):
        c = Fraction(2 * l + 1, 2 ** k * factorial(k) * dfact(2 * l + 2 * k + 1)) * weight(l, m)
        p = pmul(r2k[k], B[(l, m, part)])
        rows.append(sorted((shell_pos(v), float(c * f)) for v, f in p.items()))
    return rows


# --------------------------------------------------------------- coefficients of a variant
def radial_set(nt, l, reg):
    """The s of E_(l+s) that degree l needs: 0, and 2 .. 2 kmax when delta > 0."""
    kmax = (nt - 1 - l) // 2
    return [0] + (list(range(2, 2 * kmax + 1)) if reg else [])


def coefficient_list(nt, reg):
    """(l, m, part, s) in the order the evaluation reads them."""
    out = []
    for m in range(nt):
        for l in range(m, nt):
            for part in range(2 if m else 1):
                for s in radial_set(nt, l, reg):
                    out.append((l, m, part, s))
    return out


def padded(n):
    return (n + 3) // 4 * 4


# ------------------------------------------------------------------------- evaluation code
def lit(v):
    return f"T({float(v)!r})"


# Past X_MAX = kappa rho the exponential is 0 in either precision, and so is the result: kappa rho
# is held there, and kappa H at KH_MAX, so that no factor beside that 0 is infinite.
X_MAX, KH_MAX = 2.0 ** 20, 2.0 ** 50


class Loads:
    """A cluster's coefficients, four at a time, where they are first needed."""

    def __init__(self, L):
        self.L, self.done, self.next = L, -1, 0

    def get(self):
        q, i = divmod(self.next, 4)
        self.next += 1
        if q > self.done:
            self.L.append(f"  const V4<T> mv{q} = ld4(M, {q});")
            self.done = q
        return f"mv{q}.{'xyzw'[i]}"


def gen_eval(nt, reg, scr):
    """The potential of one cluster at d = (dx, dy, dz): `r2` = |d|^2, `add` = delta, `H` the
    length the coefficients are scaled with, M the cluster's coefficients.

    delta = 0: u = d/r, radial factors g_l = beta_l (H/r)^l / r.
    delta > 0: v = H d / rho^2 (so B_lm(v) carries (H/rho^2)^l), radial factors beta_(l+s)
    (H/rho)^2s, times 1/rho at the end."""
    L = []
    top = nt - 1
    if not reg:
        L += ["  const T ri = rsqrt_t(r2);",
              "  const T vx = dx * ri, vy = dy * ri, vz = dz * ri;"]
        if top >= 1:
            L.append("  const T eta = H * ri;")
        if scr:
            L += ["  const T x = kappa * (r2 * ri);",
                  "  const T g0 = exp_t(-x) * ri;"]
            if top >= 1:
                L.append("  const T g1 = eta * fma_t(x, g0, g0);")
            if top >= 2:
                L += [f"  const T kh = min(kappa * H, {lit(KH_MAX)});", "  const T kh2 = kh * kh;"]
            for l in range(2, nt):
                c = Fraction(1, (2 * l - 1) * (2 * l - 3))
                L.append(f"  const T g{l} = fma_t({lit(c)}, kh2 * g{l - 2}, eta * g{l - 1});")
        else:
            L.append("  const T g0 = ri;")
            for l in range(1, nt):
                L.append(f"  const T g{l} = g{l - 1} * eta;")
        rad = lambda l, s: f"g{l}"
    else:
        L += ["  const T rho2 = r2 + add;",
              "  const T ri = rsqrt_t(rho2);"]
        if top >= 1:
            L += ["  const T eta = H * ri;",
                  "  const T f = eta * ri;",
                  "  const T vx = dx * f, vy = dy * f, vz = dz * f;"]
        if top >= 2:
            L += ["  const T n2 = fma_t(vx, vx, fma_t(vy, vy, vz * vz));",
                  "  const T t1 = eta * eta;",
                  "  const T t2 = t1 * t1;"]
            for s in range(3, 2 * (top // 2) + 1):
                L.append(f"  const T t{s} = t{s - 1} * t1;")
        if scr:
            L += [f"  const T x = min(kappa * (rho2 * ri), {lit(X_MAX)});",
                  "  const T b0 = exp_t(-x);"]
            if top >= 1:
                L.append("  const T b1 = fma_t(x, b0, b0);")
            if top >= 2:
                L.append("  const T x2 = x * x;")
            for j in range(2, nt):
                c = Fraction(1, (2 * j - 1) * (2 * j - 3))
                L.append(f"  const T b{j} = fma_t({lit(c)}, x2 * b{j - 2}, b{j - 1});")
            for l in range(nt):
                for s in radial_set(nt, l, True)[1:]:
                    L.append(f"  const T w{l}_{s} = b{l + s} * t{s};")
            rad = lambda l, s: f"b{l}" if s == 0 else f"w{l}_{s}"
        else:
            rad = lambda l, s: None if s == 0 else f"t{s}"
    ld = Loads(L)

    def term(acc, l, s, m):
        """acc + m * radial(l, s), as an expression."""
        r = rad(l, s)
        if r is None:
            return m if acc is None else f"{m} + {acc}"
        return f"{m} * {r}" if acc is None else f"fma_t({m}, {r}, {acc})"

    def q_next(l, m):
        """Q_(l+1)m from Q_lm and Q_(l-1)m; None stands for 1 (Q_mm)."""
        if l == m:
            return "vz"
        c = lit(-rec_c(l, m))
        prev = f"q{m}_{l - 1}" if l - 1 > m else None
        if reg:
            tail = f"{c} * n2" if prev is None else f"{c} * (n2 * {prev})"
        else:
            tail = c if prev is None else f"{c} * {prev}"
        return f"fma_t(vz, q{m}_{l}, {tail})"

    # The monopole term, the largest of a charged cluster, is added last, so that the others
    # are summed at their own size.
    mono = ld.get()
    for m in range(nt):
        if m == 1:
            L.append("  const T c1 = vx, s1 = vy;")
        elif m > 1:
            L += [f"  const T c{m} = fma_t(vx, c{m - 1}, -(vy * s{m - 1}));",
                  f"  const T s{m} = fma_t(vx, s{m - 1}, vy * c{m - 1});"]
        sums = [None, None]  # the accumulators of Re and Im, once they hold something
        for l in range(m, nt):
            q = None
            if l > m:
                q = f"q{m}_{l}"
                L.append(f"  const T {q} = {q_next(l - 1, m)};")
            w = None
            if not reg and q is not None:
                w = f"w{m}_{l}"
                L.append(f"  const T {w} = g{l} * {q};")
            for part in range(2 if m else 1):
                P = f"{'pq'[part]}{m}"
                e = None
                if not reg:
                    if l > 0:
                        mv = ld.get()
                        f = w or f"g{l}"
                        e = f"fma_t({mv}, {f}, {P})" if sums[part] else f"{mv} * {f}"
                else:
                    acc = None
                    for s in radial_set(nt, l, True):
                        if (l, s) != (0, 0):
                            acc = term(acc, l, s, ld.get())
                    if acc is None:
                        continue
                    if q is None:  # Q = 1: the first of this m
                        e = acc
                    else:
                        nm = f"u{m}_{l}_{part}"
                        L.append(f"  const T {nm} = {acc};")
                        e = f"fma_t({nm}, {q}, {P})" if sums[part] else f"{nm} * {q}"
                if e is not None:
                    L.append(f"  {'' if sums[part] else 'T '}{P} = {e};")
                    sums[part] = P
        if m == 0:
            S = sums[0]
        elif S == "p0":
            L.append(f"  T S = fma_t(c{m}, p{m}, fma_t(s{m}, q{m}, p0));")
            S = "S"
        else:
            L.append(f"  S = fma_t(c{m}, p{m}, fma_t(s{m}, q{m}, S));")
    r0 = rad(0, 0)
    e = (f"{mono} * {r0}" if S is None else f"fma_t({mono}, {r0}, {S})") if r0 else \
        (mono if S is None else f"{mono} + {S}")
    if reg:
        e = f"({e}) * ri"
    L.append(f"  const T pot = {e};")
    L.append("  return pot;")
    return L


def grad_constants(lmax):
    """{(l, m): (k_lm, n_lm)} of the header, from Q_lm as polynomials in z and n2 = |.|^2."""
    Q = {}
    for m in range(lmax + 2):
        for l in range(m, lmax + 1):
            if l == m:
                Q[l, m] = {(0, 0): Fraction(1)}
                continue
            q = {(i + 1, j): c for (i, j), c in Q[l - 1, m].items()}
            if l - 2 >= m:
                for (i, j), c in Q[l - 2, m].items():
                    q[i, j + 1] = q.get((i, j + 1), 0) - rec_c(l - 1, m) * c
            Q[l, m] = {w: c for w, c in q.items() if c}

    def ratio(a, b):
        if not a:
            return Fraction(0)
        w = next(iter(b))
        f = a[w] / b[w]
        assert a == {v: f * c for v, c in b.items()}
        return f
    out = {}
    for (l, m), q in Q.items():
        dz, dn = {}, {}
        for (i, j), c in q.items():  # d/dz with n2 following z, d/dn2 alone
            if i:
                dz[i - 1, j] = dz.get((i - 1, j), 0) + i * c
            if j:
                dz[i + 1, j - 1] = dz.get((i + 1, j - 1), 0) + 2 * j * c
                dn[i, j - 1] = dn.get((i, j - 1), 0) + j * c
        dz = {w: c for w, c in dz.items() if c}
        out[l, m] = (ratio(dz, Q.get((l - 1, m), {(0, 0): 1})), ratio(dn, Q.get((l - 1, m + 1), {(0, 0): 1})))
    return out


GRADIENTS = [("ghc", False, False), ("ghs", False, True), ("grc", True, False)]


def gen_grad(nt, reg, scr):
    """Minus the gradient of one cluster's potential: arguments as gen_eval's, into fx, fy, fz."""
    L = []
    top = nt - 1
    K = grad_constants(top)
    if not reg:
        L += ["  const T ri = rsqrt_t(r2);",
              "  const T vx = dx * ri, vy = dy * ri, vz = dz * ri;"]
        if top >= 1:
            L.append("  const T eta = H * ri;")
        if scr:
            L += ["  const T r = r2 * ri;",
                  f"  const T x = min(kappa * r, {lit(X_MAX)});",
                  "  const T g0 = exp_t(-x) * ri;",
                  "  const T h0 = x * g0;"]
            if top >= 1:
                L += ["  const T g1 = eta * fma_t(x, g0, g0);",
                      f"  const T kh = min(kappa * H, {lit(KH_MAX)});", "  const T kr = kh * x;"]
            if top >= 2:
                L.append("  const T kh2 = kh * kh;")
            for l in range(2, nt):
                c = Fraction(1, (2 * l - 1) * (2 * l - 3))
                L.append(f"  const T g{l} = fma_t({lit(c)}, kh2 * g{l - 2}, eta * g{l - 1});")
            for l in range(1, nt):
                L.append(f"  const T h{l} = " + (f"{lit(Fraction(1, 2 * l - 1))} * (kr * g{l - 1});" if l > 1
                                                 else f"kr * g{l - 1};"))
        else:
            L.append("  const T g0 = ri;")
            for l in range(1, nt):
                L.append(f"  const T g{l} = g{l - 1} * eta;")
        n2 = None
    else:
        L += ["  const T rho2 = r2 + add;",
              "  const T ri = rsqrt_t(rho2);"]
        if top >= 1:
            L += ["  const T eta = H * ri;",
                  "  const T f = eta * ri;",
                  "  const T vx = dx * f, vy = dy * f, vz = dz * f;"]
        if top >= 2:
            L += ["  const T n2 = fma_t(vx, vx, fma_t(vy, vy, vz * vz));",
                  "  const T t1 = eta * eta;",
                  "  const T t2 = t1 * t1;"]
            for s in range(3, 2 * (top // 2) + 1):
                L.append(f"  const T t{s} = t{s - 1} * t1;")
            for s in range(2, 2 * (top // 2) + 1):
                L.append(f"  const T y{s} = {lit(2 * s)} * t{s};")
        n2 = "n2"
    ld = Loads(L)

    def column(m):
        """q{m}_l for l > m, once (Q_mm = 1)."""
        for l in range(m + 1, nt):
            if l == m + 1:
                L.append(f"  const T q{m}_{l} = vz;")
                continue
            c = lit(-rec_c(l - 1, m))
            prev = f"q{m}_{l - 2}" if l - 2 > m else None
            if n2:
                tail = f"{c} * n2" if prev is None else f"{c} * (n2 * {prev})"
            else:
                tail = c if prev is None else f"{c} * {prev}"
            L.append(f"  const T q{m}_{l} = fma_t(vz, q{m}_{l - 1}, {tail});")

    Q = lambda l, m: None if l == m else f"q{m}_{l}"
    have = set()

    def add(P, a, b):
        """P += a * b; a or b None stands for 1."""
        e = a if b is None else b if a is None else None
        if P in have:
            L.append(f"  {P} = {e} + {P};" if e else f"  {P} = fma_t({a}, {b}, {P});")
        else:
            L.append(f"  T {P} = {e};" if e else f"  T {P} = {a} * {b};")
            have.add(P)

    mono = ld.get()
    column(0)
    for m in range(nt):
        if m == 1:
            L.append("  const T c1 = vx, s1 = vy;")
        elif m > 1:
            L += [f"  const T c{m} = fma_t(vx, c{m - 1}, -(vy * s{m - 1}));",
                  f"  const T s{m} = fma_t(vx, s{m - 1}, vy * c{m - 1});"]
        if m < top:
            column(m + 1)
        for l in range(m, nt):
            if (l, m) != (0, 0):
                k, n = K[l, m]
                if l - 1 >= m:
                    w = Q(l - 1, m)
                    L.append(f"  const T z{m}_{l} = " + (f"{lit(k)} * {w};" if w else f"{lit(k)};"))
                if l - 1 >= m + 1:
                    w = Q(l - 1, m + 1)
                    L.append(f"  const T n{m}_{l} = " + (f"{lit(2 * n)} * {w};" if w else f"{lit(2 * n)};"))
            for part in range(2 if m else 1):
                pq = f"{'pq'[part]}{m}"
                nm = f"u{m}_{l}_{part}"
                if reg:
                    u = g = None
                    for s in radial_set(nt, l, True):
                        if (l, m, s) == (0, 0, 0):
                            continue
                        mv = ld.get()
                        u = (mv if s == 0 else f"{mv} * t{s}") if u is None else f"fma_t({mv}, t{s}, {u})"
                        if s:
                            g = f"{mv} * y{s}" if g is None else f"fma_t({mv}, y{s}, {g})"
                else:
                    mv = mono if (l, m) == (0, 0) else ld.get()
                    u = f"{mv} * g{l}"
                    g = f"{mv} * h{l}" if scr else None
                if u is not None:
                    L.append(f"  const T {nm} = {u};")
                    if reg or (l, m) != (0, 0):  # (delta = 0: the monopole is added at the end)
                        add(pq, nm, Q(l, m))
                    if l - 1 >= m:
                        add("z" + pq, nm, f"z{m}_{l}")
                    if l - 1 >= m + 1:
                        add("n" + pq, nm, f"n{m}_{l}")
                if g is not None:
                    L.append(f"  const T v{nm} = {g};")
                    add("g" + pq, "v" + nm, Q(l, m))
        # the sums of this m: S, its derivatives, and the radial part
        for sp, tot in (("", "S"), ("z", "Sz"), ("n", "N"), ("g", "G")):
            if sp + f"p{m}" in have:
                add(tot, sp + f"p{m}", f"c{m}" if m else None)
            if m and sp + f"q{m}" in have:
                add(tot, sp + f"q{m}", f"s{m}")
        if m and f"p{m}" in have:
            mm = lit(m)
            if m == 1:
                add("Sx", "p1", None)
                add("Sy", "q1", None)
            else:
                L.append(f"  const T a{m} = {mm} * p{m}, e{m} = {mm} * q{m};")
                add("Sx", f"a{m}", f"c{m - 1}")
                add("Sx", f"e{m}", f"s{m - 1}")
                add("Sy", f"e{m}", f"c{m - 1}")
                add("Sy", f"-a{m}", f"s{m - 1}")
    if "N" in have:
        add("Sx", "vx", "N")
        add("Sy", "vy", "N")
    e = "S" if "S" in have else None
    if "Sz" in have:
        L.append(f"  const T dot = fma_t(vx, Sx, fma_t(vy, Sy, vz * Sz));")
        e = f"fma_t(T(2), dot, {e})"
    if "G" in have:
        e = f"{e} + G" if e else "G"
    if reg:
        L.append(f"  const T R = {f'{mono} + ({e})' if e else mono};")
        L.append("  const T i2 = ri * ri;")
        for a in "xyz":  # (ri^3 would leave the range of FP32 earlier than the field does)
            w = f"(d{a} * ri)"
            L.append(f"  f{a} = i2 * " + (f"fma_t({w}, R, -(eta * S{a}));" if "Sz" in have else f"({w} * R);"))
    else:
        L.append(f"  const T R = " + (f"fma_t({mono}, g0, {e});" if e else f"{mono} * g0;"))
        for a in "xyz":
            L.append(f"  f{a} = ri * " + (f"fma_t(v{a}, R, -S{a});" if "Sz" in have else f"(v{a} * R);"))
    return L


def field_flops_per_pair(nt):
    """Flops per pair of the fields: "force" (delta > 0), "force0" (delta = 0), "curl"."""
    f = lambda reg, scr: (lambda c: 2 * c[0] + c[1])(count_ops(gen_grad(nt, reg, scr)))
    return {"force": f(True, False), "force0": f(False, False), "curl": f(False, True)}


def ops_per_pair(nt, reg, scr):
    """(fma, other) floating-point instructions of one evaluation."""
    return count_ops(gen_eval(nt, reg, scr))


def count_ops(lines):
    import re
    fma = other = 0
    for ln in lines:
        if "ld4(" in ln:
            continue
        e = re.sub(r"T\([^()]*\)", "C", ln.split("=", 1)[-1])
        fma += e.count("fma_t(")
        other += e.count("rsqrt_t(") + e.count("exp_t(") + e.count(" * ") + e.count(" + ")
    return fma, other


def flops_per_pair(nt):
    """Flops (2 per fma) per (target, cluster) pair of the kernels a potential without delta
    ("screened", "coulomb0") and with delta ("coulomb", "screened_reg") runs."""
    f = lambda reg, scr: (lambda c: 2 * c[0] + c[1])(ops_per_pair(nt, reg, scr))
    return {"coulomb0": f(False, False), "screened": f(False, True), "coulomb": f(True, False),
            "screened_reg": f(True, True)}


# -------------------------------------------------------------------------------- the file
def main(out):
    parts = ["// GENERATED by gen_harmonics.py -- do not edit.",
             "#pragma once",
             "namespace bit {"]
    rows = harmonic_table(NTMAX)
    hl = harmonic_list(NTMAX)
    pos = {h: i for i, h in enumerate(hl)}
    begin, idx, val = [0], [], []
    for r in rows:
        idx += [p for p, _ in r]
        val += [f for _, f in r]
        begin.append(len(idx))
    arr = lambda t, nm, v, f=str: parts.append(
        f"__device__ const {t} {nm}[{len(v)}] = {{" + ", ".join(map(f, v)) + "};")
    parts.append("// harmonic moment h = sum over e in [kHarmBegin[h], kHarmBegin[h + 1]) of")
    parts.append("// kHarmFactor[e] * (shell-order moment kHarmShell[e])")
    arr("unsigned short", "kHarmBegin", begin)
    arr("unsigned char", "kHarmShell", idx)
    arr("double", "kHarmFactor", val, repr)
    parts.append("// Coefficient p of an order: l, s, the harmonic moment of its k = 0, the number of k, and")
    parts.append("// the distance in the list from one k to the next is found from the degree (harm_index).")
    parts.append("struct HarmCoef { unsigned char l, s, m, part; };")
    meta = []
    offs = {}
    for reg in (False, True):
        for nt in range(1, NTMAX + 1):
            cl = coefficient_list(nt, reg)
            offs[(reg, nt)] = (len(meta), len(cl))
            meta += [f"{{{l}, {s}, {m}, {p}}}" for l, m, p, s in cl]
    arr("HarmCoef", "kHarmCoef", meta)
    for reg in (False, True):
        nm = "kHarmCoefBegin" + ("Reg" if reg else "")
        arr("unsigned short", nm, [0] + [offs[(reg, nt)][0] for nt in range(1, NTMAX + 1)])
    for reg in (False, True):
        f = "harm_count_reg" if reg else "harm_count"
        parts.append(f"__host__ __device__ constexpr int {f}(int nt) {{")
        parts.append("  constexpr int n[] = {0, " + ", ".join(
            str(offs[(reg, nt)][1]) for nt in range(1, NTMAX + 1)) + "};")
        parts.append("  return n[nt];")
        parts.append("}")
    parts.append("// index of harmonic moment (l, m, part, k): degrees below n = l + 2k hold n (n+1) (n+2) / 6,")
    parts.append("// then the larger l of degree n, then 2m - 1 + part")
    parts.append("__host__ __device__ constexpr int harm_index(int l, int m, int part, int k) {")
    parts.append("  const int n = l + 2 * k;")
    parts.append("  int i = n * (n + 1) * (n + 2) / 6;")
    parts.append("  for (int j = 0; j < k; j++) i += 2 * (n - 2 * j) + 1;")
    parts.append("  return i + (m ? 2 * m - 1 + part : 0);")
    parts.append("}")
    for (l, m, p, k), i in pos.items():
        n = l + 2 * k
        chk = n * (n + 1) * (n + 2) // 6 + sum(2 * (n - 2 * j) + 1 for j in range(k)) + (2 * m - 1 + p if m else 0)
        assert chk == i
    parts.append("template <int NT> struct Harmonics;")
    for nt in range(1, NTMAX + 1):
        parts.append(f"template <> struct Harmonics<{nt}> {{")
        for nm, reg, scr in VARIANTS:
            parts.append(f"  template <class T> static __device__ __forceinline__ T {nm}("
                         "T dx, T dy, T dz, T r2, T add, T kappa, T H, const T* __restrict__ M) {")
            parts += ["  " + ln for ln in gen_eval(nt, reg, scr)]
            parts.append("  }")
        for nm, reg, scr in GRADIENTS:
            parts.append(f"  template <class T> static __device__ __forceinline__ void {nm}("
                         "T dx, T dy, T dz, T r2, T add, T kappa, T H, const T* __restrict__ M, T& fx, T& fy, "
                         "T& fz) {")
            parts += ["  " + ln for ln in gen_grad(nt, reg, scr)]
            parts.append("  }")
        parts.append("};")
    parts.append("}  // namespace bit")
    with open(out, "w") as f:
        f.write("\n".join(parts) + "\n")


if __name__ == "__main__":
    main(sys.argv[1])
