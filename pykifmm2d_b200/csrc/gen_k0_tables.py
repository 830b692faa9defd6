"""Generate k0_tables.h: coefficients for the modified Bessel function K0 and
the Hankel function H0.

Method (derived here from the mathematics, evaluated with mpmath at 50 digits):
  0 < x <= 2:  K0(x) = P(t) - log(x/2) * I0(t),  t = x^2, with the power series
               I0 = sum_k t^k / (4^k (k!)^2),  P = sum_k (H_k - gamma) t^k / (4^k (k!)^2)
               (H_k the harmonic numbers, H_0 = 0; DLMF 10.31.2 and 10.25.2).
  x > 2:       K0(x) = exp(-x) / sqrt(x) * F(z),  z = 8/x in (0, 4),
               F(z) = sqrt(x) exp(x) K0(x) smooth on [0, 4] (F(0) = sqrt(pi/2)),
               as a Chebyshev series in u = z/2 - 1 on [-1, 1], coefficients from
               the discrete Chebyshev transform at 64 Chebyshev nodes.
and F as the polynomial in u that its first 24 Chebyshev terms make (its power
coefficients fall off nearly as fast: 0.94 x 2^-53 relative error in FP64).
Terms are kept while they matter at double (FP64) or single (FP32) precision.
The FP64 pair loops (pair_f64.cuh) take the same series in the forms
  K0(x)          = P(t) + ln(t/4) I0H(t),  I0H = -I0 / 2,
  (i/4) H0(x)    = ln(t/4) A(t) + R(t) + i (-pi) A(t),
  A = -J0 / (4 pi),  R = sum_k (-1)^k p_k t^k / (2 pi)  (p_k those of P; DLMF 10.8.2);
for 4 <= t <= 64 the same A and R (entire functions of t) as polynomials in
u = (t - 34) / 30, and for t >= 64 Hankel's form (DLMF 10.2.5)
  H0(x) = sqrt(2 / (pi x)) exp(i (x - pi/4)) (p(v) + i q(v) / x),  v = 128 / t - 1,
p and q as polynomials in v; coefficients from the Chebyshev transform at 64 nodes.

Run:  python pykifmm2d_b200/csrc/gen_k0_tables.py   (rewrites k0_tables.h beside it)
"""
import os

import mpmath as mp

mp.mp.dps = 50
HERE = os.path.dirname(os.path.abspath(__file__))


def series(nterms):
    g = mp.euler
    i0, p = [], []
    h = mp.mpf(0)
    for k in range(nterms):
        if k > 0:
            h += mp.mpf(1) / k
        c = mp.mpf(1) / (mp.mpf(4) ** k * mp.factorial(k) ** 2)
        i0.append(c)
        p.append((h - g) * c)
    return i0, p


def cheb_large(n=64):
    # F(z) = sqrt(x) e^x K0(x), x = 8/z ; u = z/2 - 1
    def F(u):
        z = 2 * (u + 1)
        if z == 0:
            return mp.sqrt(mp.pi / 2)
        x = 8 / z
        return mp.sqrt(x) * mp.exp(x) * mp.besselk(0, x)
    nodes = [mp.cos(mp.pi * (j + mp.mpf(1) / 2) / n) for j in range(n)]
    vals = [F(u) for u in nodes]
    coef = []
    for k in range(n):
        s = sum(vals[j] * mp.cos(mp.pi * k * (j + mp.mpf(1) / 2) / n) for j in range(n))
        coef.append(2 * s / n)
    coef[0] /= 2
    return coef


def monomial(c):
    """coefficients in powers of u of sum_k c[k] T_k(u)"""
    t0, t1 = [mp.mpf(1)], [mp.mpf(0), mp.mpf(1)]
    out = [mp.mpf(0)] * len(c)
    for k, ck in enumerate(c):
        for i, v in enumerate(t0):
            out[i] += ck * v
        t2 = [mp.mpf(0)] + [2 * v for v in t1]
        for i, v in enumerate(t0):
            t2[i] -= v
        t0, t1 = t1, t2
    return out


def trim(c, tol):
    scale = max(abs(v) for v in c)
    last = 0
    for i, v in enumerate(c):
        if abs(v) > tol * scale:
            last = i
    return c[: last + 1]


def fmt(vals, single):
    if single:
        return ",\n    ".join("%.9ef" % float(v) for v in vals)
    return ",\n    ".join("%.17e" % float(v) for v in vals)


def cheb_of(f, tol, n=64):
    """power coefficients of f on [-1, 1], Chebyshev terms kept above tol"""
    vals = [f(mp.cos(mp.pi * (j + mp.mpf(1) / 2) / n)) for j in range(n)]
    c = [2 * sum(vals[j] * mp.cos(mp.pi * k * (j + mp.mpf(1) / 2) / n) for j in range(n)) / n for k in range(n)]
    c[0] /= 2
    return monomial(c[: max(i for i, v in enumerate(c) if abs(v) > tol) + 1])


def hankel():
    def mid(u):  # (A, R) at t = 34 + 30 u
        t = 34 + 30 * u
        x = mp.sqrt(t)
        a = -mp.besselj(0, x) / (4 * mp.pi)
        return a, -mp.bessely(0, x) / 4 - mp.log(t / 4) * a

    def far(v):  # p + i q
        w = (v + 1) / 2
        x = 8 / mp.sqrt(w)
        s = (mp.besselj(0, x) + 1j * mp.bessely(0, x)) * mp.sqrt(mp.pi * x / 2) * mp.exp(-1j * (x - mp.pi / 4))
        return s.real, s.imag * x
    return (cheb_of(lambda u: mid(u)[0], 3e-18), cheb_of(lambda u: mid(u)[1], 1e-17),
            cheb_of(lambda v: far(v)[0], 1e-17), cheb_of(lambda v: far(v)[1], 1e-17))


def main():
    i0, p = series(40)
    # t <= 4: term k is at most 4^k c_k = 1/(k!)^2 in size; keep while above the precision
    def trim_series(c, tol):
        last = max(i for i, v in enumerate(c) if abs(v) * 4 ** i > tol)
        return c[: last + 1]
    i0_64 = trim_series(i0, 1e-19); p_64 = trim_series(p, 1e-19)
    i0_32 = trim_series(i0, 1e-9); p_32 = trim_series(p, 1e-9)
    ch = cheb_large()
    ch_64 = trim(ch, 1e-18)
    ch_32 = trim(ch, 2e-9)
    out = []
    out.append("/* Generated by gen_k0_tables.py -- do not edit.  Coefficients for K0:")
    out.append(" * x <= 2: K0 = P(x^2) - log(x/2) I0(x^2) with power series in t = x^2;")
    out.append(" * x >  2: K0 = exp(-x)/sqrt(x) * sum_k c_k T_k(u), u = 4/x - 1 (Chebyshev). */")
    out.append("#pragma once")
    nt = len(i0_64)
    i0h = [-v / 2 for v in i0_64]
    h0a = [-(-1) ** k * v / (4 * mp.pi) for k, v in enumerate(i0[:nt])]
    h0r = [(-1) ** k * v / (2 * mp.pi) for k, v in enumerate(p[:nt])]
    ma, mr, hp, hq = hankel()
    for name, vals, single in (("H0_MID_A_D", ma, False), ("H0_MID_R_D", mr, False), ("H0_P_D", hp, False),
                               ("H0_Q_D", hq, False), ("K0_I0H_D", i0h, False), ("H0_A_D", h0a, False), ("H0_R_D", h0r, False),
                               ("K0_I0_D", i0_64, False), ("K0_P_D", p_64, False), ("K0_CHEB_D", ch_64, False),
                               ("K0_FAR_D", monomial(ch[:24]), False),
                               ("K0_I0_F", i0_32, True), ("K0_P_F", p_32, True), ("K0_CHEB_F", ch_32, True)):
        ty = "float" if single else "double"
        out.append(f"#define {name}_N {len(vals)}")
        out.append(f"static __device__ __constant__ {ty} {name}[{len(vals)}] = {{\n    {fmt(vals, single)}}};")
    open(os.path.join(HERE, "k0_tables.h"), "w").write("\n".join(out) + "\n")
    print("terms: I0 %d/%d  P %d/%d  cheb %d/%d" % (len(i0_64), len(i0_32), len(p_64), len(p_32), len(ch_64), len(ch_32)))


if __name__ == "__main__":
    main()
