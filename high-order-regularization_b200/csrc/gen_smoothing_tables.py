"""Generates hr_smoothing_tables.inc (FP32) and hr_eval64_tables.inc (FP64):
piecewise polynomials for the smoothing factors of the regularized kernels, as
functions of s = (r/delta)^2.

With lam = r / delta and E(lam) = (2/sqrt(pi)) lam exp(-lam^2), the on-surface
factors of the 7th-order kernels (2S/utilities.cpp:211-254 and :292-323) are

    s1 = [erf(lam) + (11/5 - 26/15 lam^2 + 4/15 lam^4) E] / r           = G1(s) / delta
    s2 = [erf(lam) + (-1 + (118 lam^2 - 68 lam^4 + 8 lam^6)/15) E] / r^3 = G2(s) / delta^3
    s3 = [erf(lam) + (-1 - 2/3 lam^2 + 52/45 lam^4 - 8/45 lam^6) E] / r^5 = G3(s) / delta^5

where G1 = f1 / lam, G2 = f2 / lam^3, G3 = f3 / lam^5 are even in lam and
therefore analytic in s = lam^2, with the reference's r -> 0 values
(32/5, 256/15, 128/45) / sqrt(pi) as their limits at s = 0.

FP32 tables (the reduced-precision path): pieces uniform in s with the piece
index floor(s * NI32 / 64), checked by emulating their FP32 evaluation.

FP64 tables (hr_eval64_tables.inc): pieces of width 1/4 in s, piece i centred
at i / 4, monomial coefficients in t = s - i / 4 (Chebyshev interpolants solved
in 80-digit arithmetic). The factors come in pairs: with E0(s) = erf(lam) / lam,

    F(s) = (E0 - 2/sqrt(pi) e^-s) / s            = -2 E0'(s),
    T(s) = (F - 4/(3 sqrt(pi)) e^-s) / s         = -(2/3) F'(s),
    G2(s)                                        = -2 G1'(s),

so one polynomial per piece gives both of a pair, by value and by derivative
(the derivative's coefficients are fitted, the polynomial's follow from them).
The off-surface factors of a target with coefficients c1..c3 are
s1 = (E0 + P1 e^-s) / delta, s2 = (F + Q2 e^-s) / delta^3 and
s3 = (T + Q3 e^-s) / delta^5 with polynomials P1, Q2, Q3 in s.

Run from this directory: python gen_smoothing_tables.py
"""
import os

import mpmath as mp

mp.mp.dps = 80
HERE = os.path.dirname(os.path.abspath(__file__))


def E(lam):
    return 2 / mp.sqrt(mp.pi) * lam * mp.exp(-lam * lam)


def G1(s):
    if s == 0:
        return mp.mpf(32) / 5 / mp.sqrt(mp.pi)
    lam = mp.sqrt(s)
    return (mp.erf(lam) + (mp.mpf(11) / 5 - mp.mpf(26) / 15 * s + mp.mpf(4) / 15 * s * s) * E(lam)) / lam


def G2(s):
    if s == 0:
        return mp.mpf(256) / 15 / mp.sqrt(mp.pi)
    lam = mp.sqrt(s)
    return (mp.erf(lam) + (-1 + (118 * s - 68 * s * s + 8 * s ** 3) / 15) * E(lam)) / lam ** 3


def G3(s):
    if s == 0:
        return mp.mpf(128) / 45 / mp.sqrt(mp.pi)
    lam = mp.sqrt(s)
    return (mp.erf(lam) + (-1 - mp.mpf(2) / 3 * s + mp.mpf(52) / 45 * s * s - mp.mpf(8) / 45 * s ** 3) * E(lam)) / lam ** 5


def horner(coef, t):
    p = mp.mpf(0)
    for a in reversed(coef):
        p = p * t + a
    return p


# FP32 tables for the mixed-precision path: NI32 pieces uniform in s (index
# floor(s * NI32 / 64), no square root), degree DEG32, each piece stored as
# 8 floats (centre, coefficients of t^0 .. t^5, 0) = two float4.
NI32 = 128
DEG32 = 5


def piece32(f, i):
    w = mp.mpf(64) / NI32
    slo = max(mp.mpf(0), i * w - mp.mpf("0.01"))
    shi = (i + 1) * w + mp.mpf("0.01")
    c = (i + mp.mpf(1) / 2) * w
    half, mid = (shi - slo) / 2, (shi + slo) / 2
    n = DEG32 + 1
    ts = [mid + half * mp.cos(mp.pi * (k + mp.mpf(1) / 2) / n) - c for k in range(n)]
    V = mp.matrix(n, n)
    for r, t in enumerate(ts):
        for j in range(n):
            V[r, j] = t ** j
    coef = mp.lu_solve(V, mp.matrix([f(t + c) for t in ts]))
    return [coef[j] for j in range(n)], c


def build32(f):
    """Float pieces and the worst relative error of their FP32 Horner evaluation
    (emulated with numpy float32) over 21 points per piece."""
    import numpy as np
    out, worst = [], 0.0
    w = 64.0 / NI32
    for i in range(NI32):
        coef, c = piece32(f, i)
        cf = np.array([float(a) for a in coef], np.float32)
        cc = np.float32(float(c))
        for k in range(21):
            sv = np.float32(i * w + w * k / 20.0)
            t = np.float32(sv - cc)
            v = cf[-1]
            for a in cf[-2::-1]:
                v = np.float32(v * t + a)
            ex = f(mp.mpf(float(sv)))
            worst = max(worst, float(abs(mp.mpf(float(v)) - ex) / abs(ex)))
        out.append([float(cc)] + [float(a) for a in cf] + [0.0] * (6 - DEG32))
    return out, worst


# FP64 tables of the persistent kernels: (name, value function, fitted
# derivative function and its factor: derivative function = factor * d/ds of
# the value function, or None; coefficients per piece; last s).
W64 = mp.mpf(1) / 4


def E0(s):
    if s == 0:
        return 2 / mp.sqrt(mp.pi)
    return mp.erf(mp.sqrt(s)) / mp.sqrt(s)


def F0(s):
    x = 2 / mp.sqrt(mp.pi) * mp.exp(-s)
    if s < mp.mpf("1e-3"):  # the series of erf without its first term
        return x * mp.nsum(lambda k: 2 ** (k + 1) * s ** k / mp.fac2(2 * k + 3), [0, mp.inf])
    return (E0(s) - x) / s


def T0(s):
    x = 2 / mp.sqrt(mp.pi) * mp.exp(-s)
    if s < mp.mpf("1e-3"):
        return x * mp.nsum(lambda k: 2 ** (k + 2) * s ** k / mp.fac2(2 * k + 5), [0, mp.inf])
    return (F0(s) - mp.mpf(2) / 3 * x) / s


TABLES64 = [("G1", G1, G2, -2, 11, 51), ("G3", G3, None, 0, 10, 51), ("E0", E0, F0, -2, 10, 64),
            ("F0", F0, T0, -mp.mpf(2) / 3, 10, 64)]


def piece64(f, fd, factor, c, n):
    """n monomial coefficients about c: the Chebyshev interpolant of f, or that
    of fd (n - 1 coefficients) integrated, with f's value at the centre."""
    def cheb(fn, m):
        slo = max(mp.mpf(0), c - W64 * mp.mpf("0.502"))
        shi = c + W64 * mp.mpf("0.502")
        half, mid = (shi - slo) / 2, (shi + slo) / 2
        ts = [mid + half * mp.cos(mp.pi * (k + mp.mpf(1) / 2) / m) - c for k in range(m)]
        V = mp.matrix(m, m)
        for r, t in enumerate(ts):
            for j in range(m):
                V[r, j] = t ** j
        coef = mp.lu_solve(V, mp.matrix([fn(t + c) for t in ts]))
        return [coef[j] for j in range(m)]

    if fd is None:
        return cheb(f, n)
    b = cheb(fd, n - 1)
    return [f(c)] + [b[k] / (factor * (k + 1)) for k in range(n - 1)]


def build64(f, fd, factor, n, last):
    """Rounded coefficients of pieces 0 .. last / W64 and the worst relative
    errors of the value and of the derivative function (17 points per piece)."""
    out, worst, worstd = [], mp.mpf(0), mp.mpf(0)
    for i in range(int(last / W64) + 1):
        c = i * W64
        cd = [float(a) for a in piece64(f, fd, factor, c, n)]
        for k in range(17):
            t = W64 * (mp.mpf(k) / 16 - mp.mpf(1) / 2)
            if c + t < 0:
                continue
            worst = max(worst, abs(horner([mp.mpf(a) for a in cd], t) / f(c + t) - 1))
            if fd is not None:
                d = horner([j * mp.mpf(cd[j]) for j in range(1, n)], t) * factor
                worstd = max(worstd, abs(d / fd(c + t) - 1))
        out.append(cd + [0.0] * (n % 2))
    return out, worst, worstd


def main64():
    lines = ["// Generated by gen_smoothing_tables.py; do not edit.",
             "// FP64 smoothing tables on pieces of width 1/4 in s = (r/delta)^2: monomial coefficients in t = s - i/4.",
             "// The includer defines HR_SMOOTH_STORAGE (e.g. static __device__ const)."]
    for name, f, fd, factor, n, last in TABLES64:
        tab, worst, worstd = build64(f, fd, factor, n, last)
        print(name, "value", float(worst), "derivative", float(worstd))
        lines.append("// %s: pieces 0 .. %d, %d coefficients; max relative error %.2e%s" % (
            name, len(tab) - 1, n, float(worst), ", of the scaled derivative %.2e" % float(worstd) if fd else ""))
        lines.append("#define HR_T64_%s_PIECES %d" % (name, len(tab)))
        lines.append("#define HR_T64_%s_COEF %d" % (name, n))
        lines.append("HR_SMOOTH_STORAGE double kT64%s[%d * %d] = {" % (name, len(tab), len(tab[0])))
        lines += ["    " + ", ".join(repr(v) for v in cd) + "," for cd in tab]
        lines.append("};")
    lines.append("// e^{-i/4}, i = 0 .. 256")
    lines.append("HR_SMOOTH_STORAGE double kT64Exp[257] = {")
    lines += ["    %r," % float(mp.exp(-i * W64)) for i in range(257)]
    lines.append("};")
    # e^{-t} on |t| <= 1/8 (widened as the pieces): monomial coefficients
    h, n = W64 * mp.mpf("0.502"), 10
    ts = [h * mp.cos(mp.pi * (k + mp.mpf(1) / 2) / n) for k in range(n)]
    V = mp.matrix(n, n)
    for r, t in enumerate(ts):
        for j in range(n):
            V[r, j] = t ** j
    co = mp.lu_solve(V, mp.matrix([mp.exp(-t) for t in ts]))
    lines.append("// e^{-t} for |t| <= 1/8: monomial coefficients of t^0 .. t^%d" % (n - 1))
    lines.append("#define HR_T64_EXP_COEFS %s" % ", ".join(repr(float(co[j])) for j in range(n)))
    with open(os.path.join(HERE, "hr_eval64_tables.inc"), "w") as fh:
        fh.write("\n".join(lines) + "\n")


def main():
    lines = ["// Generated by gen_smoothing_tables.py; do not edit.",
             "// Piecewise polynomials G(s), s = (r/delta)^2 in [0, 64], of the on-surface smoothing factors.",
             "// The includer defines HR_SMOOTH_STORAGE (e.g. static __device__ const)."]
    lines.append("// FP32 tables: %d pieces uniform in s (width %g), degree %d; per piece 8 floats:"
                 % (NI32, 64.0 / NI32, DEG32))
    lines.append("// centre, coefficients of t^0 .. t^%d, 0." % DEG32)
    lines.append("#define HR_SMOOTH32_PIECES %d" % NI32)
    for name, f in (("G1", G1), ("G2", G2), ("G3", G3)):
        tab, worst = build32(f)
        lines.append("// %s (FP32): max relative error of the FP32 evaluation %.2e" % (name, worst))
        print(name, "FP32 max rel err", worst)
        lines.append("HR_SMOOTH_STORAGE float kSmooth32%s[%d * 8] = {" % (name, NI32))
        for row in tab:
            lines.append("    " + ", ".join("%.9ef" % v for v in row) + ",")
        lines.append("};")
    with open(os.path.join(HERE, "hr_smoothing_tables.inc"), "w") as fh:
        fh.write("\n".join(lines) + "\n")


if __name__ == "__main__":
    main()
    main64()
