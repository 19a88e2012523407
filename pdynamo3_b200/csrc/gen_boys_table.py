"""Generate the device Boys-function table ``boys_table.inc``.

F_m(x) = integral_0^1 t^(2m) exp(-x t^2) dt, m = 0 .. MMAX, on [0, XMAX): intervals of width H, on each
the polynomial in t in [-1, 1] (t = 2 (x - x_mid) / H) through the Chebyshev nodes, monomial
coefficients c_0 .. c_(N-1) contiguous, so that one evaluation reads one aligned run of N values.
FP64: H = 1/8, 8 coefficients (one 64-byte run).  The interpolation error is below
2 (H/4)^8 / 8! max|F_m^(8)| = 4.5e-17 / (2 m + 17), i.e. below 2e-17 of F_m(0) = 1 / (2 m + 1) for m <= 5;
for larger x the derivatives fall faster than F_m.  FP32: H = 1/8, 4 coefficients (one 16-byte run), error
below 2 (H/4)^4 / 4! / (2 m + 9) = 8e-8 / (2 m + 9), below one unit in the last place of F_m(0), and below
half a unit for m <= 3.
From XMAX on, exp(-x) is below 3e-22 and F_m is Gamma(m + 1/2) / (2 x^(m + 1/2)) to double precision.

Values are taken at 40 digits with mpmath (incomplete gamma function).  Re-run:  python gen_boys_table.py
"""
import os

import mpmath as mp

mp.mp.dps = 40
MMAX = 5
XMAX = 50
TABLES = (("", "double", 8, 8, "%.17e"), ("f", "float", 8, 4, "%.9ef"))  # suffix, type, 1/H, coefficients, format


def boys(m, x):
    if x == 0:
        return mp.mpf(1) / (2 * m + 1)
    return mp.gammainc(m + mp.mpf(1) / 2, 0, x) / (2 * mp.power(x, m + mp.mpf(1) / 2))


def fit(m, x0, h, n):
    """Monomial coefficients on t in [-1, 1] of the interpolant at n Chebyshev nodes of [x0, x0 + h]."""
    t = [mp.cos(mp.pi * (mp.mpf(k) + mp.mpf(1) / 2) / n) for k in range(n)]
    A = mp.matrix(n, n)
    b = mp.matrix(n, 1)
    for r in range(n):
        b[r] = boys(m, x0 + h * (t[r] + 1) / 2)
        for c in range(n):
            A[r, c] = t[r] ** c
    return mp.lu_solve(A, b)


def main():
    out = ["/* Generated by gen_boys_table.py: piecewise polynomials of the Boys functions. */",
           "#define BOYS_MMAX %d" % MMAX, "#define BOYS_XMAX %d" % XMAX]
    for suffix, ctype, inv, n, fmt in TABLES:
        nint = XMAX * inv
        out.append("#define BOYS%s_INVH %d" % (suffix.upper(), inv))
        out.append("BOYS_TABLE_QUALIFIER %s boys_table%s[%d] = {" % (ctype, suffix, (MMAX + 1) * nint * n))
        for m in range(MMAX + 1):
            for i in range(nint):
                c = fit(m, mp.mpf(i) / inv, mp.mpf(1) / inv, n)
                out.append("  " + ", ".join(fmt % float(v) for v in c) + ",")
        out.append("};")
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "boys_table.inc")
    with open(path, "w") as f:
        f.write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()
