"""The device Boys tables and the downward recursion from them against 30-digit values."""
import os
import re

import mpmath as mp
import numpy as np
import pytest

from conftest import ROOT

INC = os.path.join(ROOT, "pdynamo3_b200", "csrc", "boys_table.inc")


def load(suffix, dtype):
    text = open(INC).read()
    mmax, xmax = (int(re.search(r"#define BOYS_%s (\d+)" % k, text).group(1)) for k in ("MMAX", "XMAX"))
    inv = int(re.search(r"#define BOYS%s_INVH (\d+)" % suffix.upper(), text).group(1))
    body = re.search(r"boys_table%s\[\d+\] = \{(.*?)\};" % suffix, text, re.S).group(1)
    c = np.array([v.strip().rstrip("f") for v in body.split(",") if v.strip()], dtype=np.float64).astype(dtype)
    return c.reshape(mmax + 1, xmax * inv, -1), inv


def exact(m, x):
    if x == 0:
        return mp.mpf(1) / (2 * m + 1)
    a = m + mp.mpf(1) / 2
    return mp.gammainc(a, 0, mp.mpf(float(x))) / (2 * mp.power(mp.mpf(float(x)), a))


# the polynomial's own error (below 2e-17 and one unit of F_m(0)) and the rounding of its evaluation; each
# step of F_(m-1) = (2 x F_m + exp(-x)) / (2 m - 1) adds a unit or two
@pytest.mark.parametrize("suffix,dtype,table_units,step_units", [("", np.float64, 4, 2), ("f", np.float32, 4, 2)])
def test_tables_and_downward_recursion(suffix, dtype, table_units, step_units):
    table, inv = load(suffix, dtype)
    rng = np.random.default_rng(3)
    h = 1.0 / inv
    xs = np.concatenate([[0.0, 1e-12, h, np.nextafter(h, 0), 3 * h, 49.999], rng.uniform(0, 50, 60), 10 ** rng.uniform(-4, 1.6, 30)])
    eps = np.finfo(dtype).eps
    with mp.workdps(30):
        for x in xs.astype(dtype):
            it = int(x * dtype(inv))
            t = dtype(2 * inv) * x - dtype(2 * it + 1)  # exact but for one rounding
            for M in range(len(table)):
                F = dtype(0)
                for c in table[M, it][::-1]:
                    F = dtype(F * t + c)
                worst = table_units * eps
                for m in range(M, -1, -1):
                    ref = exact(m, x)
                    assert abs(mp.mpf(float(F)) - ref) < worst * ref, (M, m, x)
                    if m:
                        F = dtype((dtype(2) * x * F + np.exp(-x)) / dtype(2 * m - 1))
                        worst += step_units * eps


def test_limit_beyond_the_tables():
    with mp.workdps(30):
        for m in range(6):
            ref = exact(m, 50.0)
            assert abs(mp.gamma(m + 0.5) / (2 * mp.power(50, m + 0.5)) - ref) < 1e-13 * ref
