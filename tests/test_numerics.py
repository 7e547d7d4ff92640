"""The number helpers that stand for FP64 sums, divisions and roots on the GPU
(csrc/imfcs_num.cuh), compiled for the host, against exact arithmetic: no
further from the exact value than the FP64 operation they replace."""
import ctypes as C
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("num") / "numerics.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "imaging_fcs_1_52_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "numerics_host.cpp"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    d = C.c_double
    for name, args in (("num_sum2", [C.c_void_p, C.c_int]), ("num_sum3", [C.c_void_p, C.c_int]),
                       ("num_sum3_low", [C.c_void_p, C.c_void_p, C.c_int]), ("num_f2d", [C.c_float]),
                       ("num_sum3_squares", [C.c_void_p, C.c_int, C.c_int]),
                       ("num_div", [d, d, C.c_int]), ("num_rcp", [d, C.c_int]), ("num_div_by", [d, d]),
                       ("num_sqrt", [d, C.c_int])):
        getattr(L, name).argtypes, getattr(L, name).restype = args, d
    L.num_div_small_misses.restype = C.c_int
    return L


def ulps(got, exact):
    """|got - exact| in units of the last place of the FP64 value nearest to exact (a Fraction)."""
    return float(abs(Fraction(got) - exact) / Fraction(math.ulp(float(exact))))


@pytest.mark.parametrize("n", [2, 30, 200, 5000])
def test_sums_are_no_further_off_than_fp64(lib, n):
    rng = np.random.default_rng(n)
    worst3 = worst64 = worst2 = 0.0
    for k in range(60):
        # sums and totals of block statistics: one sign or both, spread magnitudes
        x = (rng.lognormal(0, 3, n) * (rng.choice([-1, 1], n) if k % 2 else 1)).astype(np.float32)
        exact = sum((Fraction(float(v)) for v in x), Fraction(0))
        run = 0.0
        for v in x:
            run += float(v)
        scale = Fraction(math.ulp(float(sum((abs(Fraction(float(v))) for v in x), Fraction(0)))))
        off = lambda s: float(abs(Fraction(s) - exact) / scale)
        worst3 = max(worst3, off(lib.num_sum3(x.ctypes.data, n)))
        worst2 = max(worst2, off(lib.num_sum2(x.ctypes.data, n)))
        worst64 = max(worst64, off(run))
        low = (x * rng.uniform(-1, 1, n) * 2.0 ** -25).astype(np.float32)
        exact += sum((Fraction(float(v)) for v in low), Fraction(0))
        worst3 = max(worst3, off(lib.num_sum3_low(x.ctypes.data, low.ctypes.data, n)))
    assert worst3 <= 0.51                       # one rounding, whatever the number of values
    assert n < 200 or worst3 <= worst64
    assert n < 200 or worst2 > 1.0              # what two terms lose


def test_squares_of_block_sums(lib):
    rng = np.random.default_rng(3)
    for k in (2, 8, 64, 1024):
        for sign in (False, True):
            x = (rng.lognormal(0, 3, 16 * k) * (rng.choice([-1, 1], 16 * k) if sign else 1)).astype(np.float32)
            b = [sum((Fraction(float(v)) for v in x[i:i + k]), Fraction(0)) for i in range(0, 16 * k, k)]
            assert ulps(lib.num_sum3_squares(x.ctypes.data, 16 * k, k), sum(v * v for v in b)) <= 0.51


def test_quotients_and_roots_are_those_of_fp64(lib):
    rng = np.random.default_rng(1)
    for _ in range(4000):
        x = float(rng.choice([-1, 1]) * rng.lognormal(0, 15))
        y = float(rng.choice([-1, 1]) * rng.lognormal(0, 15))
        for off in (-3, 0, 3):
            assert abs(Fraction(lib.num_rcp(y, off)) * Fraction(y) - 1) <= Fraction(1, 2 ** 40)
            assert ulps(lib.num_div(x, y, off), Fraction(x) / Fraction(y)) <= 0.5 + 1e-9
        n = float(rng.integers(1, 5_000_000))
        assert lib.num_div_by(x, n) == x / n
        r = abs(x)
        root = math.isqrt(int(Fraction(r) * 4 ** 600))       # floor of sqrt(r) 2^600
        for off in (-2, 0, 2):
            assert ulps(lib.num_sqrt(r, off), Fraction(root, 2 ** 600)) <= 0.5 + 1e-9


def test_values_at_the_ends_of_the_range(lib):
    inf, nan = math.inf, math.nan
    vals = [0.0, -0.0, 1.0, -3.0, 5e-324, 1e-310, 1e-200, 1e-31, 1e-29, 1e29, 1e31, 1e200, 1.7e308, inf, -inf, nan]
    same = lambda a, b: a == b or (a != a and b != b)
    with np.errstate(all="ignore"):
        for x in vals:
            for y in vals:
                assert same(lib.num_div(x, y, 0), float(np.float64(x) / np.float64(y))), (x, y)
            assert same(lib.num_sqrt(x, 0), float(np.sqrt(np.float64(x)))), x
            assert same(lib.num_sqrt(-x, 0), float(np.sqrt(np.float64(-x)))), x
        for v in [0.0, -0.0, 1.5, -1e-45, 1e-45, 1.1754942e-38, 1.1754944e-38, 3.4e38, inf, -inf, nan, 2.0 ** -140]:
            f = float(np.float32(v))
            assert same(lib.num_f2d(f), f)


def test_small_divisors_give_the_bits_of_the_division(lib):
    assert lib.num_div_small_misses() == 0       # every mantissa, 2 .. 8
