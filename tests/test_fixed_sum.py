"""The arithmetic of the solvers' fixed-point sums, compiled for the host
(tests/c/fixed_sum.cpp), against exact rational sums.  A float-float sum that is
given is right to 2^-46 of itself, an FP64 one to its last two bits, whatever
the last sum (the window) was; where it cannot be, it is refused and the
caller sums another way."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed_sum") / "fixed_sum.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "nbots_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "fixed_sum.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.sum_ff.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_float, C.c_void_p]
    lib.sum_f64.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_void_p]
    return lib


def sum_ff(lib, v, last):
    hi = v.astype(np.float32)
    lo = (v - hi.astype(np.float64)).astype(np.float32)
    out = np.zeros(2, np.float32)
    bad = lib.sum_ff(len(v), hi.ctypes.data, lo.ctypes.data, last, out.ctypes.data)
    exact = sum((Fraction(float(a)) + Fraction(float(b)) for a, b in zip(hi, lo)), Fraction(0))
    return bad, Fraction(float(out[0])) + Fraction(float(out[1])) if not bad else None, exact


def sum_f64(lib, v, last):
    v = np.ascontiguousarray(v)
    out = C.c_double()
    bad = lib.sum_f64(len(v), v.ctypes.data, last, C.byref(out))
    return bad, Fraction(out.value) if not bad else None, sum(map(Fraction, v), Fraction(0))


# exponents of the last sum, and how far the next one is from it
@pytest.mark.parametrize("n", [1, 7, 1000])
@pytest.mark.parametrize("drop", [-17, 0, 3, 20])
@pytest.mark.parametrize("ex", [-60, -20, 0, 60])
def test_sums_are_right(lib, ex, drop, n):
    rng = np.random.default_rng(abs(1000 * ex + 10 * drop + n))
    v = np.ldexp(rng.uniform(0.5, 1.0, n) / n, ex - drop)
    bad, got, exact = sum_ff(lib, v, 2.0 ** ex)
    assert not bad and abs(got - exact) <= exact * Fraction(1, 2 ** 46)
    bad, got, exact = sum_f64(lib, v, 2.0 ** ex)
    assert not bad and abs(got - exact) <= exact * Fraction(1, 2 ** 52)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 2.0 ** 21])
def test_values_outside_the_window_are_refused(lib, bad):
    v = np.array([0.25, bad, 0.25])
    hi, lo, out = v.astype(np.float32), np.zeros(3, np.float32), np.zeros(2, np.float32)
    assert lib.sum_ff(3, hi.ctypes.data, lo.ctypes.data, 1.0, out.ctypes.data) == 1
    d = C.c_double()
    assert lib.sum_f64(3, v.ctypes.data, 1.0, C.byref(d)) == 1


# a last value down to the window's lower end, the next sum far below it: read
# out as float-float, 2^-97 is the least (test_sums_are_right has the rest)
@pytest.mark.parametrize("drop", range(12, 32))
@pytest.mark.parametrize("ex", [-82, -81, -80, -79, -78, -75, -70, -67, -66, -65, -60])
def test_float_float_sums_at_the_lower_end(lib, ex, drop):
    rng = np.random.default_rng(1000 - 40 * ex + drop)
    for sign in (1.0, -1.0):
        v = sign * np.ldexp(rng.uniform(0.5, 1.0, 3) / 3, ex - drop)
        bad, got, exact = sum_ff(lib, v, 2.0 ** ex)
        assert bad or abs(got - exact) <= abs(exact) * Fraction(1, 2 ** 46)
        if ex >= -80 and ex - drop >= -95 and drop <= 20:
            assert not bad


# 100,000 equal addends just below half a unit (2^-80 of the last sum) above a
# whole one: every one is rounded the same way.  What is given is within the bound
# of a sum by FP64 adds, (n - 1) 2^-53 of itself.
@pytest.mark.parametrize("drop", range(20, 32))
def test_sums_that_fall_far_keep_fp64_accuracy(lib, drop):
    n = 100_000
    k = 2 ** (80 - drop) // n
    v = np.full(n, (k + 0.49) * 2.0 ** -80)
    bad, got, exact = sum_f64(lib, v, 1.0)
    assert bad or abs(got - exact) <= exact * Fraction(n - 1, 2 ** 53)
    assert not bad or drop > 23


def test_every_grid_counts_itself(lib):
    lib.grid_counts.argtypes = [C.c_uint, C.c_ulonglong]
    for blocks in (1, 2, 152, 254, 255, 256, 257, 304, 511, 512, 608):
        for before in (0, 200 << 56, 255 << 56 | 12345):
            assert lib.grid_counts(blocks, before)
