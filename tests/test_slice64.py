"""The digits of the sliced FP64 update (csrc/slice64.h), compiled for the host: a value scaled to its
row's largest magnitude is its eight digits to 2^-56, and the values added to the matrix are exact."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

SRC = r"""
#include "slice64.h"
extern "C" {
void t_digits(long n, const double* x, double rowmax, int* d, int* e) {
  *e = slice64::row_exponent(slice64::abs_hi(rowmax));
  for (long i = 0; i < n; ++i) slice64::digits(slice64::fixed55(x[i], *e), d + 8 * i);
}
double t_neg(float D, int sh) { return slice64::neg_scaled(D, sh); }
int t_exp(double x) { return slice64::row_exponent(slice64::abs_hi(x)); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("slice64")
    src = d / "t.cpp"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "beast.jl_gb300", "csrc")
    so = d / "t.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", inc, str(src), "-o", str(so)], check=True)
    h = C.CDLL(str(so))
    h.t_neg.restype, h.t_neg.argtypes = C.c_double, [C.c_float, C.c_int]
    h.t_exp.argtypes = [C.c_double]
    return h


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -1000, 2.0 ** 1000, 3e-310])
def test_digits_hold_the_value(lib, scale):
    rng = np.random.default_rng(1)
    x = rng.normal(size=4000) * 2.0 ** rng.integers(-70, 1, size=4000)
    x[:3] = [0.0, np.abs(x).max(), -np.abs(x).max()]
    x = x * scale
    big = float(np.abs(x).max())
    d = np.zeros((len(x), 8), dtype=np.int32)
    e = C.c_int()
    lib.t_digits(C.c_long(len(x)), x.ctypes.data_as(C.c_void_p), C.c_double(big), d.ctypes.data_as(C.c_void_p), C.byref(e))
    assert np.abs(d).max() <= 64
    assert big < 2.0 ** min(e.value, 1023) * (2.0 if e.value > 1023 else 1.0)
    # the digits as an exact integer multiple of 2^-55
    X = [sum(int(v) << (7 * (7 - i)) for i, v in enumerate(row)) for row in d]
    from fractions import Fraction
    for v, k in zip(x, X):
        err = abs(Fraction(float(v)) / Fraction(2) ** e.value - Fraction(k, 2 ** 55))
        assert err <= Fraction(1, 2 ** 56)


def test_largest_fraction_and_exponents(lib):
    x = np.array([1.0 - 2.0 ** -53, -(1.0 - 2.0 ** -53), 0.5])
    d = np.zeros((3, 8), dtype=np.int32)
    e = C.c_int()
    lib.t_digits(C.c_long(3), x.ctypes.data_as(C.c_void_p), C.c_double(x[0]), d.ctypes.data_as(C.c_void_p), C.byref(e))
    assert e.value == 0 and np.abs(d).max() <= 64
    assert lib.t_exp(1.0) == 1 and lib.t_exp(0.0) == -1021
    assert lib.t_exp(float("inf")) == lib.t_exp(float("nan")) == 1 << 20


def test_scaled_value_is_exact(lib):
    rng = np.random.default_rng(2)
    for D in [0, 1, -1, 2 ** 24, -(2 ** 24), 4095] + [int(v) for v in rng.integers(-2 ** 24, 2 ** 24, size=200)]:
        for sh in (0, -61, 37, -900, 900):
            assert lib.t_neg(float(D), sh) == -float(D) * 2.0 ** sh
    assert lib.t_neg(3.0, 1100) == -np.inf and lib.t_neg(-3.0, 1100) == np.inf
    assert lib.t_neg(0.0, 1100) == 0.0 and lib.t_neg(1.0, -1100) == 0.0
    assert np.isnan(lib.t_neg(0.0, 1 << 20)) and np.isnan(lib.t_neg(5.0, (1 << 20) - 1200))
