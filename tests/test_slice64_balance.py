"""What the sliced FP64 update adds to the digits (csrc/slice64.h), compiled for the host: the exponents that level the
columns of an operand, the magnitudes that decide which blocks need more than eight digits, the ninth digit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

SRC = r"""
#include "slice64.h"
extern "C" {
// digits of x[i] 2^-s[i] relative to their common exponent (returned)
int t_scaled(long n, const double* x, const int* s, int* d) {
  int key = slice64::KEY_ZERO;
  for (long i = 0; i < n; ++i) {
    const int k = slice64::scaled_key(x[i], -s[i]);
    key = k > key ? k : key;
  }
  const int e = slice64::key_exponent(key);
  for (long i = 0; i < n; ++i) slice64::digits(slice64::fixed55(x[i], e + s[i]), d + 8 * i);
  return e;
}
int t_balance(double x) { return slice64::balance_exponent(slice64::abs_hi(x)); }
float t_spread(double x, double y, int e) {
  return slice64::spread_magnitude(slice64::fixed62(x, e), slice64::fixed62(y, e), x == 0.0 && y == 0.0);
}
int t_small(double x, double y, int e) { return slice64::spread_small(x, y, e, 10); }
void t_nine(long n, const double* x, int e, int* d) {
  for (long i = 0; i < n; ++i) slice64::digits9(slice64::fixed62(x[i], e), d + 9 * i);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("slice64_balance")
    src = d / "t.cpp"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "beast.jl_gb300", "csrc")
    so = d / "t.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", inc, str(src), "-o", str(so)], check=True)
    h = C.CDLL(str(so))
    h.t_balance.argtypes = [C.c_double]
    h.t_small.argtypes = [C.c_double, C.c_double, C.c_int]
    h.t_spread.restype, h.t_spread.argtypes = C.c_float, [C.c_double, C.c_double, C.c_int]
    return h


def _scaled(lib, x, s):
    x, s = np.ascontiguousarray(x), np.ascontiguousarray(s, dtype=np.int32)
    d = np.zeros((len(x), 8), dtype=np.int32)
    e = lib.t_scaled(C.c_long(len(x)), x.ctypes.data_as(C.c_void_p), s.ctypes.data_as(C.c_void_p), d.ctypes.data_as(C.c_void_p))
    return e, [sum(int(v) << (7 * (7 - i)) for i, v in enumerate(row)) for row in d], np.abs(d).max()


@pytest.mark.parametrize("spread", [0, 60, 900])
def test_balanced_digits_of_differently_scaled_columns(lib, spread):
    """a row whose entries have the columns' scales 2^s taken out: every digit string is its own value to 2^-56 of
    the largest scaled one"""
    from fractions import Fraction
    rng = np.random.default_rng(spread)
    s = rng.integers(-spread, spread + 1, size=200)
    x = rng.normal(size=200) * 2.0 ** s.astype(float)
    x[5] = 0.0
    e, X, dmax = _scaled(lib, x, s)
    assert dmax <= 64
    y = [Fraction(float(v)) / Fraction(2) ** int(k) for v, k in zip(x, s)]
    big = max(abs(v) for v in y)
    assert Fraction(2) ** (e - 1) <= big < Fraction(2) ** e
    for v, k in zip(y, X):
        assert abs(v / Fraction(2) ** e - Fraction(k, 2 ** 55)) <= Fraction(1, 2 ** 56)


def test_exponents_at_the_ends_of_the_range(lib):
    assert lib.t_balance(0.75) == 0 and lib.t_balance(1.0) == 1
    assert lib.t_balance(float("inf")) == 0 and lib.t_balance(float("nan")) == 0
    assert _scaled(lib, np.zeros(3), np.zeros(3))[0] == -1021
    assert _scaled(lib, np.array([0.0, np.nan]), np.array([3, -3]))[0] == 1 << 20
    # a subnormal beside zeros, its column's scale taken out: below 2^e
    e, X, dmax = _scaled(lib, np.array([0.0, 5e-324, 2.0]), np.array([0, -1021, 1000]))
    assert dmax <= 64 and X[1] < 2 ** 55 and e >= -52


def test_magnitudes(lib):
    """within 2^-29 of max(|x|, |y|) / 2^e, but 2^-24 at least; exactly zero for a zero alone"""
    for x, y in ((0.7, -0.9), (0.0, 1e-3), (-3e-5, 0.0)):
        assert abs(lib.t_spread(x, y, 0) - max(abs(x), abs(y))) <= 2.0 ** -29 + 2.0 ** -24 * max(abs(x), abs(y))
    assert lib.t_spread(0.0, 0.0, 0) == 0.0
    assert lib.t_spread(1e-300, 0.0, 0) == 2.0 ** -24 and lib.t_spread(0.0, 2.0 ** -40, 0) == 2.0 ** -24


def test_balanced_update_of_scaled_rows(lib):
    """sum over k of a_ik b_kj with a_ik ~ d_i / d_k and b_kj ~ d_k (half the d 2^-27): from the balanced digits the
    error is that of a 64-bit sum, from digits of the entries as they are it is a million times that"""
    rng = np.random.default_rng(4)
    K, d = 64, np.where(np.arange(64) < 32, 1.0, 2.0 ** -27)
    a = rng.uniform(0.5, 1.0, K) * rng.choice([-1, 1], K) * d[-1] / d  # a row of the small kind
    b = rng.uniform(0.5, 1.0, K) * rng.choice([-1, 1], K) * d
    s = np.array([lib.t_balance(v) for v in a], dtype=np.int32)
    from fractions import Fraction
    exact = sum(Fraction(float(u)) * Fraction(float(v)) for u, v in zip(a, b))
    err = []
    for k in (s, np.zeros(K, dtype=np.int32)):
        ea, A, _ = _scaled(lib, a, k)
        eb, B, _ = _scaled(lib, b, -k)
        p = sum(u * v for u, v in zip(A, B)) * Fraction(2) ** (ea + eb - 110)
        err.append(float(abs(p - exact) / Fraction(d[-1])))
    assert err[0] <= K * 2.0 ** -53 and err[1] >= 1e6 * err[0]


def test_small_entries(lib):
    """max(|x|, |y|) below 2^-10 of 2^e: zeros and subnormals of any ordinary scale are, infinities are not"""
    for e in (0, 7, -300):
        t = 2.0 ** (e - 10)
        assert lib.t_small(0.99 * t, 0.0, e) and lib.t_small(0.0, -0.99 * t, e) and lib.t_small(0.0, 0.0, e)
        assert not lib.t_small(t, 0.0, e) and not lib.t_small(0.0, -1.5 * t, e)
        assert lib.t_small(5e-324, 0.0, e) and not lib.t_small(float("inf"), 0.0, e)


def test_nine_digits_hold_the_value(lib):
    """the digits of the wider form: all of a value to 2^-63 of its row's largest, each at most 64"""
    from fractions import Fraction
    rng = np.random.default_rng(11)
    x = np.concatenate([[0.0, 1.0 - 2.0**-53, -(1.0 - 2.0**-53), 2.0**-70], rng.uniform(-1, 1, 500) * 2.0 ** -rng.integers(0, 60, 500)])
    d = np.zeros((len(x), 9), dtype=np.int32)
    lib.t_nine(C.c_long(len(x)), x.ctypes.data_as(C.c_void_p), 0, d.ctypes.data_as(C.c_void_p))
    assert np.abs(d).max() <= 64
    for v, row in zip(x, d):
        X = sum(int(k) << (7 * (8 - i)) for i, k in enumerate(row))
        assert abs(Fraction(float(v)) - Fraction(X, 2**62)) <= Fraction(1, 2**63)
