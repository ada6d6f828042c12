"""The FP64 Green's function pieces of csrc/green64.h (1/R, R, cos kR, sin kR with most of the work on
FP32 pairs and integers), compiled for the host, against 40-digit values."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

mpmath = pytest.importorskip("mpmath")
CSRC = os.path.join(ROOT, "beast.jl_gb300", "csrc")

HARNESS = r"""
#include "green64.h"
static g64::Entry tab[g64::TABLE];
extern "C" {
void t_init() {
  for (int i = 0; i < g64::TABLE; ++i) {
    const double x = g64::sin_table_host[i];
    const float h = (float)x;
    tab[i] = g64::Entry{x, h, (float)(x - (double)h)};
  }
}
void t_eval(long n, const double* R2, double k, double* out) {
  const g64::Wave w = g64::make_wave(k);
  for (long i = 0; i < n; ++i) {
    const g64::Value v = g64::eval(R2[i], w, tab);
    out[4 * i] = v.iR; out[4 * i + 1] = v.R; out[4 * i + 2] = v.c; out[4 * i + 3] = v.s;
  }
}
void t_turn(long n, const double* phi, double* out) {
  for (long i = 0; i < n; ++i) g64::turn(phi[i], 0.f, tab, out[2 * i], out[2 * i + 1]);
}
void t_turn_signed(long n, const double* phi, double* out) {
  for (long i = 0; i < n; ++i) g64::turn_signed(phi[i], 0.f, tab, out[2 * i], out[2 * i + 1]);
}
void t_fixed(long n, const double* R2, double k, double* out, int* ok) {
  static g64::EntryX tx[g64::TABLE];
  for (int i = 0; i < g64::TABLE; ++i) tx[i] = g64::to_entryx(g64::sin_table_host[i]);
  const g64::Wave w = g64::make_wave(k);
  for (long i = 0; i < n; ++i) {
    g64::ValueX v{0.0, 0, 0};
    ok[i] = g64::eval_fixed(R2[i], w, tx, v);
    out[3 * i] = v.iR; out[3 * i + 1] = (double)v.c / 4611686018427387904.0; out[3 * i + 2] = (double)v.s / 4611686018427387904.0;
  }
}
int64_t t_to_fixed(double x, int e) { return g64::to_fixed(x, e); }
double t_from_fixed(int64_t x, int e) { return g64::from_fixed(x, e); }
double t_pair(float h, float l) { return g64::pair_to_double(h, l); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("green64")
    src, so = d / "h.cpp", d / "h.so"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)])
    L = C.CDLL(str(so))
    L.t_pair.restype, L.t_pair.argtypes = C.c_double, [C.c_float, C.c_float]
    L.t_to_fixed.restype, L.t_from_fixed.restype = C.c_int64, C.c_double
    L.t_init()
    return L


def _eval(lib, R2, k):
    out = np.zeros((len(R2), 4))
    lib.t_eval(C.c_long(len(R2)), R2.ctypes.data_as(C.c_void_p), C.c_double(k), out.ctypes.data_as(C.c_void_p))
    return out


@pytest.mark.parametrize("k", [0.0, 1e-3, 0.7, -3.0, 40.0, 1e4])
def test_values(lib, k):
    """1/R and R to 1 ulp; cos and sin to 2^-52 plus the rounding of the argument (half an ulp of kR)"""
    rng = np.random.default_rng(1)
    R2 = np.concatenate([10.0 ** rng.uniform(-6, 2, size=300), [1.0, 0.25, 4.0, 2.0 ** -100, 2.0 ** 89, 1e-40, 1e40]])
    v = _eval(lib, R2, k)
    mpmath.mp.dps = 40
    for r2, (iR, R, c, s) in zip(R2, v):
        r = mpmath.sqrt(mpmath.mpf(float(r2)))
        assert abs(iR * r - 1) <= 2.0 ** -52 and abs(R / r - 1) <= 2.0 ** -52
        th = mpmath.mpf(abs(k)) * mpmath.mpf(float(R))
        tol = 2.0 ** -52 + float(th) * 2.0 ** -53
        assert abs(c - mpmath.cos(th)) <= tol and abs(s - mpmath.sin(th)) <= tol


def test_turn(lib):
    """steps of 2 pi / 4096 near the table's points, halfway between them and over the whole range"""
    rng = np.random.default_rng(2)
    n = rng.integers(64, 2 ** 29, size=400).astype(float)
    phi = np.concatenate([n, n + 0.5, n + 2.0 ** -20, n + 0.5 - 2.0 ** -22, rng.uniform(64, 5000, size=400),
                          [64.0, 1023.5, 1024.0, 2.0 ** 30 - 1]])
    out = np.zeros((len(phi), 2))
    lib.t_turn(C.c_long(len(phi)), phi.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    mpmath.mp.dps = 40
    for p, (c, s) in zip(phi, out):
        th = mpmath.mpf(float(p)) * mpmath.pi / 2048
        assert abs(c - mpmath.cos(th)) <= 2.0 ** -52 and abs(s - mpmath.sin(th)) <= 2.0 ** -52


def test_pair_to_double(lib):
    rng = np.random.default_rng(3)
    for _ in range(500):
        h = np.float32(rng.normal() * 2.0 ** rng.integers(-20, 20))
        l = np.float32(h * rng.uniform(-1, 1) * 2.0 ** -24)
        exact = float(h) + float(l)
        assert abs(lib.t_pair(h, l) - exact) <= abs(exact) * 2.0 ** -53
    for h in (1.0, -1.0, 0.5, 2.0 ** -30):  # a low part that reaches below a power of two
        l = -h * 2.0 ** -26
        assert lib.t_pair(h, l) == h + l
    assert lib.t_pair(0.0, 0.0) == 0.0


def test_turn_signed(lib):
    """any angle below 2^30 steps, of either sign, absolutely"""
    rng = np.random.default_rng(4)
    phi = np.concatenate([rng.uniform(-3000, 3000, size=600), rng.uniform(-1, 1, size=200), [0.0, 0.5, -0.5, 1.0, -1.5, 1e-30, 2.0 ** 30 - 1],
                          2.0 ** rng.uniform(-70, 29, size=200)])
    out = np.zeros((len(phi), 2))
    lib.t_turn_signed(C.c_long(len(phi)), phi.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    mpmath.mp.dps = 40
    for p, (c, s) in zip(phi, out):
        th = mpmath.mpf(float(p)) * mpmath.pi / 2048
        assert abs(c - mpmath.cos(th)) <= 2.0 ** -52 and abs(s - mpmath.sin(th)) <= 2.0 ** -52


@pytest.mark.parametrize("k", [0.7, 40.0, 1e4])
def test_fixed_point_values(lib, k):
    """cos and sin as 62-bit integers to 2^-52 plus the rounding of the argument; out of range below
    four steps and above 2^30"""
    rng = np.random.default_rng(6)
    R2 = 10.0 ** rng.uniform(-6, 2, size=400)
    out, ok = np.zeros((len(R2), 3)), np.zeros(len(R2), dtype=np.int32)
    lib.t_fixed(C.c_long(len(R2)), R2.ctypes.data_as(C.c_void_p), C.c_double(k), out.ctypes.data_as(C.c_void_p),
                ok.ctypes.data_as(C.c_void_p))
    mpmath.mp.dps = 40
    for r2, (iR, c, s), good in zip(R2, out, ok):
        th = mpmath.sqrt(mpmath.mpf(float(r2))) * k
        assert bool(good) == (4 <= th * 2048 / mpmath.pi < 2 ** 30)
        if good:
            tol = 2.0 ** -52 + float(th) * 2.0 ** -52
            assert abs(c - mpmath.cos(th)) <= tol and abs(s - mpmath.sin(th)) <= tol


def test_fixed_point_conversions(lib):
    rng = np.random.default_rng(7)
    x = rng.uniform(-1, 1, size=2000) * 2.0 ** rng.integers(-70, 1, size=2000)
    x[:4] = [0.0, 0.5, -0.5, 1.0 - 2.0 ** -53]
    for v in x:
        for e in (0, 3):
            f = lib.t_to_fixed(C.c_double(v), e)
            assert abs(f * 2.0 ** (e - 62) - v) < 2.0 ** (e - 62) + abs(v) * 2.0 ** -53
            assert lib.t_from_fixed(C.c_int64(f), 0) == float(f)
    for v in [1, -1, 2 ** 53 + 1, -(2 ** 62) + 1, 2 ** 62, (1 << 63) - 1]:
        r = lib.t_from_fixed(C.c_int64(v), -10)
        assert abs(int(r * 1024) - v) * 2 ** 53 <= abs(v)
