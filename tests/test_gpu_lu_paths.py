"""GPU: the dense solves at the sizes where their kernels' routes change (odd leading dimensions,
partial blocks and tiles of the tensor-core updates)."""
import numpy as np
import pytest

import beastgpu as bg

pytestmark = pytest.mark.gpu


def _matrix(n, sym, seed, dominance=3.0):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    A = (A + A.T) / 2 ** 0.5 if sym else A
    return A + dominance * n ** 0.5 * np.eye(n)


@pytest.mark.parametrize("n,sym", [(1025, True), (1025, False), (1087, True), (2113, True), (2113, False)])
def test_mixed_solve_of_odd_order(n, sym):
    """odd orders factor a copy whose columns are padded to whole lines, so the tensor-core updates
    take them too; the refinement brings the residual to the tolerance"""
    A = _matrix(n, sym, n)
    b = np.random.default_rng(n + 1).normal(size=(n, 2)) + 0j
    ctx = bg.get_context(0)
    x, it, res = bg.solve(A, b, precision=bg.MIXED_ACCURATE, tol=1e-12, ctx=ctx)
    assert ctx.last_factor_mode() == (2 if sym else 1)
    assert res <= 1e-12
    assert np.linalg.norm(A @ x - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [65, 97, 130, 192, 577, 1089, 1345, 2113])
def test_fp64_solve_backward_error(n):
    """the FP64 solve with its updates on the tensor cores, at partial panels, tiles and blocks: a
    random matrix (rows interchanged in every panel), normwise backward error within 4 n u"""
    A = _matrix(n, False, n, dominance=0.0)
    b = np.random.default_rng(n + 1).normal(size=(n, 2)) + 0j
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    r = np.linalg.norm(A @ x - b) / (np.linalg.norm(A) * np.linalg.norm(x))
    assert r <= 4 * n * 2.0 ** -53


def test_fp64_solve_is_invariant_under_column_scaling():
    """columns scaled by powers of two between 2^-40 and 2^40: the pivots, the multipliers and the
    digits of the updates are the same, so the solution is the scaled one bit by bit"""
    n = 700
    A = _matrix(n, False, 5, dominance=0.0)
    b = np.random.default_rng(6).normal(size=n) + 0j
    s = 2.0 ** np.random.default_rng(7).integers(-40, 41, size=n)
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    y, _, _ = bg.solve(A * s[None, :], b, precision=bg.FP64)
    assert np.array_equal(y * s, x)


@pytest.mark.parametrize("n", [97, 577, 1345, 2113])
def test_fp64_solve_backward_error_of_a_64_bit_lu(n):
    """20 u: LAPACK leaves 2 to 10 u of these; one digit level less would be 300 u"""
    A = _matrix(n, False, n + 7, dominance=0.0)
    b = np.random.default_rng(n + 1).normal(size=(n, 2)) + 0j
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    assert np.linalg.norm(A @ x - b) <= 20 * 2.0 ** -53 * np.linalg.norm(A) * np.linalg.norm(x)


@pytest.mark.parametrize("n", [40, 300])
@pytest.mark.parametrize("e", [-900, -520, -512, 508, 520, 900])
def test_fp64_solve_far_from_one(n, e):
    """matrices scaled by 2^e, where the square of a pivot or its reciprocal leaves the FP64 range: the
    solution is the unscaled one's (a few roundings of the reciprocals apart, condition about 10)"""
    A = _matrix(n, False, n, dominance=2.0)
    b = np.random.default_rng(n).normal(size=n) + 0j
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    y, _, _ = bg.solve(A * 2.0 ** e, b, precision=bg.FP64)
    assert np.linalg.norm(y * 2.0 ** e - x) <= 1e-13 * np.linalg.norm(x)


def test_fp64_solve_refuses_a_pivot_without_a_reciprocal():
    A = np.diag([1.0, 2.0, 1e-309, 3.0]).astype(np.complex128)
    with pytest.raises(bg.BeastError):
        bg.solve(A, np.ones(4), precision=bg.FP64)


def _exact(A, b, scale):
    """the solution of A x = b to well below 64-bit rounding: residuals in extended precision, corrections
    from a matrix without its row scale"""
    M = np.linalg.inv(A / scale[:, None])
    x = np.zeros(b.shape, dtype=np.clongdouble)
    Al, bl = A.astype(np.clongdouble), b.astype(np.clongdouble)
    for _ in range(5):
        x = x + M @ ((bl - Al @ x) / scale).astype(np.complex128)
    return x


def _row_scales(n, which, rng):
    s = np.ones(n)
    if which == "border":  # half of them, the border inside a panel
        s[n // 2 + 6:] = 2.0 ** -27
    elif which == "shuffled":
        s[rng.permutation(n)[: n // 2]] = 2.0 ** -40
    elif which == "377":  # an unscaled electric / magnetic system
        s[rng.permutation(n)[: n // 3]] = 377.0 ** -2
    else:
        s = 2.0 ** rng.integers(-40, 41, size=n)
    return s


@pytest.mark.parametrize("n", [300, 1089])
@pytest.mark.parametrize("which", ["border", "shuffled", "377", "random"])
def test_fp64_solve_of_scaled_rows(n, which):
    """rows in different units: the forward error is that of a 64-bit LU with the same pivot rule (LAPACK's,
    within a factor of 4 for the sums' other order and pivots that differ in near ties)"""
    rng = np.random.default_rng(n)
    s = _row_scales(n, which, rng)
    A = _matrix(n, False, n, dominance=2.0) * s[:, None]
    b = s * (rng.normal(size=n) + 1j * rng.normal(size=n))
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    ref = _exact(A, b, s)
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    lapack = np.linalg.norm(np.linalg.solve(A, b) - ref) / np.linalg.norm(ref)
    assert err <= 4 * lapack


@pytest.mark.parametrize("n,coupling,part", [(300, -20, 0.5), (2113, -33, 0.5), (2113, -33, 0.1)])
def test_fp64_solve_of_weakly_coupled_blocks(n, coupling, part):
    """two blocks of unknowns, numbered at random or one after the other, coupled by 2^coupling: no scaling of rows
    and columns levels that, so the updates go to the FP64 units (all tiles, or those of the border); the part of
    the solution that only the coupling excites keeps its own relative accuracy (LAPACK's, within a factor of 4)"""
    rng = np.random.default_rng(n)
    order = rng.permutation(n) if part == 0.5 else np.arange(n)
    a, c = order[: int(part * n)], order[int(part * n):]
    A = _matrix(n, False, n, dominance=2.0)
    A[np.ix_(a, c)] *= 2.0 ** coupling
    A[np.ix_(c, a)] *= 2.0 ** coupling
    b = np.zeros(n, dtype=np.complex128)
    b[c] = rng.normal(size=len(c)) + 1j * rng.normal(size=len(c))
    x, _, _ = bg.solve(A, b, precision=bg.FP64)
    ref, lap = _exact(A, b, np.ones(n)), np.linalg.solve(A, b)
    for part_ in (a, c):
        err, lapack = (np.linalg.norm(y[part_] - ref[part_]) for y in (x, lap))
        assert err <= 4 * lapack


@pytest.mark.parametrize("n,restart,dtype", [(1, 0, "c128"), (37, 5, "c128"), (63, 0, "c64"), (64, 1, "c128"), (65, 33, "c128"),
                                             (301, 0, "c64"), (1030, 7, "c128"), (2111, 0, "c128")])
def test_gmres_at_the_edges_of_its_row_blocks(n, restart, dtype):
    """orders around the 64-row blocks of the orthogonalisation, restarts down to one vector (a basis
    of four vectors a warp, partial groups): the residual of the returned solution reaches reltol"""
    A = (_matrix(n, False, n, dominance=0.0) * 0.3 / max(n, 1) ** 0.5 + 2.0 * np.eye(n)).astype(np.complex64 if dtype == "c64" else np.complex128)
    b = np.random.default_rng(n + 1).normal(size=n) + 1j * np.random.default_rng(n + 2).normal(size=n)
    x, it, res = bg.gmres(A, b, reltol=1e-11, restart=restart, maxiter=3000)
    assert it >= 1 and res <= 1e-11
    assert np.linalg.norm(A.astype(np.complex128) @ x - b) <= 2e-11 * np.linalg.norm(b)


def test_gmres_zero_right_hand_side_and_limit():
    A = _matrix(70, False, 3, dominance=0.0)
    x, it, res = bg.gmres(A, np.zeros(70), reltol=1e-10)
    assert it == 0 and np.array_equal(x, np.zeros(70))
    with pytest.raises(bg.BeastError):
        bg.gmres(A, np.ones(70), reltol=1e-14, restart=4, maxiter=6)


_GMRES_OOM = r"""
import ctypes as C, torch, beastgpu as bg
ctx = bg.get_context(0)
def used():
    v = [C.c_size_t() for _ in range(4)]
    ctx.check(ctx.lib.beast_pool_stats(ctx.handle, *[C.byref(x) for x in v]))
    return v[2].value
t = torch.zeros(64, dtype=torch.complex128, device="cuda")
_, total = torch.cuda.mem_get_info()
n = int(0.6 * total) // 1060  # the matvec's sums take 1 KiB a row, the basis of 66 vectors as much: 1.2 of the memory
before = used()
it, res = C.c_int(), C.c_double()
rc = ctx.lib.beast_gmres(ctx.handle, n, t.data_ptr(), n, bg.C128, t.data_ptr(), t.data_ptr(), bg.lib.DEVICE, 1e-8, 65,
                         65, C.byref(it), C.byref(res))
print(rc == bg.lib.ERR_OOM, used() - before)
"""


def test_gmres_out_of_memory_gives_everything_back():
    """a call that fails in the middle of its allocations (an order beyond the device's memory; nothing of it is read)
    leaves none of them behind"""
    import os
    import subprocess
    import sys
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", _GMRES_OOM], env=env, capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["True", "0"], (r.stdout, r.stderr[-2000:])


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n,col", [(300, 64), (300, 65), (300, 127), (65, 64), (130, 129)])
def test_zero_pivot_of_a_pair(n, col, symmetric, monkeypatch):
    """the diagonal block's elimination takes two pivots at a time: a zero first or second pivot, also the
    last one of a matrix, ends as it does one pivot at a time (4 x 4 tiles)"""
    import torch
    rng = np.random.default_rng(n + col)
    A = np.diag(rng.uniform(1.0, 2.0, n) + 1j * rng.uniform(-1.0, 1.0, n)).astype(np.complex64)
    A[col, col] = 0.0
    b = rng.normal(size=n) + 0j
    if not symmetric:
        A[1, 0] = 0.5
    out = []
    for tile in ("4", "2"):
        monkeypatch.setenv("BEAST_LU_DIAG_TILE", tile)
        try:
            x, it, res = bg.solve(torch.from_numpy(np.ascontiguousarray(A.T)).cuda().T, b, precision=bg.MIXED)
            out.append(("solved", x.tobytes()))
        except bg.BeastError as e:
            out.append(("refused", str(e)))
    assert out[0] == out[1]
