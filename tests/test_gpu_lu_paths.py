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
