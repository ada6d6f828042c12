"""GPU: calls of several host threads on contexts of their own, at sizes whose kernels take different amounts of shared
memory: none is refused, and each gives what it gives alone."""
import threading

import numpy as np
import pytest

import beastgpu as bg

pytestmark = pytest.mark.gpu


def _together(jobs, repeat):
    """every job (a function of a context) `repeat` times on a thread and context of its own"""
    alone = []
    for f in jobs:
        c = bg.Context(0)
        alone.append(f(c))
    failed = []

    def work(f, want):
        c = bg.Context(0)
        for _ in range(repeat):
            try:
                if not np.array_equal(f(c), want):
                    failed.append("differs")
            except bg.BeastError as e:
                failed.append(str(e))

    ts = [threading.Thread(target=work, args=a) for a in zip(jobs, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, (len(failed), failed[:3])


def test_far_pairs_of_rules_of_different_size():
    X = bg.raviartthomas(bg.ellipsoid(0, (1.0, 0.8, 1.3)))
    op = bg.Maxwell3D.singlelayer(wavenumber=2.0)

    def job(outer, inner):
        qs = bg.DoubleNumWiltonSauterQStrat(outer, inner, 2, 3, 3, 3, 3, 3)
        return lambda c: bg.assemble(op, X, X, quadstrat=qs, precision=bg.FP64, ctx=c)

    _together([job(2, 3), job(6, 7), job(10, 8), job(8, 10)], 1500)


def test_fp64_solves_of_different_order():
    def job(n):
        rng = np.random.default_rng(n)
        A = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)) + 3 * n**0.5 * np.eye(n)
        b = rng.normal(size=n) + 0j
        return lambda c: bg.solve(A, b, precision=bg.FP64, ctx=c)[0]

    _together([job(70), job(640), job(150)], 60)


def test_noalloc_solves_take_turns():
    """the triangular solves without an allocation share one scratch array a GPU: contexts on threads of their own, at
    orders that end in different places of it"""
    import ctypes as C

    import torch

    def job(n):
        rng = np.random.default_rng(n)
        A = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)) + 4 * n**0.5 * np.eye(n)
        At = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        b = torch.from_numpy(rng.normal(size=n) + 0j).cuda()
        torch.cuda.synchronize()
        held = {}

        def run(c):
            if c not in held:
                F, h = At.clone(), C.c_void_p()
                torch.cuda.synchronize()
                c.check(c.lib.beast_lu_factor(c.handle, n, F.data_ptr(), n, bg.C128, C.byref(h)))
                held[c] = F, h
            x = b.clone()
            torch.cuda.synchronize()
            c.check(c.lib.beast_lu_solve_noalloc(c.handle, held[c][1], 1, x.data_ptr(), n))
            return x.cpu().numpy()

        return run

    _together([job(700), job(1100), job(300)], 40)
