"""GPU: the FP64 far and Sauter-Schwab kernels where their routes differ -- wavenumber of either sign,
complex, tiny (CUDA's sine), zero and large, rules other than the default's, node counts on either
side of the one-warp / whole-CTA split, grids of few and of many CTAs -- against the CPU oracle with
the FP64 contract: 1e-10 per entry with a floor of 1e-3 of the largest entry."""
import os
import re

import numpy as np
import pytest

import beastgpu as bg
import oracle as O
from conftest import ROOT

pytestmark = pytest.mark.gpu


def _check(op, X, Y, qs):
    Z = bg.assemble(op, X, Y, quadstrat=qs, precision=bg.FP64)
    Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*qs.orders()), X, Y)
    err = np.abs(Z - Zo) / (np.abs(Zo) + 1e-3 * np.abs(Zo).max())
    assert err.max() < 1e-10


def _mesh(level=1, seed=3):
    return bg.ellipsoid(level, (1.0, 0.8, 1.3), perturb=0.02, rng=seed)


WS = bg.DoubleNumWiltonSauterQStrat
GAMMAS = [2j, -3j, 0.4 + 2j, 1.5, 1e-3j, 60j]


@pytest.mark.parametrize("gamma", GAMMAS)
@pytest.mark.parametrize("kind", ["sl", "dl", "nxdl"])
def test_maxwell(kind, gamma):
    X = bg.raviartthomas(_mesh())
    op = {"sl": bg.Maxwell3D.singlelayer, "dl": bg.Maxwell3D.doublelayer, "nxdl": bg.nxdoublelayer}[kind](gamma=gamma)
    _check(op, X, X, bg.DoubleNumQStrat(6, 7) if kind == "nxdl" else WS(2, 3, 6, 7, 5, 5, 4, 3))


@pytest.mark.parametrize("gamma", GAMMAS + [0.0])
@pytest.mark.parametrize("kind,spaces", [("sl", "p1p1"), ("dl", "p1p0"), ("dlt", "p0p1"), ("dl", "p0p0"), ("dlt", "p1p1")])
def test_helmholtz(kind, spaces, gamma):
    m = _mesh()
    s = {"p0": bg.lagrangecxd0(m), "p1": bg.lagrangec0d1(m)}
    H = bg.Helmholtz3D
    op = {"sl": H.singlelayer, "dl": H.doublelayer, "dlt": H.doublelayer_transposed}[kind](gamma=gamma)
    _check(op, s[spaces[:2]], s[spaces[2:]], WS(2, 3, 2, 3, 4, 4, 4, 4))


@pytest.mark.parametrize("qs", [WS(1, 1, 2, 3, 3, 3, 3, 3), WS(5, 4, 6, 7, 2, 2, 2, 5), WS(8, 10, 6, 7, 5, 5, 4, 4),
                                WS(2, 3, 6, 7, 5, 11, 4, 3), bg.DoubleNumSauterQstrat(3, 4, 5, 5, 4, 3),
                                bg.DoubleNumQStrat(5, 4)])  # (equal rules meet at R = 0 on a cell with itself)
def test_rules(qs):
    X = bg.raviartthomas(_mesh())
    _check(bg.Maxwell3D.singlelayer(wavenumber=2.0), X, X, qs)
    _check(bg.Maxwell3D.doublelayer(wavenumber=2.0), X, X, qs)


@pytest.mark.parametrize("test_cells,trial_cells", [(1, 80), (80, 1), (3, 77), (80, 80)])
def test_small_blocks(test_cells, trial_cells):
    """P0 functions of part of a mesh: from one pair per thread to the full tile"""
    X = bg.lagrangecxd0(_mesh())
    op = bg.Helmholtz3D.doublelayer(wavenumber=2.0)
    _check(op, X.subset(np.arange(test_cells)), X.subset(np.arange(trial_cells)), WS(2, 3, 2, 3, 4, 4, 4, 4))


def test_many_ctas():
    X = bg.lagrangecxd0(_mesh(level=4))
    op = bg.Helmholtz3D.doublelayer_transposed(wavenumber=4.0)
    Z = bg.assemble(op, X, X, precision=bg.FP64)
    rows = X.subset(np.arange(0, X.numfunctions(), 331))
    Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*bg.defaultquadstrat(op, X, X).orders()), rows, X)
    err = np.abs(Z[::331] - Zo) / (np.abs(Zo) + 1e-3 * np.abs(Zo).max())
    assert err.max() < 1e-10


def _farfield_sum(X, u, d, gamma):
    """the far field as a plain sum over the package's own rule points (the oracle's rule of degree 10
    agrees with them to about 1e-13, which 80 radians per unit length magnify)"""
    with open(os.path.join(ROOT, "beast.jl_gb300", "csrc", "rules_gen.h")) as fh:
        rows = re.findall(r"\{([-0-9.e]+), ([-0-9.e]+), ([-0-9.e]+)\}", fh.read())
    q = np.array([[float(x) for x in r] for r in rows[88:113]])
    v, area = X.mesh.vertices[X.mesh.cells], X.mesh.areas()
    x = np.einsum("qk,ckx->cqx", np.column_stack([q[:, :2], 1 - q[:, 0] - q[:, 1]]), v)
    J = np.zeros(x.shape, dtype=complex)
    for i, fn in enumerate(X.fns):
        for c, r, w in fn:
            J[c] += u[i] * w * (x[c] - v[c, r]) / (2 * area[c])
    F = np.array([np.einsum("q,c,cq,cqx->x", q[:, 2], area, np.exp(gamma * (x @ y)), J) for y in d])
    return np.cross(np.cross(d, F), d)


@pytest.mark.parametrize("gamma", [2j, -3j, 0.4 + 2j, 0.5, 80j, 1e-4j])
@pytest.mark.parametrize("level,npts", [(0, 1), (2, 7), (3, 130)])
def test_farfield(level, npts, gamma):
    """one cell chunk and several, the last one partial; directions that are not unit vectors too"""
    X = bg.raviartthomas(_mesh(level))
    rng = np.random.default_rng(level)
    u = rng.normal(size=X.numfunctions()) + 1j * rng.normal(size=X.numfunctions())
    d = rng.normal(size=(npts, 3))
    d[::2] /= np.linalg.norm(d[::2], axis=1, keepdims=True)
    ff = bg.farfield(X, u, d, gamma)
    fo = _farfield_sum(X, u, d, gamma)
    assert np.abs(ff - fo).max() <= 1e-12 * np.abs(fo).max()


def test_farfield_of_many_directions():
    """more directions than a grid's second dimension: those of a long list are bit for bit those of a short one"""
    X = bg.raviartthomas(bg.ellipsoid(0, (1.0, 0.8, 1.3)))
    rng = np.random.default_rng(0)
    u = rng.normal(size=X.numfunctions()) + 1j * rng.normal(size=X.numfunctions())
    d = rng.normal(size=(131073, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    ff = bg.farfield(X, u, d, 2j)
    pick = [0, 1, 65534, 65535, 65536, 131069, 131070, 131071, 131072]
    assert np.array_equal(ff[pick], bg.farfield(X, u, d[pick], 2j))
