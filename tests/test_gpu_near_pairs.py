"""GPU: the pair kernels where their routes part -- singularity-extraction pairs several per warp, the
FP32 far pairs of the Helmholtz single layer (packed points; odd point counts, complex and very large
wavenumbers), touching pairs summed over their radial coordinate (k rho up to 2) or node by node (above),
and the pair classification without FP64 instructions."""
import numpy as np
import pytest

import beastgpu as bg
import oracle as O

pytestmark = pytest.mark.gpu

WS = bg.DoubleNumWiltonSauterQStrat


def _mesh(level=1, seed=3):
    return bg.ellipsoid(level, (1.0, 0.8, 1.3), perturb=0.02, rng=seed)


@pytest.mark.parametrize("outer,inner", [(1, 1), (2, 3), (4, 2), (5, 5), (7, 3), (10, 6)])
@pytest.mark.parametrize("kind", ["p0", "rt"])
def test_singularity_extraction(kind, outer, inner):
    """1 to 25 outer points: 32 pairs per warp to one; the FP64 contract against the oracle, 1e-10 with a
    floor of 1e-3 of the largest entry"""
    m = _mesh()
    X = bg.lagrangecxd0(m) if kind == "p0" else bg.raviartthomas(m)
    op = (bg.Helmholtz3D if kind == "p0" else bg.Maxwell3D).singlelayer(wavenumber=0.7)
    qs = WS(2, 3, outer, inner, 3, 3, 3, 3)
    for Y in (X, X.subset(np.arange(1))):
        Z = bg.assemble(op, Y, X, quadstrat=qs, precision=bg.FP64)
        Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*qs.orders()), Y, X)
        err = np.abs(Z - Zo) / (np.abs(Zo) + 1e-3 * np.abs(Zo).max())
        assert err.max() < 1e-10


@pytest.mark.parametrize("gamma", [2j, -3j, 0.4 + 2j, 0.0, 60j, 2e4j])
@pytest.mark.parametrize("far", [(1, 1), (2, 3), (3, 5), (4, 7)])
def test_fp32_far_pairs(far, gamma):
    """a point's phase |gamma| R carries a few FP32 roundings, the rest of its term a dozen: 2^-24 (12 + 4
    |gamma| R) of the sum of the terms' sizes, which the static kernel's entry is"""
    X = bg.lagrangecxd0(_mesh(level=2))
    H, qs = bg.Helmholtz3D.singlelayer, WS(far[0], far[1], 2, 3, 4, 4, 4, 4)
    Z = bg.assemble(H(gamma=gamma), X, X, quadstrat=qs, precision=bg.MIXED)
    Zr = bg.assemble(H(gamma=gamma), X, X, quadstrat=qs, precision=bg.FP64)
    Zs = bg.assemble(H(gamma=0.0), X, X, quadstrat=qs, precision=bg.FP64).real
    assert np.all(np.abs(Z - Zr) <= 2.0**-24 * (12 + 4 * abs(gamma) * 2.7) * Zs)


@pytest.mark.parametrize("precision", [bg.MIXED, bg.FP64])
@pytest.mark.parametrize("kind", ["sl", "dlt"])
def test_batch_of_one_small_tile(kind, precision):
    """the batch's kernels against the per-mesh ones: runs of tiles that end in the middle of a mesh"""
    ms = [_mesh(level, seed) for level, seed in ((0, 1), (2, 2), (1, 3), (2, 4))]
    H = bg.Helmholtz3D
    make = H.singlelayer if kind == "sl" else H.doublelayer_transposed
    spaces, ops = [bg.lagrangecxd0(m) for m in ms], [make(gamma=g) for g in (1j, 0.3 + 2j, -4j, 0.0)]
    b = bg.Batch(ops, spaces, precision=precision, tile_m=32, tile_q=5)
    try:
        Zs = [Z.cpu().numpy() for Z in b.assemble()]
    finally:
        b.close()
    tol = 1e-13 if precision == bg.FP64 else 2.0**-21  # a few FP32 roundings of a far entry
    for op, X, Z in zip(ops, spaces, Zs):
        ref = bg.assemble(op, X, X, precision=precision)
        assert np.abs(Z - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("k", [0.0, 0.3, -2.0, 2.5, 6.0])
@pytest.mark.parametrize("orders", [(1, 1, 1), (2, 3, 5), (4, 4, 4), (7, 5, 6)])
@pytest.mark.parametrize("kind", ["p0", "rt"])
def test_radial_sums(kind, orders, k):
    """pair arithmetic's sine (1e-11) bounds a node's error; a Maxwell entry adds blocks that are up to ten
    times its size"""
    m = _mesh()
    X = bg.lagrangecxd0(m) if kind == "p0" else bg.raviartthomas(m)
    if kind == "p0":
        op = bg.Helmholtz3D.singlelayer(gamma=1j * k)
    else:
        op = bg.Maxwell3D.singlelayer(gamma=1j * k, alpha=-1.3j, beta=0.7)
    qs = WS(2, 3, 2, 3, orders[0], orders[1], orders[2], 3)
    Z = bg.assemble(op, X, X, quadstrat=qs, precision=bg.MIXED_ACCURATE)
    Zr = bg.assemble(op, X, X, quadstrat=qs, precision=bg.FP64)
    assert np.abs(Z - Zr).max() <= (1e-11 if kind == "p0" else 1e-10) * np.abs(Zr).max()


def test_classification():
    """vertices that are shared to rounding only, and meshes far from size one, are classified as before:
    the assembly scales, and does not change with the last bits of the vertices"""
    m = _mesh()
    H = bg.Helmholtz3D.singlelayer
    Z = bg.assemble(H(wavenumber=2.0), bg.lagrangecxd0(m), bg.lagrangecxd0(m), precision=bg.FP64)
    rng = np.random.default_rng(1)
    v = m.vertices[m.cells].reshape(-1, 3)
    loose = bg.Mesh(v * (1.0 + 1e-15 * rng.integers(-1, 2, v.shape)), np.arange(len(v)).reshape(-1, 3))
    X = bg.lagrangecxd0(loose)
    assert np.abs(bg.assemble(H(wavenumber=2.0), X, X, precision=bg.FP64) - Z).max() <= 1e-12 * np.abs(Z).max()
    for e in (-30, -20, 25):
        X = bg.lagrangecxd0(bg.Mesh(np.ldexp(m.vertices, e), m.cells))
        Zs = bg.assemble(H(wavenumber=np.ldexp(2.0, -e)), X, X, precision=bg.FP64)
        assert np.abs(np.ldexp(Zs.real, -3 * e) + 1j * np.ldexp(Zs.imag, -3 * e) - Z).max() <= 1e-12 * np.abs(Z).max()


@pytest.mark.parametrize("k", [0.0, 0.004, -0.5, 0.9])
@pytest.mark.parametrize("orders", [(1, 1, 1), (2, 3, 5), (11, 4, 4)])
@pytest.mark.parametrize("kind,spaces", [("mwsl", "rtrt"), ("mwdl", "rtrt"), ("sl", "p0p0"), ("sl", "p1p0"), ("dl", "p1p1"),
                                         ("dl", "p0p1"), ("dlt", "p0p0"), ("dlt", "p1p0")])
def test_radial_sums_fp64(kind, spaces, orders, k):
    """k rho below 2 on the whole mesh: the integer sums, against the oracle with the FP64 contract"""
    m = _mesh()
    make = {"p0": bg.lagrangecxd0, "p1": bg.lagrangec0d1, "rt": bg.raviartthomas}
    H, M = bg.Helmholtz3D, bg.Maxwell3D
    op = {"mwsl": lambda: M.singlelayer(gamma=1j * k, alpha=-1.3j, beta=0.7), "mwdl": lambda: M.doublelayer(gamma=1j * k),
          "sl": lambda: H.singlelayer(gamma=1j * k), "dl": lambda: H.doublelayer(gamma=1j * k),
          "dlt": lambda: H.doublelayer_transposed(gamma=1j * k)}[kind]()
    X, Y, qs = make[spaces[:2]](m), make[spaces[2:]](m), WS(2, 3, 2, 3, orders[0], orders[1], orders[2], 3)
    Z = bg.assemble(op, X, Y, quadstrat=qs, precision=bg.FP64)
    Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*qs.orders()), X, Y)
    err = np.abs(Z - Zo) / (np.abs(Zo) + 1e-3 * np.abs(Zo).max())
    assert err.max() < 1e-10


@pytest.mark.parametrize("kind", ["sl", "dl"])
def test_few_and_many_pairs(kind):
    """four warps per pair and one give the same bits (integer sums)"""
    X = bg.lagrangecxd0(_mesh(level=3))
    op = (bg.Helmholtz3D.singlelayer if kind == "sl" else bg.Helmholtz3D.doublelayer)(wavenumber=3.0)
    Z = bg.assemble(op, X, X, precision=bg.FP64)
    rows = np.arange(0, X.numfunctions(), 97)
    Zs = bg.assemble(op, X.subset(rows), X, precision=bg.FP64)
    near = np.abs(Zs) > 0.05 * np.abs(Zs).max(axis=1, keepdims=True)
    assert near.any(axis=1).all() and np.array_equal(Zs[near], Z[rows][near])


@pytest.mark.parametrize("k,tol", [(0.5, 1e-10), (2.0, 1e-10), (300.0, 1e-9), (3e4, 1e-7)])
def test_balanced_beta_term(k, tol):
    """the beta term alone: pair arithmetic (4e-12 per value and 2^-45 of the phase; an entry adds blocks up
    to ten times its size), phases below and above the packed core's 2^14"""
    X = bg.raviartthomas(_mesh())
    make = lambda g: bg.Maxwell3D.singlelayer(gamma=g, alpha=0.0, beta=1.0)
    Z = bg.assemble(make(1j * k), X, X, precision=bg.MIXED_BALANCED)
    Zr = bg.assemble(make(1j * k), X, X, precision=bg.FP64)
    scale = np.abs(bg.assemble(make(0.0), X, X, precision=bg.FP64)).max()
    assert np.abs(Z - Zr).max() <= tol * scale



def _overlap(h, order):
    """two cells with one shared vertex, the second the first scaled by one over the largest Gauss node and turned by
    h about an axis in its plane: one quadrature node finds a distance of h"""
    g = 0.5 + 0.5 * np.polynomial.legendre.leggauss(order)[0].max()
    t = np.array([[1.0, 0.2, 0.3], [0.1, 0.9, -0.4]])
    u, n = t.sum(0) / np.linalg.norm(t.sum(0)), np.cross(t[0], t[1]) / np.linalg.norm(np.cross(t[0], t[1]))
    s = t / g + h * (t @ np.cross(n, u))[:, None] * n + h * n
    return bg.Mesh(np.vstack([np.zeros(3), t, s]), np.array([[0, 1, 2], [0, 3, 4]], dtype=np.int32))


@pytest.mark.parametrize("h", [1e-2, 1e-6, 1e-9])
@pytest.mark.parametrize("kind", ["sl", "dl", "dlt"])
def test_touching_cells_on_top_of_each_other(kind, h):
    """the radially summed FP64 pairs size their integers from FP32 distances, which cells nearly on top of each other
    leave no digits of: against the oracle within the FP64 contract plus the roundings of a distance h between
    coordinates of size one, 40 u / h of the largest entry"""
    m = _overlap(h, 4)
    X = bg.lagrangecxd0(m)
    op = {"sl": bg.Helmholtz3D.singlelayer, "dl": bg.Helmholtz3D.doublelayer,
          "dlt": bg.Helmholtz3D.doublelayer_transposed}[kind](wavenumber=0.3)
    qs = bg.DoubleNumSauterQstrat(2, 3, 4, 4, 4, 4)
    Z = bg.assemble(op, X, X, quadstrat=qs, precision=bg.FP64)
    Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*qs.orders()), X, X)
    assert np.abs(Z - Zo).max() <= (1e-10 + 40 * 2.0**-53 / h) * np.abs(Zo).max()


@pytest.mark.parametrize("wavenumber", [0.4, 3.0])
def test_maxwell_double_layer_on_long_thin_cells(wavenumber):
    """a staircase of strips of length 1 and width h = 1e-3, neighbours at right angles (k rho up to 2 and above: both
    FP64 kernels of touching pairs): the kernel's 1 / |x - y|^3 meets no cancelling terms beyond the roundings of h
    itself, 40 u / h of the largest entry"""
    h = 1e-3
    yz = np.cumsum([[0, 0]] + [[h, 0], [0, h]] * 3, axis=0)
    v = np.array([[x, y, z] for y, z in yz for x in (0.0, 1.0)])
    c = [t for i in range(len(yz) - 1) for t in ([2 * i, 2 * i + 1, 2 * i + 2], [2 * i + 1, 2 * i + 3, 2 * i + 2])]
    q, _ = np.linalg.qr(np.random.default_rng(2).normal(size=(3, 3)))
    X = bg.raviartthomas(bg.Mesh(v @ q, np.array(c, dtype=np.int32)))
    op, qs = bg.Maxwell3D.doublelayer(wavenumber=wavenumber), bg.DoubleNumSauterQstrat(2, 3, 4, 4, 4, 4)
    Z = bg.assemble(op, X, X, quadstrat=qs, precision=bg.FP64)
    Zo = O.assemble(O.make_op(op.kind, op.gamma, op.alpha, op.beta), O.OrcQs(*qs.orders()), X, X)
    assert np.abs(Z - Zo).max() <= 40 * 2.0**-53 / h * np.abs(Zo).max()


def test_integer_sums_of_touching_pairs_do_not_drift():
    """touching P1 pairs are differences of integer moments, sums of thousands of truncated products: the static kernel
    against the same rule node by node in FP64 (a real part of 1e-300 takes that route), 4 u of the largest entry
    each: 1 / R, the weight and the three factors of a block"""
    X = bg.lagrangec0d1(_mesh())
    qs = WS(2, 3, 6, 7, 5, 5, 4, 3)
    Z, Zn = (bg.assemble(bg.Helmholtz3D.singlelayer(gamma=g), X, X, quadstrat=qs, precision=bg.FP64) for g in (0.0, 1e-300))
    assert np.abs(Z - Zn).max() <= 8 * 2.0**-53 * np.abs(Zn).max()
