"""The work this framework is measured on: Galerkin assembly, dense solves and post-processing
through the public entry points of `beastgpu`, from the smallest calls to the largest.

    listed()             the cases, each a dict of plain values
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call: meshes, spaces, operators, matrices
    run(state)           one pass through the public entry points; returns its outputs
    work(case)           bytes and flops a pass cannot do without
    exact(case, seed)    the same outputs in 64-bit torch, without the package's kernels

Meshes are closed triangulated spheres and ellipsoids of 20 f^2 triangles (the icosahedron with
every edge cut into f; the icosphere level L of the package's own workloads is f = 2^L), vertices
moved radially by 1% of the edge length, so every size of the range exists, not powers of two only.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "beast.jl_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "beast.jl_gb300"))

import beastgpu as bg  # noqa: E402

_PREC = {"fp64": bg.FP64, "mixed": bg.MIXED, "accurate": bg.MIXED_ACCURATE, "balanced": bg.MIXED_BALANCED}


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---- the cases ---------------------------------------------------------------------------


def listed():
    return [
        # a few rows and columns of an EFIE matrix: what an ACA / H-matrix compressor asks for,
        # many times over; the smallest call of the assembly path
        {"name": "block-efie", "kind": "block", "f": 12, "rows": 37, "cols": 53, "prec": "fp64"},
        # solve(eq) on a small scatterer (320 triangles, 480 unknowns): assembly, excitation and
        # LU in one call, bound by latency and launches
        {"name": "job-small", "kind": "job", "f": 4, "prec": "fp64"},
        # the reference's own arithmetic: a complex FP64 EFIE matrix at an ordinary size
        {"name": "efie-fp64", "kind": "efie", "f": 13, "prec": "fp64"},
        # a large EFIE matrix in the mode the benchmark runs
        {"name": "efie-balanced", "kind": "efie", "f": 27, "prec": "balanced"},
        # the MFIE: n x K - 1/2 Id with its 12 x 13 point rules on every pair
        {"name": "mfie-fp64", "kind": "mfie", "f": 9, "prec": "fp64"},
        # acoustics: a double layer on continuous piecewise linear functions
        {"name": "helmholtz-dl-p1", "kind": "helmholtz", "op": "dl", "space": "p1", "f": 17, "prec": "fp64"},
        # Z \ b in complex FP64: LU with partial pivoting of a nonsymmetric (second-kind) matrix,
        # a few right-hand sides, as an MFIE or combined-field user runs it
        {"name": "solve-fp64", "kind": "solve", "n": 6007, "nrhs": 3, "sym": False, "prec": "fp64"},
        # Z \ b in the mixed factorisation with FP64 refinement, a complex-symmetric matrix
        {"name": "solve-mixed", "kind": "solve", "n": 9001, "nrhs": 1, "sym": True, "prec": "accurate"},
        # GMRES on a stored complex FP64 matrix
        {"name": "gmres", "kind": "gmres", "n": 7213, "sym": True},
        # the far field of a solved current in a cut of 721 directions
        {"name": "farfield", "kind": "farfield", "f": 20, "npts": 721},
        # many small Helmholtz meshes assembled in one call (shape studies, parameter sweeps)
        {"name": "batch-helmholtz", "kind": "batch", "jobs": 24, "fmin": 4, "fmax": 16, "prec": "mixed"},
        # the benchmark's own step: EFIE at 30720 unknowns, assembled, factored and refined
        {"name": "job-large", "kind": "job", "f": 32, "prec": "balanced"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "job", "efie", "mfie", "helmholtz", "solve", "gmres", "farfield", "batch"])
    c = {"kind": kind}
    if kind == "block":
        c.update(f=_log(rng, 4, 24), rows=_log(rng, 1, 400), cols=_log(rng, 1, 400), prec=rng.choice(["fp64", "accurate"]))
    elif kind == "job":
        c.update(prec=rng.choice(["fp64", "mixed", "accurate", "balanced"]))
        c.update(f=_log(rng, 3, 12) if c["prec"] == "fp64" else _log(rng, 3, 28))
    elif kind == "efie":
        c.update(f=_log(rng, 2, 26), prec=rng.choice(["fp64", "mixed", "accurate", "balanced"]))
    elif kind == "mfie":
        c.update(f=_log(rng, 2, 11), prec=rng.choice(["fp64", "mixed"]))
    elif kind == "helmholtz":
        c.update(op=rng.choice(["sl", "dl", "dlt"]), space=rng.choice(["p0", "p1"]), f=_log(rng, 3, 24), prec=rng.choice(["fp64", "accurate"]))
    elif kind == "solve":
        c.update(sym=rng.random() < 0.5, prec=rng.choice(["fp64", "accurate"]), nrhs=rng.choice([1, 1, 2, 5, 8]))
        c.update(n=_log(rng, 200, 6000) if c["prec"] == "fp64" else _log(rng, 300, 14000))
    elif kind == "gmres":
        c.update(n=_log(rng, 300, 12000), sym=rng.random() < 0.5)
    elif kind == "farfield":
        c.update(f=_log(rng, 3, 28), npts=_log(rng, 1, 1000))
    else:
        c.update(jobs=_log(rng, 3, 40), fmin=3, fmax=rng.randint(4, 16), prec=rng.choice(["mixed", "accurate"]))
    return c


# ---- meshes and spaces -------------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _sphere(f):
    """icosahedron with every edge cut into f, on the unit sphere: (vertices, cells)"""
    t = (1.0 + 5.0 ** 0.5) / 2.0
    v = np.array([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t],
                  [0, -1, -t], [0, 1, -t], [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]]) / math.hypot(1.0, t)
    d = ((v[:, None] - v[None]) ** 2).sum(-1)
    near = (d > 1e-9) & (d < 1.5 * d[d > 1e-9].min())
    faces = [(a, b, c) for a in range(12) for b in range(a + 1, 12) for c in range(b + 1, 12)
             if near[a, b] and near[b, c] and near[a, c]]
    pts, cells = [], []
    for a, b, c in faces:
        idx = {}
        for i in range(f + 1):
            for j in range(f + 1 - i):
                idx[i, j] = len(pts)
                pts.append((i * v[a] + j * v[b] + (f - i - j) * v[c]) / f)
        for i in range(f):
            for j in range(f - i):
                cells.append((idx[i, j], idx[i + 1, j], idx[i, j + 1]))
                if i + j < f - 1:
                    cells.append((idx[i + 1, j], idx[i + 1, j + 1], idx[i, j + 1]))
    p = np.array(pts)
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    _, first, inv = np.unique(np.round(p, 9), axis=0, return_index=True, return_inverse=True)
    p, cells = p[first], inv.reshape(-1)[np.array(cells)]
    q = p[cells]
    out = (np.cross(q[:, 0] - q[:, 2], q[:, 1] - q[:, 2]) * q.sum(1)).sum(1) < 0
    cells[out] = cells[out][:, [1, 0, 2]]
    return p, cells.astype(np.int32)


_MAKE = {"rt": bg.raviartthomas, "p0": bg.lagrangecxd0, "p1": bg.lagrangec0d1}


@functools.lru_cache(maxsize=64)
def _space(f, kind):
    return _MAKE[kind](bg.Mesh(*_sphere(f)))


def _mesh_space(f, kind, rng, lo=0.9, hi=1.1):
    """a perturbed ellipsoid and the space on it (the sphere's own numbering of the functions)"""
    v, cells = _sphere(f)
    v = v * np.array([rng.uniform(lo, hi) for _ in range(3)])
    h = math.sqrt(4 * math.pi / cells.shape[0] * 4 / math.sqrt(3.0))
    noise = np.random.default_rng(rng.randrange(1 << 30)).normal(0.0, 0.01 * h, size=(v.shape[0], 1))
    v = v * (1.0 + noise / np.linalg.norm(v, axis=1, keepdims=True))
    m, s = bg.Mesh(v, cells), _space(f, kind)
    return bg.spaces.Space(s.kind, m, s.fns, s.pos)


def _wavenumber(f, rng):
    """about 20 cells per wavelength at the benchmark's size (k = 10 at f = 32)"""
    return 10.0 * f / 32.0 * rng.uniform(0.8, 1.2) + 0.3


def _unit(rng):
    d = np.array([rng.gauss(0, 1) for _ in range(3)])
    return d / np.linalg.norm(d)


# ---- matrices of the solve cases: point-collocated boundary operators on a sphere ----------


def _points_matrix(n, sym, seed):
    """first kind (sym: the Helmholtz single layer, complex symmetric) or second kind (identity
    half plus the adjoint double layer) on n scattered points, stored column-major"""
    dev = _dev()
    g = torch.Generator().manual_seed(seed)
    i = torch.arange(n, dtype=torch.float64)
    z = 1 - (2 * i + 1) / n
    phi = i * (math.pi * (3 - math.sqrt(5.0)))
    x = torch.stack([torch.sqrt(1 - z * z) * torch.cos(phi), torch.sqrt(1 - z * z) * torch.sin(phi), z], 1)
    x = x * (1 + 0.2 * (torch.rand(3, generator=g, dtype=torch.float64) - 0.5))
    x = (x * (1 + 0.01 / math.sqrt(n) * torch.randn(n, 1, generator=g, dtype=torch.float64))).to(dev)
    k = (2.0 + 6.0 * float(torch.rand(1, generator=g))) * min(1.0, math.sqrt(n / 4000.0))
    w = 4 * math.pi / n
    a = torch.empty((n, n), dtype=torch.complex128, device=dev)  # row c: the matrix's column c
    for c0 in range(0, n, 1024):
        d = x[None, :, :] - x[c0:c0 + 1024, None, :]
        r = d.norm(dim=2)
        r[torch.arange(r.shape[0]), torch.arange(c0, c0 + r.shape[0])] = 1.0
        e = torch.polar(1.0 / (4 * math.pi * r), k * r)
        if not sym:
            nrm = x / x.norm(dim=1, keepdim=True)
            e = e * torch.complex(-1.0 / r, torch.full_like(r, k)) * ((d * nrm[None]).sum(2) / r)
        a[c0:c0 + 1024] = w * e
    diag = torch.arange(n, device=dev)
    a[diag, diag] = complex(0.5 * math.sqrt(w / math.pi), w * k / (4 * math.pi)) if sym else 0.5
    return a.T


def _rhs(n, nrhs, seed):
    r = np.random.default_rng(seed + 1)
    b = r.normal(size=(n, nrhs)) + 1j * r.normal(size=(n, nrhs))
    return b[:, 0] if nrhs == 1 else b


# ---- prepare and run -----------------------------------------------------------------------


def _operator(c, k):
    if c["kind"] == "mfie":
        return bg.nxdoublelayer(wavenumber=k) - 0.5 * bg.Identity()
    if c["kind"] == "helmholtz":
        H = bg.Helmholtz3D
        return {"sl": H.singlelayer, "dl": H.doublelayer, "dlt": H.doublelayer_transposed}[c["op"]](wavenumber=k)
    return bg.Maxwell3D.singlelayer(wavenumber=k)


def _problem(c, seed):
    rng = random.Random("%d %s" % (seed, sorted(c.items())))
    if c["kind"] == "batch":
        sizes = random.Random(str(sorted(c.items())))  # the meshes' sizes belong to the case
        fs = [sizes.randint(c["fmin"], c["fmax"]) for _ in range(c["jobs"] - 2)] + [c["fmin"], c["fmax"]]
        X = [_mesh_space(f, "p0", rng, 0.5, 2.0) for f in fs]
        return {"X": X, "k": [rng.uniform(0.5, 4.0) for _ in fs]}
    X = _mesh_space(c["f"], c.get("space", "rt"), rng)
    s = {"X": X, "k": _wavenumber(c["f"], rng)}
    n = X.numfunctions()
    if c["kind"] == "block":
        s["rows"] = np.array(sorted(rng.sample(range(n), min(c["rows"], n))))
        s["cols"] = np.array(sorted(rng.sample(range(n), min(c["cols"], n))))
    elif c["kind"] == "job":
        s["dir"] = _unit(rng)
        s["pol"] = np.cross(s["dir"], _unit(rng))
    elif c["kind"] == "farfield":
        r = np.random.default_rng(rng.randrange(1 << 30))
        s["u"] = r.normal(size=n) + 1j * r.normal(size=n)
        a, b = 2 * np.pi * np.arange(c["npts"]) / c["npts"], rng.uniform(0, np.pi)
        s["dirs"] = np.stack([np.cos(a) * np.cos(b), np.cos(a) * np.sin(b), np.sin(a)], 1)
    return s


def _count(c):
    """unknowns of a case that assembles one matrix"""
    f = c["f"]
    return {"rt": 30 * f * f, "p0": 20 * f * f, "p1": 10 * f * f + 2}[c.get("space", "rt")]


def prepare(case, seed):
    c = dict(case)
    c.pop("name", None)
    if c["kind"] in ("solve", "gmres"):
        n = c["n"]
        return {"c": c, "A": _points_matrix(n, c["sym"], seed), "b": _rhs(n, c.get("nrhs", 1), seed)}
    s = _problem(c, seed)
    s["c"] = c
    prec = s["prec"] = _PREC[c.get("prec", "fp64")]
    if c["kind"] == "batch":
        ops = [bg.Helmholtz3D.singlelayer(wavenumber=k) for k in s["k"]]
        s["batch"] = bg.Batch(ops, s["X"], precision=prec)
        return s
    s["op"] = _operator(c, s["k"])
    if c["kind"] == "block":
        s["block"] = bg.blockassembler(s["op"], s["X"], precision=prec)
    elif c["kind"] == "job":
        wave = bg.Maxwell3D.planewave(direction=s["dir"], polarization=s["pol"], wavenumber=s["k"])
        s["exc"] = bg.tangential_trace(wave)
    elif c["kind"] in ("efie", "mfie", "helmholtz"):
        n = s["X"].numfunctions()
        dt = torch.complex64 if prec == bg.MIXED else torch.complex128
        s["Z"] = torch.empty((n, n), dtype=dt, device="cuda").T
    return s


def run(state):
    s = state
    kind = s["c"]["kind"]
    if kind == "block":
        return s["block"](s["rows"], s["cols"])
    if kind == "job":
        return bg.solve_job(s["op"], s["X"], s["exc"], precision=s["prec"], tol=1e-12)[0]
    if kind in ("efie", "mfie", "helmholtz"):
        return bg.assemble(s["op"], s["X"], precision=s["prec"], out=s["Z"])
    if kind == "solve":
        return bg.solve(s["A"], s["b"], precision=_PREC[s["c"]["prec"]])[0]
    if kind == "gmres":
        return bg.gmres(s["A"], s["b"], reltol=1e-10)[0]
    if kind == "farfield":
        return bg.farfield(s["X"], s["u"], s["dirs"], 1j * s["k"])
    return s["batch"].assemble()


# ---- bytes and flops -----------------------------------------------------------------------


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("solve", "gmres"):
        n, r = c["n"], c.get("nrhs", 1)
        # the matrix read once, right-hand sides and solutions; LU 8/3 n^3 real operations (half
        # for a symmetric one), 8 n^2 per triangular pair.  GMRES: at least ten products
        lu = 8.0 / 3.0 * n ** 3 * (0.5 if c["sym"] else 1.0) + 8.0 * n * n * r
        return {"bytes": 16.0 * n * n * (10 if kind == "gmres" else 1) + 32.0 * n * r, "flops": lu if kind == "solve" else 80.0 * n * n}
    if kind == "batch":
        cells = [20.0 * f * f for f in range(c["fmin"], c["fmax"] + 1)]
        sq = c["jobs"] * sum(x * x for x in cells) / len(cells)
        return {"bytes": sq * (8 if c["prec"] == "mixed" else 16), "flops": 228.0 * sq}
    cells, n = 20.0 * c["f"] ** 2, float(_count(c))
    geo = cells * 72.0 + n * 40.0
    if kind == "block":
        # two cells per function
        return {"bytes": 16.0 * c["rows"] * c["cols"] + geo, "flops": 4.0 * c["rows"] * c["cols"] * 1200.0}
    if kind == "farfield":
        # 25-point rule: a phase (20 operations) and three shapes' two transverse components
        return {"bytes": geo + 16.0 * n + 72.0 * c["npts"], "flops": cells * c["npts"] * 25 * 60.0}
    # far-pair operations: 12 kernel values per pair with their products (156 for n x K)
    pair = {"efie": 1200.0, "job": 1200.0, "mfie": 29600.0}.get(kind) or {("sl", "p0"): 228.0, ("sl", "p1"): 480.0}.get((c["op"], c["space"]), 600.0)
    w = {"bytes": n * n * (8.0 if c["prec"] == "mixed" else 16.0) + geo, "flops": pair * cells * cells}
    if kind == "job":
        w["flops"] += 8.0 / 3.0 * n ** 3 * (1.0 if c["prec"] == "fp64" else 0.5)
        w["bytes"] *= 2.0  # written once, read once
    return w


# ---- the same in 64-bit torch ----------------------------------------------------------------

# symmetric triangle rules (first two barycentric coordinates, weight summing to 1):
# degrees 2 and 3 of the Strang-Fix family; degrees 6 and 7 of D. A. Dunavant, 1985
_RULE_ORBITS = {
    2: [(3, 1 / 6, None, 1 / 3)],
    3: [(1, None, None, -0.5625), (3, 0.2, None, 25 / 48)],
    6: [(3, 0.2492867451708833, None, 0.11678627572642424), (3, 0.06308901449150754, None, 0.050844906370214556),
        (6, 0.05314504984479855, 0.3103524510338049, 0.08285107561834727)],
    7: [(1, None, None, -0.1495700444679589), (3, 0.26034596607904864, None, 0.17561525743332668),
        (3, 0.06513010290221988, None, 0.053347235608843975), (6, 0.048690315425303526, 0.31286549600488267, 0.07711376089024116)],
}


def _rule(degree):
    """(barycentric points [q, 3], weights [q])"""
    pts, w = [], []
    for m, a, b, wt in _RULE_ORBITS[degree]:
        if m == 1:
            p = [(1 / 3, 1 / 3, 1 / 3)]
        elif m == 3:
            p = [(a, a, 1 - 2 * a), (a, 1 - 2 * a, a), (1 - 2 * a, a, a)]
        else:
            t = (a, b, 1 - a - b)
            p = [(t[i], t[j], t[3 - i - j]) for i in range(3) for j in range(3) if i != j]
        pts += p
        w += [wt] * len(p)
    return np.array(pts), np.array(w)


def _ss_rule(hits, n):
    """Sauter-Schwab nodes (Boundary Element Methods, 2011, chapter 5) of a pair that shares
    `hits` vertices: barycentric coordinates on both triangles, shared vertices first"""
    g, gw = np.polynomial.legendre.leggauss(n)
    g, gw = 0.5 * (g + 1), 0.5 * gw
    xi, e1, e2, e3 = (v.ravel() for v in np.meshgrid(g, g, g, g, indexing="ij"))
    w = np.einsum("a,b,c,d->abcd", gw, gw, gw, gw).ravel() * xi ** 3
    reg = []
    if hits == 1:
        reg.append((xi, xi * e1, xi * e2, xi * e2 * e3, w * e2))
    elif hits == 2:
        for s in range(3):
            p = [e1, e1 * e2, e1 * e3]
            a, b, c = [(p[0], p[1], p[2]), (p[1], p[0], p[2]), (p[1], p[2], p[0])][s]
            reg.append((xi, xi * b, xi * (1 - a), xi * (1 - a) * c, w * (1 - a) * e1 * e1))
    else:
        s, t, u = e1, e2, e3
        wt = w * s * (1 - s)
        b, c = (1 - s) * u, (1 - s) * u
        reg.append((xi, xi * b, xi * (1 - s * t), xi * (b + s * (1 - t)), wt))
        reg.append((xi, xi * (c + s * t), xi * (1 - s), xi * c, wt))
        reg.append((xi, xi * (c + s), xi * (1 - s * t), xi * c, wt))
    bary = lambda p, q: np.stack([1 - p, p - q, q], 1)  # noqa: E731
    X = [bary(r[0], r[1]) for r in reg] + [bary(r[2], r[3]) for r in reg]
    Y = [bary(r[2], r[3]) for r in reg] + [bary(r[0], r[1]) for r in reg]
    return np.concatenate(X), np.concatenate(Y), np.concatenate([r[4] for r in reg] * 2)


class _Reference:
    """one integral operator on X x X, cell pair by cell pair"""

    def __init__(self, op, X):
        dev = _dev()
        self.op, self.kind = op, X.kind
        self.v = torch.from_numpy(X.mesh.vertices[X.mesh.cells]).to(dev)  # [nc, 3, 3]
        c = torch.linalg.cross(self.v[:, 0] - self.v[:, 2], self.v[:, 1] - self.v[:, 2])
        self.area = 0.5 * c.norm(dim=1)
        self.nrm = c / (2 * self.area)[:, None]
        self.nc, self.n = self.v.shape[0], X.numfunctions()
        self.ns = 1 if X.kind == bg.P0 else 3
        e = np.array([(cc, r, i, w) for i, fn in enumerate(X.fns) for cc, r, w in fn])
        slot = torch.from_numpy((e[:, 0] * self.ns + e[:, 1]).astype(np.int64))
        self.dof = torch.zeros(self.nc * self.ns, dtype=torch.int64)
        self.sgn = torch.zeros(self.nc * self.ns, dtype=torch.float64)
        self.dof[slot] = torch.from_numpy(e[:, 2].astype(np.int64))
        self.sgn[slot] = torch.from_numpy(e[:, 3])
        self.dof, self.sgn = self.dof.to(dev), self.sgn.to(dev)
        self._touching(X.mesh.cells)

    def _touching(self, cells):
        at = {}
        for c, tri in enumerate(cells.tolist()):
            for i in tri:
                at.setdefault(i, []).append(c)
        pairs = {}
        for cs in at.values():
            for a in cs:
                for b in cs:
                    pairs[a, b] = pairs.get((a, b), 0) + 1
        p = np.array(sorted(pairs))
        self.pt, self.ps = p[:, 0], p[:, 1]
        self.hits = np.array([pairs[a, b] for a, b in p.tolist()])
        ct, cs = cells[self.pt], cells[self.ps]
        eq = ct[:, :, None] == cs[:, None, :]
        # shared vertices first, in the order in which the test cell has them, then the others
        self.ot = np.argsort(~eq.any(2), axis=1, kind="stable")
        pos = np.where(eq.any(1), eq.argmax(1), 3 + np.arange(3)[None])
        self.os = np.argsort(pos, axis=1, kind="stable")

    def _values(self, x, y, nx, ny, bx, by, vx, vy, ax, ay, w):
        """sum over the nodes of w k(x, y) on the shapes: x [..., q, 3] on cells vx, y on vy ->
        [..., ns, ns]; the cells' own arrays have the leading axes of x and y"""
        op, g = self.op, complex(self.op.gamma)
        r = x - y
        R = r.norm(dim=-1)
        G = torch.exp(-g * R) / (4 * math.pi * R) * w
        ns, kind = self.ns, op.kind
        grad = -(g + 1 / R) * G / R
        out = []
        for i in range(ns):
            for j in range(ns):
                if self.kind == bg.RT:
                    f = (x - vx[..., None, i, :]) / (2 * ax)[..., None, None]
                    h = (y - vy[..., None, j, :]) / (2 * ay)[..., None, None]
                    if kind == 1:
                        k = G * (op.alpha * (f * h).sum(-1) + op.beta / (ax * ay)[..., None])
                    else:  # n x K: f . (n x (r x h)) = (f . r)(n . h) - (f . h)(n . r)
                        nn = nx[..., None, :]
                        k = grad * ((f * r).sum(-1) * (nn * h).sum(-1) - (f * h).sum(-1) * (nn * r).sum(-1))
                else:
                    fg = bx[..., i] * by[..., j] if self.kind == bg.P1 else 1.0
                    if kind == 4:
                        k = op.alpha * G * fg
                    elif kind == 5:
                        k = -op.alpha * grad * (ny[..., None, :] * r).sum(-1) * fg
                    else:
                        k = op.alpha * grad * (nx[..., None, :] * r).sum(-1) * fg
                out.append(k.sum(-1))
        return torch.stack(out, -1).reshape(*out[0].shape, ns, ns)

    def near(self, orders):
        """touching pairs: Sauter-Schwab (face, edge, vertex orders), or the plain rule"""
        dev = self.v.device
        self.blocks = torch.zeros((len(self.hits), self.ns, self.ns), dtype=torch.complex128, device=dev)
        for hits, n in zip((3, 2, 1), orders):
            at = np.nonzero(self.hits == hits)[0]
            if hits == 3 and self.op.kind in (2, 3, 5, 6):
                continue  # every vector of the triple product lies in the plane
            X, Y, w = (torch.from_numpy(a).to(dev) for a in _ss_rule(hits, n))
            for c0 in range(0, len(at), max(1, 2000000 // len(w))):
                a = at[c0:c0 + max(1, 2000000 // len(w))]
                t, s = (torch.from_numpy(p[a].astype(np.int64)).to(dev) for p in (self.pt, self.ps))
                ot, os_ = (torch.from_numpy(np.argsort(p[a], axis=1)).to(dev) for p in (self.ot, self.os))
                bx, by = X[:, ot].permute(1, 0, 2), Y[:, os_].permute(1, 0, 2)  # by the cells' own vertices
                x, y = bx @ self.v[t], by @ self.v[s]
                b = self._values(x, y, self.nrm[t], self.nrm[s], bx, by, self.v[t], self.v[s], self.area[t], self.area[s],
                                 w * (4 * self.area[t] * self.area[s])[:, None])
                self.blocks[torch.from_numpy(a).to(dev)] = b

    def matrix(self, far, ss, rows=None, cols=None):
        """the matrix (rows, cols: those of its functions); None if a pair that does not touch is
        so close that the default strategy extracts its singularity"""
        dev, ns, nc = self.v.device, self.ns, self.nc
        bo, wo = (torch.from_numpy(a).to(dev) for a in _rule(far[0]))
        bi, wi = (torch.from_numpy(a).to(dev) for a in _rule(far[1]))
        xs, ys = bo @ self.v, bi @ self.v
        if ss is not None:
            self.near(ss)
        out = torch.zeros((self.n, self.n if cols is None else len(cols)), dtype=torch.complex128, device=dev)
        want = np.arange(nc) if rows is None else np.unique(np.nonzero(np.isin(self.dof.cpu().numpy(), rows))[0] // ns)
        step = max(1, int(2e7 // nc))
        for c0 in range(0, len(want), step):
            tc = torch.from_numpy(want[c0:c0 + step]).to(dev)
            C = len(tc)
            z = torch.zeros((C, nc, ns, ns), dtype=torch.complex128, device=dev)
            pairs = lambda a, b: (a[tc][:, None].expand(C, nc, *a.shape[1:]), b[None].expand(C, nc, *b.shape[1:]))  # noqa: E731
            (vx, vy), (nx, ny), (ax, ay) = pairs(self.v, self.v), pairs(self.nrm, self.nrm), pairs(self.area, self.area)
            hit = torch.zeros((C, nc), dtype=torch.int64, device=dev)
            sel = np.nonzero(np.isin(self.pt, want[c0:c0 + step]))[0]
            li = torch.from_numpy(np.searchsorted(want[c0:c0 + step], self.pt[sel])).to(dev)
            lj = torch.from_numpy(self.ps[sel].astype(np.int64)).to(dev)
            hit[li, lj] = torch.from_numpy(self.hits[sel]).to(dev)
            if ss is not None:
                d2 = torch.full((C, nc), 1e300, dtype=torch.float64, device=dev)
                for i in range(3):
                    for j in range(3):
                        d2 = torch.minimum(d2, ((vx[:, :, i] - vy[:, :, j]) ** 2).sum(-1))
                if bool(((hit == 0) & (torch.maximum(d2 * abs(self.op.gamma) ** 2, d2 / (16 * ay)) < 0.04)).any()):
                    return None
                del d2
            for a in range(len(wo)):
                for b in range(len(wi)):
                    x, y = pairs(xs[:, a:a + 1], ys[:, b:b + 1])
                    bx, by = bo[a:a + 1].expand(C, nc, 1, 3), bi[b:b + 1].expand(C, nc, 1, 3)
                    z += self._values(x, y, nx, ny, bx, by, vx, vy, ax, ay, (wo[a] * wi[b] * ax * ay)[..., None])
            if ss is not None:
                z[li, lj] = self.blocks[torch.from_numpy(sel).to(dev)]
            else:
                z[hit == 3] = 0
            z = z.permute(0, 2, 1, 3).reshape(C * ns, nc * ns) * self.sgn
            if cols is None:
                m = torch.zeros((C * ns, self.n, 2), dtype=torch.float64, device=dev)
                m.index_add_(1, self.dof, torch.view_as_real(z))
            else:
                m = torch.zeros((C * ns, len(cols), 2), dtype=torch.float64, device=dev)
                place = torch.full((self.n,), -1, dtype=torch.int64, device=dev)
                place[torch.from_numpy(cols).to(dev)] = torch.arange(len(cols), device=dev)
                keep = torch.nonzero(place[self.dof] >= 0)[:, 0]
                m.index_add_(1, place[self.dof[keep]], torch.view_as_real(z[:, keep].contiguous()))
            slots = (tc[:, None] * ns + torch.arange(ns, device=dev)).reshape(-1)
            torch.view_as_real(out).index_add_(0, self.dof[slots], m * self.sgn[slots][:, None, None])
        return out if rows is None else out[torch.from_numpy(rows).to(dev)]

    def identity(self):
        b, w = (torch.from_numpy(a).to(self.v.device) for a in _rule(2))
        x = b @ self.v
        f = (x[:, :, None] - self.v[:, None]) / (2 * self.area)[:, None, None, None]  # [nc, q, 3, xyz]
        m = torch.einsum("q,cqix,cqjx,c->cij", w, f, f, self.area) * self.sgn.reshape(-1, 3, 1) * self.sgn.reshape(-1, 1, 3)
        d = self.dof.reshape(-1, 3)
        out = torch.zeros(self.n * self.n, dtype=torch.float64, device=self.v.device)
        out.index_add_(0, (d[:, :, None] * self.n + d[:, None, :]).reshape(-1), m.reshape(-1))
        return out.reshape(self.n, self.n)


def _tensor_rule(n):
    """a collapsed Gauss-Legendre rule on the triangle: barycentric points and weights (sum 1)"""
    g, gw = np.polynomial.legendre.leggauss(n)
    g, gw = 0.5 * (g + 1), 0.5 * gw
    u, v = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    w = np.outer(gw, gw).ravel() * 2 * u
    return np.stack([1 - u, u * (1 - v), u * v], 1), w


def _shape_points(ref):
    """points [nc, q, xyz], RT shape values [nc, q, 3, xyz] and weights [nc, q] of a fine rule"""
    b, w = (torch.from_numpy(a).to(ref.v.device) for a in _tensor_rule(8))
    x = b @ ref.v
    f = (x[:, :, None] - ref.v[:, None]) / (2 * ref.area)[:, None, None, None]
    return x, f, w[None] * ref.area[:, None]


def exact(case, seed):
    c = dict(case)
    c.pop("name", None)
    kind = c["kind"]
    if kind in ("solve", "gmres"):
        a, b = _points_matrix(c["n"], c["sym"], seed), torch.from_numpy(_rhs(c["n"], c.get("nrhs", 1), seed)).to(_dev())
        return torch.linalg.solve(a.contiguous(), b.reshape(c["n"], -1)).reshape(b.shape)
    s = _problem(c, seed)
    if kind == "batch":
        got = []
        for X, k in zip(s["X"], s["k"]):
            ref = _Reference(bg.Helmholtz3D.singlelayer(wavenumber=k), X)
            got.append(ref.matrix((2, 3), (4, 4, 4)))
        return got
    if kind == "mfie":
        ref = _Reference(bg.nxdoublelayer(wavenumber=s["k"]), s["X"])
        return ref.matrix((6, 7), None) - 0.5 * ref.identity()
    if kind == "farfield":
        ref = _Reference(bg.Maxwell3D.singlelayer(wavenumber=s["k"]), s["X"])
        x, f, w = _shape_points(ref)
        u = torch.from_numpy(s["u"]).to(x.device)[ref.dof] * ref.sgn
        j = torch.einsum("cqix,ci->cqx", f.to(u.dtype), u.reshape(-1, 3)) * w[..., None]
        out = []
        for d in torch.from_numpy(s["dirs"]).to(x.device):
            m = (torch.exp(1j * s["k"] * (x @ d))[..., None] * j).sum((0, 1))
            out.append(m - d * (m * d).sum())
        return torch.stack(out)
    if kind == "job" and c["f"] > 16:
        return None  # the assembly and the LU of a matrix of this size take too long
    ref = _Reference(_operator(c, s["k"]), s["X"])
    rt = kind != "helmholtz"
    z = ref.matrix((2, 3), (5, 4, 3) if rt else (4, 4, 4), s.get("rows"), s.get("cols"))
    if z is None or kind != "job":
        return z
    x, f, w = _shape_points(ref)
    d, p = (torch.from_numpy(s[q]).to(x.device) for q in ("dir", "pol"))
    loc = torch.einsum("cqix,x,cq->ci", f.to(z.dtype), p.to(z.dtype), w * torch.exp(-1j * s["k"] * (x @ d)))
    b = torch.zeros((ref.n, 2), dtype=torch.float64, device=x.device)
    b.index_add_(0, ref.dof, torch.view_as_real((loc.reshape(-1) * ref.sgn).contiguous()))
    return torch.linalg.solve(z, torch.view_as_complex(b))
