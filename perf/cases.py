"""The measured work of this library: what a user's program asks of it, by kind.

Every case goes through the Python binding of the C ABI (mesh2hrtf_gb300.capi).
A case is a dict: "kind" (which entry point), sizes, and options.

  solve     one frequency step on a resident mesh and solver (bem_solve_frequency)
  batch     several frequency steps of one head, or of many heads, together (bem_solve_batch)
  multi     several sources on one matrix (bem_solve_multi)
  project   the solved field on a further grid (bem_project)
  static    the solved field at a few new listener positions, device buffers (bem_project_static)
  server    a group of requests through the serving loop (bem_server_*)
  oneshot   a new head: mesh upload, solver, one step, everything released
  direct    the dense direct solver (bem_assemble, bem_solve_direct, bem_project)

Sizes are those of this repository's configurations: the 1280-triangle sphere,
the graded 20480-triangle head with its 1730-point grid and 0.1-20 kHz, the
perturbed ellipsoids of 2000-30000 triangles, the 69620-triangle case with 8
sources and 11950 points, half meshes with a symmetry plane, the 2400-element
direct solve.  `n` is the subdivision: 20 n^2 triangles on a geodesic mesh,
3 n^2 quadrilaterals (6 n^2 triangles) on half a cube sphere.

Results of a mixed-precision solver are kept as complex64: its matrix and its
field sums are single precision, and a program that asked for it keeps (and
NumCalc's result files print) single precision.  FP64 results stay complex128.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from mesh2hrtf_gb300 import capi, meshes

C0, RHO = 343.0, 1.21
HEAD = np.array([0.09, 0.075, 0.11])


def listed():
    return [
        # the smallest mesh users solve: a sphere check at 1 kHz; launches and latency count
        dict(name="sphere1280", kind="solve", shape="sphere", n=8, hz=1000.0, points=1000, prec="mixed"),
        # one step of the 20480-triangle head, as the drop-in executable runs them one by one
        dict(name="head20480", kind="solve", shape="head", n=32, hz=10000.0, points=1730, prec="mixed"),
        # a head that vibrates on a patch with an absorbing surface, half of it meshed with
        # quadrilaterals on a symmetry plane
        dict(name="half3072_quads", kind="solve", shape="half_quads", n=32, hz=3000.0, points=1730, prec="mixed"),
        # the plain double-precision path, as used for reference results
        dict(name="head5120_fp64", kind="solve", shape="head", n=16, hz=5000.0, points=1730, prec="fp64"),
        # throughput of one head over its frequencies: the batched steps of a project
        dict(name="head20480_batch8", kind="batch", shape="head", n=32, count=8, points=1730, copy="blr"),
        # many heads at once: a data set of uneven meshes, each at its own frequency
        dict(name="ellipsoids_batch16", kind="batch", shape="ellipsoids", n=30, count=16, points=500, copy="fp16"),
        # the largest single matrix: 8 sources on 69620 triangles, a 2-degree grid
        dict(name="large69620_rhs8", kind="multi", shape="head", n=59, hz=16000.0, count=8, points=11950),
        # a further evaluation grid on a solved head, some of it close to the surface
        dict(name="project11950", kind="project", shape="head", n=32, hz=8000.0, points=11950, near=1000),
        # a renderer asking for a few listener positions per block: the smallest call
        dict(name="static64", kind="static", shape="head", n=16, hz=4000.0, points=64),
        # requests of different sizes arriving together at the serving loop
        dict(name="server12", kind="server", shape="ellipsoids", n=24, count=12, points=1730),
        # a new head: everything from the mesh upload to the release
        dict(name="oneshot5120", kind="oneshot", shape="head", n=16, hz=6000.0, points=1730, prec="mixed"),
        # Gaussian elimination (NC.inp's ISOLVER 4)
        dict(name="direct2420", kind="direct", shape="head", n=11, hz=2000.0, points=1000, prec="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kind by weight, sizes over the kind's range (on a log scale)."""
    kind = rng.choice(["solve", "solve", "solve", "batch", "batch", "multi", "project", "static", "server",
                       "oneshot", "direct"])
    hz = round(math.exp(rng.uniform(math.log(150.0), math.log(16000.0))), 1)
    pts = _log_int(rng, 33, 8000)
    if kind == "solve":
        prec = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        shape = rng.choice(["head", "sphere", "half_quads", "half_tris"])
        top = {"head": 38, "sphere": 32, "half_quads": 48, "half_tris": 36}[shape]
        n = _log_int(rng, 5, top if prec == "mixed" else 18)
        if shape.startswith("half"):
            n += n % 2
        return dict(kind=kind, shape=shape, n=n, hz=hz, points=pts, prec=prec)
    if kind == "batch":
        shape = rng.choice(["head", "ellipsoids"])
        return dict(kind=kind, shape=shape, n=_log_int(rng, 8, 32), count=rng.randint(2, 8), points=min(pts, 2000),
                    copy=rng.choice(["blr", "fp16"]))
    if kind == "multi":
        return dict(kind=kind, shape="head", n=_log_int(rng, 8, 44), hz=hz, count=rng.randint(2, 8), points=pts)
    if kind == "project":
        return dict(kind=kind, shape=rng.choice(["head", "sphere"]), n=_log_int(rng, 8, 32), hz=hz,
                    points=_log_int(rng, 200, 12000), near=rng.choice([0, 0, 37, 500]))
    if kind == "static":
        return dict(kind=kind, shape="head", n=_log_int(rng, 5, 32), hz=hz, points=_log_int(rng, 1, 2000))
    if kind == "server":
        return dict(kind=kind, shape="ellipsoids", n=_log_int(rng, 10, 28), count=rng.randint(2, 14), points=min(pts, 2000))
    if kind == "oneshot":
        return dict(kind=kind, shape="head", n=_log_int(rng, 6, 28), hz=hz, points=pts, prec="mixed")
    return dict(kind=kind, shape="head", n=_log_int(rng, 4, 14), hz=hz, points=min(pts, 2000),
                prec=rng.choice(["mixed", "fp64"]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=32)
def _sphere(n):
    return meshes.geodesic_sphere(n, 1.0)


@functools.lru_cache(maxsize=8)
def _half(n, tris):
    v, q = meshes.sphere_sector(n, 1.0, (1,), triangles=tris)
    return v, q


def _radius(u, axes):
    return 1.0 / np.sqrt(((u / axes) ** 2).sum(axis=1))


def _shape(shape, n, rng):
    """Vertices, elements and a source point 1 mm off the surface (or away from a sphere)."""
    if shape == "sphere":
        u, f = _sphere(n)
        v = u * (0.1 * (1.0 + 0.02 * rng.uniform(-1, 1)))
        d = rng.normal(size=3)
        return v, f, d / np.linalg.norm(d)
    if shape in ("half_quads", "half_tris"):
        u, f = _half(n, shape == "half_tris")
        # even in y, so that the nodes on the plane y = 0 stay there and the whole is smooth
        a = rng.uniform(-0.06, 0.06, size=3)
        r = _radius(u, HEAD) * (1.0 + a[0] * u[:, 0] + a[1] * u[:, 1] ** 2 + a[2] * u[:, 2])
        return u * r[:, None], f, np.array([0.7, 0.4, 0.2]) + 0.1 * rng.uniform(-1, 1, size=3)
    u, f = _sphere(n)
    if shape == "ellipsoids":
        k = rng.normal(size=(24, 3)) * 2.0
        w = np.cos(u @ k.T + rng.uniform(0, 2 * np.pi, size=24)).sum(axis=1)
        v = u * (_radius(u, HEAD) + 0.003 * (w - w.mean()) / w.std())[:, None]
    else:
        # the head: vertices graded towards an ear at +y, bumps at both ears
        ears = []
        for side in (1.0, -1.0):
            d = np.array([rng.normal(0, 0.15), side, rng.normal(0, 0.15)])
            ears.append(d / np.linalg.norm(d))
        c = np.clip(u @ ears[0], -1.0, 1.0)
        th = 2.0 * np.arctan(0.577 * np.tan(0.5 * np.arccos(c)))
        e = u - c[:, None] * ears[0]
        m = np.linalg.norm(e, axis=1)
        e = e / np.where(m > 1e-12, m, 1.0)[:, None]
        g = np.cos(th)[:, None] * ears[0] + np.sin(th)[:, None] * e
        g[m <= 1e-12] = np.where(c[m <= 1e-12] > 0, 1.0, -1.0)[:, None] * ears[0]
        r = _radius(g, HEAD)
        for d in ears:
            t = np.arccos(np.clip(g @ d, -1.0, 1.0)) / rng.uniform(0.18, 0.26)
            r = r + rng.uniform(0.006, 0.010) * np.exp(-0.5 * t * t)
        v = g * r[:, None]
    t = v[f[int(rng.integers(len(f)))]]
    nrm = np.cross(t[0] - t[2], t[1] - t[2])
    nrm *= np.sign(nrm @ t.mean(axis=0)) / np.linalg.norm(nrm)
    return v, f, t.mean(axis=0) + 0.001 * nrm


def _grid(count, rng, near=0, v=None, f=None):
    """`count` points on a 1.2 m sphere, the first `near` of them 2.5 mm to 3 cm off the surface."""
    p = meshes.equal_angle_grid() if count == 1730 else meshes.fibonacci_sphere(count, 1.2)
    p = p * (1.0 + 0.01 * rng.uniform())
    if near:
        near = min(near, count)
        t = v[f[rng.integers(len(f), size=near)]]
        nrm = np.cross(t[:, 0] - t[:, 2], t[:, 1] - t[:, 2])
        nrm /= np.linalg.norm(nrm, axis=1)[:, None]
        p[:near] = t.mean(axis=1) + nrm * np.exp(rng.uniform(np.log(0.0025), np.log(0.03), size=near))[:, None]
    return p


def _problem(shape, n, hz, points, rng, near=0):
    """Everything that defines one step, as host data."""
    v, f, src = _shape(shape, n, rng)
    p = dict(v=v, f=f, k=2 * np.pi * hz / C0, sources=[src], amps=[0.1 / (1j * RHO * 2 * np.pi * hz)], planes=(0, 0, 0),
             adm=None, bcv=None, pts=_grid(points, rng, near, v, f))
    if shape.startswith("half"):
        # symmetric plane y = 0, an absorbing surface, a vibrating patch (elements near one direction)
        p["planes"] = (0, 1, 0)
        cen = v[f].mean(axis=1)
        g = np.exp(-8.0 * ((cen / np.linalg.norm(cen, axis=1)[:, None] - np.array([0.0, 1.0, 0.0])) ** 2).sum(axis=1))
        p["adm"] = 1j * p["k"] * (0.2 + 0.1j) * g
        p["bcv"] = np.zeros((len(f), 4), complex)
        p["bcv"][np.argsort(-g)[: max(4, len(f) // 64)], : f.shape[1]] = 1e-3 * (1 + 0.3j) * rng.uniform(0.5, 1.5)
    return p


def _problems(case, seed):
    """The problems of a case, one per instance."""
    rng = np.random.default_rng([seed, 77])
    kind, shape, n = case["kind"], case["shape"], case["n"]
    if kind not in ("batch", "server"):
        p = _problem(shape, n, case["hz"], case["points"], rng, case.get("near", 0))
        if kind == "multi":
            v, f = p["v"], p["f"]
            t = v[f[rng.integers(len(f), size=case["count"])]]
            nrm = np.cross(t[:, 0] - t[:, 2], t[:, 1] - t[:, 2])
            nrm /= np.linalg.norm(nrm, axis=1)[:, None]
            src = t.mean(axis=1) + 0.001 * nrm
            return [dict(p, sources=[s]) for s in src]
        return [p]
    count, out = case["count"], []
    if shape == "head":   # one head, frequencies spread over 0.1 - 20 kHz
        base = _problem(shape, n, 1000.0, case["points"], rng)
        for i in range(count):
            hz = 100.0 + 19900.0 * (i + rng.uniform()) / count
            out.append(dict(base, k=2 * np.pi * hz / C0, amps=[0.1 / (1j * RHO * 2 * np.pi * hz)]))
        return out
    for i in range(count):   # element counts log-uniform down to a tenth of the largest's
        ni = max(5, int(round(n * 10.0 ** (-0.5 * i / max(1, count - 1)))))
        out.append(_problem(shape, ni, 200.0 + 15800.0 * ((7 * i + 3) % count + rng.uniform()) / count, case["points"], rng))
    return out


def _mesh(p):
    return capi.Mesh(p["v"], p["f"], sym_planes=p["planes"])


def _freq(p):
    bct = None if p["adm"] is None else np.full(len(p["f"]), 2, np.int32)
    return capi.Frequency(p["k"], len(p["f"]), bc_type=bct, bc_value=p["bcv"], admittance=p["adm"],
                          point_sources=p["sources"], point_amps=p["amps"])


def _prec(case):
    return capi.PREC_FP64 if case.get("prec") == "fp64" else capi.PREC_MIXED


def prepare(case, seed):
    ps = _problems(case, seed)
    kind = case["kind"]
    st = {"kind": kind, "pts": [p["pts"] for p in ps], "freqs": [_freq(p) for p in ps], "fp64": case.get("prec") == "fp64"}
    if kind == "oneshot":
        st["problem"], st["prec"] = ps[0], _prec(case)
        return st
    one_mesh = kind != "server" and case["shape"] != "ellipsoids"
    st["meshes"] = [_mesh(ps[0])] if one_mesh else [_mesh(p) for p in ps]
    if kind == "server":
        need = sum(capi.footprint_bytes(len(p["f"])) + 3e7 for p in ps)
        st["server"] = capi.Server(hbm_budget=min(60e9, 1.1 * need + 1e8), tol=1e-9)
        return st
    if kind == "batch":
        copy = capi.KRYLOV_BLR if case["copy"] == "blr" else False
        ms = st["meshes"] * len(ps) if one_mesh else st["meshes"]
        st["solvers"] = [capi.Solver(m, precision=capi.PREC_MIXED, complex64_krylov=copy) for m in ms]
        return st
    st["solver"] = capi.Solver(st["meshes"][0], precision=_prec(case), n_rhs=len(ps) if kind == "multi" else 1)
    if kind in ("project", "static"):   # a solved head is what the program has in hand
        st["solver"].solve_frequency(st["freqs"][0], np.zeros((0, 3)))
    if kind == "static":
        m = case["points"]
        st["pts_dev"] = torch.from_numpy(np.ascontiguousarray(ps[0]["pts"])).cuda()
        st["pot_dev"] = torch.zeros(m, dtype=torch.complex128, device="cuda")
        st["grad_dev"] = torch.zeros(m, 3, dtype=torch.complex128, device="cuda")
    return st


def _keep(st, a):
    return a if st["fp64"] else a.astype(np.complex64)


def _out(st, xs, pots, grads):
    return {"x": [_keep(st, a) for a in xs], "pot": [_keep(st, a) for a in pots], "grad": [_keep(st, a) for a in grads]}


def run(st):
    kind = st["kind"]
    if kind == "batch":
        r = capi.solve_batch(st["solvers"], st["freqs"], st["pts"])
        return _out(st, [q[0] for q in r], [q[1] for q in r], [q[2] for q in r])
    if kind == "multi":
        xs, pots, grads, _ = st["solver"].solve_multi(st["freqs"], st["pts"][0])
        return _out(st, xs, pots, grads)
    if kind == "server":
        srv = st["server"]
        tickets = [srv.submit(m, f, p) for m, f, p in zip(st["meshes"], st["freqs"], st["pts"])]
        r = [srv.wait(t) for t in tickets]
        return _out(st, [q[0] for q in r], [q[1] for q in r], [q[2] for q in r])
    if kind == "static":
        st["solver"].project_static(len(st["pts"][0]), st["pts_dev"].data_ptr(), st["pot_dev"].data_ptr(),
                                    st["grad_dev"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"pot": [st["pot_dev"].to(torch.complex64)], "grad": [st["grad_dev"].to(torch.complex64)]}
    if kind == "project":
        pot, grad = st["solver"].project(st["pts"][0])
        return {"pot": [_keep(st, pot)], "grad": [_keep(st, grad)]}
    if kind == "oneshot":
        mesh = _mesh(st["problem"])
        s = capi.Solver(mesh, precision=st["prec"])
        x, pot, grad = s.solve_frequency(st["freqs"][0], st["pts"][0])
        s.close()
        mesh.close()
        return _out(st, [x], [pot], [grad])
    s = st["solver"]
    if kind == "direct":
        s.assemble(st["freqs"][0])
        s.solve_direct()
        x = s.solution()
        pot, grad = s.project(st["pts"][0])
    else:
        x, pot, grad = s.solve_frequency(st["freqs"][0], st["pts"][0])
    return _out(st, [x], [pot], [grad])


def _sizes(case):
    n, shape = case["n"], case["shape"]
    if shape == "ellipsoids":
        c = case["count"]
        return [20 * max(5, int(round(n * 10.0 ** (-0.5 * i / max(1, c - 1))))) ** 2 for i in range(c)]
    one = {"half_quads": 3, "half_tris": 6}.get(shape, 20) * n * n
    return [one] * (case["count"] if case["kind"] in ("batch", "multi") else 1)


def work(case):
    """Bytes: mesh, points and results once.  Operations: per element pair (and image) the 4-point
    rule at 60 operations per evaluation, 30 complex products with the matrix (8 N^2 / 3 N operations of
    an elimination for the direct solver), per (point, element) pair 4 evaluations of 80."""
    m, b, fl = case["points"], 0.0, 0.0
    kind, img = case["kind"], 2 if case["shape"].startswith("half") else 1
    for i, n in enumerate(_sizes(case)):
        fresh = not (kind == "multi" and i)
        b += (100.0 * n if fresh else 0.0) + 24.0 * m + 64.0 * m
        fl += 4.0 * 80.0 * m * n * img
        if kind in ("project", "static"):
            b += 16.0 * n
            continue
        b += 16.0 * n
        fl += (4.0 * 60.0 * n * n * img if fresh else 0.0) + (8.0 / 3.0 * n ** 3 if kind == "direct" else 30 * 8.0 * n * n)
    return {"bytes": b, "flops": fl}


# ------------------------------------------------------------------ the results in 64 bits
# The collocation method itself (Burton-Miller, constant elements, the subdivision and Gauss orders by
# distance) in plain torch: the system as a dense complex128 matrix, solved to 1e-13.
def _gl(m):
    x, w = np.polynomial.legendre.leggauss(m)
    return x, w


def _rule(nv, order):
    """Points and weights of the element rules: (points, 3) as s, t, weight."""
    if nv == 4:
        x, w = _gl(order)
        return np.array([(x[i], x[j], w[i] * w[j]) for i in range(order) for j in range(order)])

    def sym(a, w):
        return [(a, a, w), (1 - 2 * a, a, w), (a, 1 - 2 * a, w)]

    if order <= 2:   # Strang-Fix
        return np.array([(1 / 3, 1 / 3, -27 / 96)] + sym(0.2, 25 / 96))
    if order == 3:   # Radon
        r = math.sqrt(15.0)
        return np.array([(1 / 3, 1 / 3, 9 / 80)] + sym((6 - r) / 21, (155 - r) / 2400) + sym((6 + r) / 21, (155 + r) / 2400))
    a, b = 0.0486903154253, 0.3128654960049   # 13 points, degree 7
    c = 1 - a - b
    six = [(s, t, 0.0771137608903 / 2) for s, t in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b))]
    return np.array([(1 / 3, 1 / 3, -0.1495700444677 / 2)] + sym(0.2603459660790, 0.1756152574332 / 2)
                    + sym(0.0651301029022, 0.0533472356088 / 2) + six)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), dtype=dtype, device=_dev())


def _shapes(nv, s, t):
    """Shape functions and their derivatives, stacked on the last axis."""
    if nv == 3:
        o, z = torch.ones_like(s), torch.zeros_like(s)
        return torch.stack([s, t, 1 - s - t], -1), torch.stack([o, z, -o], -1), torch.stack([z, o, -o], -1)
    p, q = s + 1, t + 1
    m, n = s - 1, t - 1
    return (torch.stack([p * q, -m * q, m * n, -p * n], -1) / 4, torch.stack([q, -q, n, -n], -1) / 4,
            torch.stack([p, -m, m, -p], -1) / 4)


def _place(verts, s, t):
    """Points, unit normals and Jacobians at (s, t) of elements `verts` (..., nv, 3), s and t (..., g)."""
    sh, ds, dt = _shapes(verts.shape[-2], s, t)
    y, a, b = sh @ verts, ds @ verts, dt @ verts
    c = torch.linalg.cross(a, b)
    j = torch.linalg.norm(c, dim=-1)
    return y, c / j[..., None], j, sh


class _Exact:
    def __init__(self, p):
        self.v, self.f = _t(p["v"]), np.asarray(p["f"])
        self.nv, self.n, self.k = self.f.shape[1], len(self.f), float(p["k"])
        el = self.v[torch.as_tensor(self.f, device=_dev())]
        self.images = [(el, 1.0)]
        if p["planes"][1]:
            im = el.clone()
            im[..., 1] = -im[..., 1]
            self.images.append((im[:, [1, 0, 2] if self.nv == 3 else [1, 0, 3, 2]], 1.0))
        s0 = torch.full((self.n, 1), 1 / 3 if self.nv == 3 else 0.0, dtype=torch.float64, device=_dev())
        y, nr, j, _ = _place(el, s0, s0)
        self.cen, self.nrm, self.sqa = y[:, 0], nr[:, 0], torch.sqrt(j[:, 0] * (0.5 if self.nv == 3 else 4.0))
        self.adm = None if p["adm"] is None else _t(p["adm"], torch.complex128)
        self.bcv = None if p["bcv"] is None else _t(p["bcv"], torch.complex128)
        self.src, self.amp = _t(p["sources"]), [complex(a) for a in p["amps"]]
        self.pts, self.sym = _t(p["pts"]), bool(p["planes"][1])

    # the order accepted by the three error estimates at a distance ratio; 0: subdivide
    @staticmethod
    def order(ratio):
        d = 0.5 / ratio
        o = torch.full_like(ratio, 6.0)
        for m in (5, 4, 3, 2):
            e = 128.0 * (m + 1) * (2 * m + 1) * d ** (2 * m + 3)
            h = 64.0 * (2 * m + 1) * d ** (2 * m + 2)
            g = 32.0 * d ** (2 * m + 1)
            o = torch.where((e < 0.001) & (h < 0.001) & (g < 0.001), torch.full_like(o, float(m)), o)
        return torch.where(ratio < 1.3, torch.zeros_like(o), o).to(torch.int8)

    def integrate(self, x, el, j, fn, width):
        """Sum over the quadrature of pairs (x[i], element el[j[i]]) of fn(pair, y, ny, wj, shapes), subdivided
        towards the point; `width` complex values per pair."""
        out = torch.zeros(len(j), width, dtype=torch.complex128, device=_dev())
        nv = self.nv
        loc = [(1, 0), (0, 1), (0, 0)] if nv == 3 else [(1, 1), (-1, 1), (-1, -1), (1, -1)]
        pid = torch.arange(len(j), device=_dev())
        sub = _t(loc).expand(len(j), nv, 2)
        fac = 1.0
        for _ in range(23):
            c = sub.mean(dim=1)
            verts = el[j[pid]]
            y = (_shapes(nv, c[:, :1], c[:, 1:])[0] @ verts)[:, 0]
            ratio = torch.linalg.norm(y - x[pid], dim=1) / (self.sqa[j[pid]] * fac)
            o = self.order(ratio)
            if nv == 3:
                off = c[:, None] - sub
                jr = (off[..., 0] - off[..., 1]).abs().argmin(dim=1)
                at = torch.arange(len(jr), device=_dev())
                org, f = sub[at, jr], torch.where(off[at, jr, 0] >= 0, fac, -fac)
            else:
                org, f = c, torch.full((len(pid),), fac, dtype=torch.float64, device=_dev())
            for m in range(2, 7):
                sel = torch.nonzero(o == m)[:, 0]
                rule = _t(_rule(nv, m))
                for ch in torch.split(sel, max(1, 4000000 // len(rule))):
                    s = org[ch, 0, None] + rule[None, :, 0] * f[ch, None]
                    t = org[ch, 1, None] + rule[None, :, 1] * f[ch, None]
                    yy, nn, jj, sh = _place(verts[ch], s, t)
                    out.index_add_(0, pid[ch], fn(pid[ch], yy, nn, jj * rule[None, :, 2] * fac * fac, sh))
            sel = torch.nonzero(o == 0)[:, 0]
            if not len(sel):
                return out
            a = sub[sel]
            mid = 0.5 * (a + a.roll(-1, dims=1))
            if nv == 3:
                kids = [torch.stack([a[:, i], mid[:, i], mid[:, i - 1]], 1) for i in range(3)] + [mid]
            else:
                cc = c[sel]
                kids = [torch.stack([a[:, i], mid[:, i], cc, mid[:, i - 1]], 1) for i in range(4)]
            sub, pid, fac = torch.cat(kids), pid[sel].repeat(4), 0.5 * fac
        raise RuntimeError("point on the surface")

    def kernels(self, x, nx, y, ny, wj):
        """G, H, H^T, E at quadrature points y for collocation points x (broadcast)."""
        d = y - x
        r = torch.linalg.norm(d, dim=-1)
        g = torch.polar(wj / (4 * math.pi * r), self.k * r)
        re1, re2 = (d * ny).sum(-1) / r, -(d * nx).sum(-1) / r
        rq, nn = re1 * re2, (nx * ny).sum(-1)
        z1 = torch.complex(-1 / r, torch.full_like(r, self.k))
        e = torch.complex((3 / r ** 2 - self.k ** 2) * rq + nn / r ** 2, -self.k / r * (3 * rq + nn))
        return g, g * z1 * re1, g * z1 * re2, g * e

    def entry(self, g, h, ht, e, adm):
        beta = 1j / self.k
        z = h + e * beta
        return z if adm is None else z + (g + ht * beta) * adm

    def singular(self, rows):
        """G, H, H^T, E of the self pairs and the right-hand-side term of their own velocities."""
        el, x, nx, nv = self.images[0][0][rows], self.cen[rows], self.nrm[rows], self.nv
        k = self.k
        g3, w3 = (_t(a) for a in _gl(3))
        e = torch.zeros(len(rows), dtype=torch.complex128, device=_dev())
        for i in range(nv):
            a, b = el[:, i], el[:, (i + 1) % nv]
            dif = b - a
            ln = torch.linalg.norm(dif, dim=1)
            for sec in range(4):
                for q in range(3):
                    sg = -0.75 + 0.5 * sec + g3[q] / 4
                    d = a + dif * ((sg + 1) / 2) - x
                    r = torch.linalg.norm(d, dim=1)
                    g = torch.polar(1 / (4 * math.pi * r), k * r) * torch.complex(-1 / r, torch.full_like(r, k))
                    cr = torch.linalg.cross(d / r[:, None], dif / ln[:, None])
                    e = e + g * (cr * nx).sum(1) * (w3[q] * ln / 8)
        g4, w4 = _gl(4)
        if nv == 3:
            cs, me, area = [(1, 0), (0, 1), (0, 0)], [(0.5, 0.5), (0, 0.5), (0.5, 0)], 1 / 48
            c = (1 / 3, 1 / 3)
        else:
            cs, me, area = [(1, 1), (-1, 1), (-1, -1), (1, -1)], [(0, 1), (-1, 0), (0, -1), (1, 0)], 0.125
            c = (0.0, 0.0)
        st = []
        for i in range(nv):
            for p, q in ((cs[i], me[i]), (me[i], cs[(i + 1) % nv])):
                for a in range(4):
                    for b in range(4):
                        s, t = g4[a], g4[b]
                        st.append([0.5 * (1 - s) * c[z] + 0.25 * (1 + s) * ((1 - t) * p[z] + (1 + t) * q[z]) for z in (0, 1)]
                                  + [w4[a] * w4[b] * (1 + s) * area])
        st = _t(st)
        y, ny, jj, sh = _place(el, st[:, 0].expand(len(rows), -1), st[:, 1].expand(len(rows), -1))
        g, h, ht, _ = self.kernels(x[:, None], nx[:, None], y, ny, jj * st[:, 2])
        e = e + (g * (k * k * (nx[:, None] * ny).sum(-1))).sum(1)
        rhs = None
        if self.bcv is not None:
            rhs = ((g + ht * (1j / k)) * (sh.to(torch.complex128) @ self.bcv[rows, :nv, None])[..., 0]).sum(1)
        return g.sum(1), h.sum(1), ht.sum(1), e, rhs

    def system(self):
        n, cen, nrm, nv = self.n, self.cen, self.nrm, self.nv
        a = torch.zeros(n, n, dtype=torch.complex128, device=_dev())
        rule = _t(_rule(nv, 2))
        step = max(1, 24000000 // (n * len(rule)))
        for el, sg in self.images:
            first = el is self.images[0][0]
            y, ny, jj, _ = _place(el, rule[:, 0].expand(n, -1), rule[:, 1].expand(n, -1))
            w = jj * rule[:, 2]
            c = cen if first else torch.stack([cen[:, 0], -cen[:, 1], cen[:, 2]], 1)
            left = []
            for r0 in range(0, n, step):
                r1 = min(n, r0 + step)
                o = self.order(torch.linalg.norm(c[None] - cen[r0:r1, None], dim=-1) / self.sqa[None])
                kv = self.kernels(cen[r0:r1, None, None], nrm[r0:r1, None, None], y[None], ny[None], w[None])
                z = self.entry(*(v.sum(-1) for v in kv), self.adm)
                if first:   # the self pairs come below
                    at = torch.arange(r0, r1, device=_dev())
                    o[at - r0, at] = 1
                a[r0:r1] += sg * torch.where(o == 2, z, torch.zeros_like(z))
                q = torch.nonzero((o != 2) & (o != 1))
                left.append(torch.stack([q[:, 0] + r0, q[:, 1]], 1))
                del kv, z
            for q in torch.split(torch.cat(left), 1000000):
                i, j = q[:, 0], q[:, 1]

                def fn(pid, yy, nn, ww, sh):
                    kv = self.kernels(cen[i[pid], None], nrm[i[pid], None], yy, nn, ww)
                    return torch.stack([v.sum(1) for v in kv], 1)

                kv = self.integrate(cen[i], el, j, fn, 4)
                a[i, j] += sg * self.entry(*kv.unbind(1), None if self.adm is None else self.adm[j])
        rows = torch.arange(n, device=_dev())
        g, h, ht, e, rhs = self.singular(rows)
        beta = 1j / self.k
        a[rows, rows] += self.entry(g, h, ht, e, self.adm) - 0.5
        if self.adm is not None:
            a[rows, rows] += 0.5 * beta * self.adm
        b = self.incident(cen, nrm)
        if self.bcv is not None:
            b = b + 0.5 * beta * self.bcv[:, :nv].mean(1)
            cols = torch.nonzero(self.bcv.abs().sum(1) > 0)[:, 0]
            for el, sg in self.images:
                first = el is self.images[0][0]
                val = self.bcv[:, :nv] if first else self.bcv[:, [1, 0, 2] if nv == 3 else [1, 0, 3, 2]]
                i = rows.repeat_interleave(len(cols))
                j = cols.repeat(n)
                if first:
                    i, j = i[i != j], j[rows.repeat_interleave(len(cols)) != j]
                for q in torch.split(torch.arange(len(i), device=_dev()), 1000000):
                    ii, jj = i[q], j[q]

                    def fn(pid, yy, nn, ww, sh):
                        g, _, ht, _ = self.kernels(cen[ii[pid], None], nrm[ii[pid], None], yy, nn, ww)
                        return ((g + ht * beta) * (sh.to(torch.complex128) @ val[jj[pid], :, None])[..., 0]).sum(1)[:, None]

                    b.index_add_(0, ii, self.integrate(cen[ii], el, jj, fn, 1)[:, 0])
            b[cols] += rhs[cols]
        return a, b

    def incident(self, x, nx=None):
        """Right-hand side at collocation points, or potential and gradient at field points."""
        p = torch.zeros(len(x), dtype=torch.complex128, device=_dev())
        gr = torch.zeros(len(x), 3, dtype=torch.complex128, device=_dev())
        for s, amp in zip(self.src, self.amp):
            for at in [s] + ([s * _t([1.0, -1.0, 1.0])] if self.sym else []):
                d = x - at
                r = torch.linalg.norm(d, dim=1)
                g = torch.polar(1 / (4 * math.pi * r), self.k * r) * amp
                p += g
                gr += (g * torch.complex(-1 / r, torch.full_like(r, self.k)))[:, None] * (d / r[:, None])
        if nx is None:
            return p, gr
        return -(p + (gr * nx).sum(1) * (1j / self.k))

    def solve(self, a, b):
        if self.n <= 6000:
            return torch.linalg.solve(a, b)
        # GMRES without restarts, its whole basis kept
        x, m = torch.zeros_like(b), 300
        for _ in range(4):
            r = b - a @ x
            beta = torch.linalg.norm(r)
            if beta <= 1e-13 * torch.linalg.norm(b):
                break
            v = torch.zeros(m + 1, self.n, dtype=torch.complex128, device=_dev())
            h = np.zeros((m + 1, m), complex)
            v[0] = r / beta
            used = m
            for q in range(m):
                w = a @ v[q]
                for _ in range(2):
                    c = v[: q + 1].conj() @ w
                    w = w - v[: q + 1].T @ c
                    h[: q + 1, q] += c.cpu().numpy()
                nw = torch.linalg.norm(w)
                h[q + 1, q] = float(nw)
                v[q + 1] = w / nw
                if q % 10 == 9:
                    y, res = self.small(h[: q + 2, : q + 1], float(beta))
                    if res <= 1e-13 * float(torch.linalg.norm(b)):
                        used = q + 1
                        break
            y, _ = self.small(h[: used + 1, :used], float(beta))
            x = x + v[:used].T @ _t(y, torch.complex128)
        return x

    @staticmethod
    def small(h, beta):
        e = np.zeros(len(h), complex)
        e[0] = beta
        y = np.linalg.lstsq(h, e, rcond=None)[0]
        return y, np.linalg.norm(e - h @ y)

    def field(self, x):
        """Potential and gradient at the evaluation points from the boundary values x."""
        pts, nv, k = self.pts, self.nv, self.k
        vel = None
        if self.bcv is not None or self.adm is not None:
            vel = torch.zeros(self.n, nv, dtype=torch.complex128, device=_dev())
            if self.bcv is not None:
                vel = vel + self.bcv[:, :nv]
            if self.adm is not None:
                vel = vel - (self.adm * x)[:, None]
        out = torch.zeros(len(pts), 4, dtype=torch.complex128, device=_dev())

        def point(xp, y, ny, w, sh, ph, vl):
            d = y - xp
            r = torch.linalg.norm(d, dim=-1)
            dh = d / r[..., None]
            g = torch.polar(1 / (4 * math.pi * r), k * r)
            gi = g * torch.complex(-1 / r, torch.full_like(r, k))
            dn = (dh * ny).sum(-1)
            f1 = g * torch.complex(dn * (k * k - 3 / r ** 2), 3 * k * dn / r)
            z = ph * w
            p = gi * dn * z
            gr = ((f1 * z)[..., None] * dh) - ((gi / r) * z)[..., None] * ny
            if vl is not None:
                q = w * vl
                p = p - g * q
                gr = gr + (gi * q)[..., None] * dh
            return torch.cat([p[..., None], gr], -1)

        rule = _t(_rule(nv, 2))
        step = max(1, 6000000 // (self.n * len(rule)))
        for el, sg in self.images:
            first = el is self.images[0][0]
            y, ny, jj, sh = _place(el, rule[:, 0].expand(self.n, -1), rule[:, 1].expand(self.n, -1))
            c = self.cen if first else torch.stack([self.cen[:, 0], -self.cen[:, 1], self.cen[:, 2]], 1)
            vi = None
            if vel is not None:
                vi = vel if first else vel[:, [1, 0, 2] if nv == 3 else [1, 0, 3, 2]]
            vq = None if vi is None else (sh.to(torch.complex128) @ vi[..., None])[..., 0]
            left = []
            for p0 in range(0, len(pts), step):
                xp = pts[p0:p0 + step]
                o = self.order(torch.linalg.norm(c[None] - xp[:, None], dim=-1) / self.sqa[None])
                z = point(xp[:, None, None], y[None], ny[None], (jj * rule[:, 2])[None], None, x[None, :, None],
                          None if vq is None else vq[None]).sum(2)
                out[p0:p0 + step] += sg * (z * (o == 2)[..., None]).sum(1)
                q = torch.nonzero(o != 2)
                left.append(torch.stack([q[:, 0] + p0, q[:, 1]], 1))
                del z
            for q in torch.split(torch.cat(left), 400000):
                i, j = q[:, 0], q[:, 1]

                def fn(pid, yy, nn, ww, sh):
                    vl = None if vi is None else (sh.to(torch.complex128) @ vi[j[pid], :, None])[..., 0]
                    return point(pts[i[pid], None], yy, nn, ww, sh, x[j[pid], None], vl).sum(1)

                out.index_add_(0, i, sg * self.integrate(pts[i], el, j, fn, 4))
        p, gr = self.incident(pts)
        return out[:, 0] + p, out[:, 1:] + gr


def exact(case, seed):
    ps, kind = _problems(case, seed), case["kind"]
    none = {"x": [None] * len(ps), "pot": [None] * len(ps), "grad": [None] * len(ps)}
    a = b = None
    budget = 1.2e9   # element pairs per call
    for i, p in enumerate(ps):
        n = len(p["f"])
        pairs = float(n) * n * (2 if p["planes"][1] else 1) + 1.5 * n * len(p["pts"])
        if kind == "multi" and i and a is not None:
            e = _Exact(p)
            b = e.incident(e.cen, e.nrm)
            pairs *= 0.3
        else:
            if n > 22000 or pairs > budget:
                continue
            a = b = None
            e = _Exact(p)
            a, b = e.system()
        budget -= pairs
        x = e.solve(a, b)
        pot, grad = e.field(x)
        for key, val in (("x", x), ("pot", pot), ("grad", grad)):
            none[key][i] = val.cpu().numpy()
        if kind == "multi" and i and budget < 0:
            break
    if all(v is None for v in none["pot"]):
        return None
    if kind in ("project", "static"):
        del none["x"]
    return none
