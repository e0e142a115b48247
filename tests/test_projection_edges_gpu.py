"""The field projection at the edges of its work split (32- and 64-point
groups, element slices, blocks of few and many groups), against the FP64
restatement of the reference with the same boundary values.

FP64: 1e-12 of the largest value, the plain path's bar, also for points close
to the surface.  Mixed: an evaluation's relative error is at most
4 (k r + 8) 2^-24 (phase, distance and amplitude each rounded a few times), so
a potential is within that times the sum of the terms' sizes
|phi| A |ik - 1/r| / (4 pi r) + |v| A / (4 pi r) (their centroid values, twice
for the variation over an element)."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu
K = 20.0


def _problem(kind):
    rng = np.random.default_rng(11)
    if kind == "tri":
        v, f = meshes.geodesic_sphere(7, 0.1)   # 980 triangles: slices with a ragged end
        sym, adm = (0, 0, 0), None
    else:
        v, f = meshes.sphere_sector(14, 0.1, (1,), triangles=kind == "half_tri")
        sym, adm = (0, 2, 0), 1j * K * (0.2 + 0.1j) * (rng.random(len(f)) < 0.6)
    n = len(f)
    bct = None if adm is None else np.full(n, 2, np.int32)
    bcv = np.zeros((n, 4), complex)
    if kind != "tri":
        bcv[: n // 9, : f.shape[1]] = rng.normal(size=(n // 9, f.shape[1])) * 1e-2
    return v, f, sym, bct, adm, bcv


def _points(m, near):
    p = meshes.fibonacci_sphere(m, 0.5 if m % 2 else 1.2)
    p[:, 1] = np.abs(p[:, 1])
    if near:
        p[: m // 2] *= 0.104 / np.linalg.norm(p[: m // 2], axis=1)[:, None]
    return p


@pytest.mark.parametrize("kind", ["tri", "half_tri", "half_quad"])
@pytest.mark.parametrize("prec", [capi.PREC_FP64, capi.PREC_MIXED])
def test_point_counts(prec, kind):
    v, f, sym, bct, adm, bcv = _problem(kind)
    n = len(f)
    src, amp = [[0.5, 0.3, 0.2]], [1e-2]
    om, of = oracle.OracleMesh(v, f, bct, bcv, adm, sym=sym), oracle.OracleFreq(K, src, amp)
    mesh = capi.Mesh(v, f, sym_planes=sym)
    s = capi.Solver(mesh, precision=prec)
    s.assemble(capi.Frequency(K, n, bc_type=bct, bc_value=bcv, admittance=adm, point_sources=src, point_amps=amp))
    s.solve()
    phi, vel = oracle.boundary_fields(om, s.solution())
    area = om.areas
    for m in (1, 31, 32, 33, 64, 65, 129, 400, 641, 2433):
        fp64 = prec == capi.PREC_FP64
        p = _points(m, near=fp64)
        pot, grad = s.project(p)
        sel = slice(None) if m < 700 else slice(0, m, 37)
        q, g = oracle.project(om, of, phi, vel, p[sel])
        if fp64:
            assert np.abs(pot[sel] - q).max() <= 1e-12 * np.abs(q).max(), m
            assert np.abs(grad[sel] - g).max() <= 1e-12 * np.abs(g).max(), m
            continue
        r = np.linalg.norm(p[sel][:, None] - om.centers[None], axis=2)
        images = 2 if any(sym) else 1
        terms = (np.abs(phi) * area / (4 * np.pi * r) * np.hypot(K, 1 / r)
                 + np.abs(vel).max(axis=1) * area / (4 * np.pi * r)).sum(axis=1) * 2 * images
        bound = 4 * (K * (r.max() + 0.3) + 8) * 2.0 ** -24 * terms
        assert (np.abs(pot[sel] - q) <= bound + 1e-12 * np.abs(q).max()).all(), m
    s.close()
    mesh.close()


@pytest.mark.parametrize("count", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("kind", ["tri", "half_quad"])
def test_right_hand_sides_share_evaluations(kind, count):
    """Every right-hand side's field is the one its own projection gives: the
    same operations in the same order, so equal up to the unknowns' own
    difference (1e-7, the agreement of grouped and single solves)."""
    v, f, sym, bct, adm, bcv = _problem(kind)
    n = len(f)
    mesh = capi.Mesh(v, f, sym_planes=sym)
    fr = [capi.Frequency(K, n, bc_type=bct, bc_value=bcv if r % 2 else None, admittance=adm,
                         point_sources=[[0.5, 0.3 + 0.01 * r, 0.2]], point_amps=[1e-2]) for r in range(count)]
    p = _points(130, near=False)
    s = capi.Solver(mesh, precision=capi.PREC_MIXED, tol=1e-10, n_rhs=count)
    xs, pots, grads, _ = s.solve_multi(fr, p)
    one = capi.Solver(mesh, precision=capi.PREC_MIXED, tol=1e-10)
    for r in range(count):
        x0, p0, g0 = one.solve_frequency(fr[r], p)
        assert np.linalg.norm(xs[r] - x0) <= 1e-7 * np.linalg.norm(x0)
        assert np.linalg.norm(pots[r] - p0) <= 3e-7 * np.linalg.norm(p0)
        assert np.linalg.norm(grads[r] - g0) <= 3e-7 * np.linalg.norm(g0)
    s.close()
    one.close()
    mesh.close()
