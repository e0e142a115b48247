"""Field points at which a staged element's 4-point rule is not the one to take,
exactly on that rule's second point: in the plane of a long triangle (1 : 32), where
the distance ratio asks for a higher order, while other points of the warp take
the 4-point rule.  Zero distance there must not reach the field.

FP64: 1e-12 of the largest value, the plain path's bar; mixed: 1e-5 of it (the
rule's nearest points are 0.04 of the length away; phases below 1 radian)."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu
H = 2.0**-5
V = np.array([[1.0, 0, 0], [0, H, 0], [0, 0, 0]])   # P0 - P2 and P1 - P2 along the axes


def _points_mixed():
    """Points whose offset from the rule's point, as the kernel forms it in
    float from high and low parts, is zero."""
    f = np.float32
    third, out = f(1) / f(3), []
    c = (V[0] * (1 / 3) + V[1] * (1 / 3)) + V[2] * (1 - 1 / 3 - 1 / 3)
    o = np.array([f(0.6) - third, (f(0.2) - third) * f(H), f(0)], f)
    for q in range(-40, 41):
        x = c + o.astype(float) * (1 + q * 2.0**-30)
        xh, ch = x.astype(f), c.astype(f)
        D = (ch - xh) + ((c - ch).astype(f) - (x - xh).astype(f))
        if np.array_equal(D, -o):
            out.append(x)
    return out


def _points_fp64():
    """The rule's point itself and its neighbours in double precision."""
    p = np.array([0.6, 0.2 * H, 0.0])
    return [p + [i * 2.0**-53, j * 2.0**-60, 0.0] for i in range(-4, 5) for j in range(-4, 5)]


@pytest.mark.parametrize("prec,bar", [(capi.PREC_FP64, 1e-12), (capi.PREC_MIXED, 1e-5)])
def test_points_on_another_rule(prec, bar):
    on = _points_fp64() if prec == capi.PREC_FP64 else _points_mixed()
    assert on
    far = 3.0 * meshes.fibonacci_sphere(2 * len(on), 1.0)
    pts = np.empty((3 * len(on), 3))
    pts[0::3], pts[1::3], pts[2::3] = on, far[::2], far[1::2]
    f, k = np.array([[0, 1, 2]], np.int32), 0.7
    bcv = np.full((1, 4), 1 + 0.5j)
    bcv[:, 3] = 0
    om, of = oracle.OracleMesh(V, f, None, bcv), oracle.OracleFreq(k, [[5.0, 1, 2]], [1e-2])
    m = capi.Mesh(V, f)
    s = capi.Solver(m, precision=prec)
    s.assemble(capi.Frequency(k, 1, bc_value=bcv, point_sources=[[5.0, 1, 2]], point_amps=[1e-2]))
    s.solve()
    pot, grad = s.project(pts)
    q, g = oracle.project(om, of, *oracle.boundary_fields(om, s.solution()), pts)
    s.close()
    m.close()
    assert np.abs(pot - q).max() <= bar * np.abs(q).max()
    assert np.abs(grad - g).max() <= bar * np.abs(g).max()
