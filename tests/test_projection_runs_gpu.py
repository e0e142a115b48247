"""FP32 sums of the field over long slices of elements: 60000 points on 8000
elements leave scratch for a few slices only, so that a lane adds one to two
thousand elements.  On a pulsating sphere at a low frequency their terms have one
sign and the sum's roundings show.

Bar, mean relative error in units of u = 2^-24: of some 25 runs of 64 elements each
has up to 512 roundings at a 25th of the sum or less, sqrt(512) / 2 / 25 = 0.5 u a
run and 2.3 u over all; adding the runs 2.5 u; one evaluation's error that all terms
share (reciprocal root, sine and cosine, products) 6 u: 12 u.  One sum over the
slice has 10^4 roundings: sqrt(10^4) / 3 = 33 u."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quads", [False, True])
def test_long_slices(quads):
    v, f = meshes.cube_sphere(36, 0.1) if quads else meshes.geodesic_sphere(20, 0.1)
    f = np.asarray(f)
    n, k = len(f), 0.5
    bcv = np.zeros((n, 4), complex)
    bcv[:, : f.shape[1]] = 1.0
    src, amp = [[5.0, 0.0, 0.0]], [1e-30]
    m = capi.Mesh(v, f)
    s = capi.Solver(m, precision=capi.PREC_MIXED)
    s.assemble(capi.Frequency(k, n, bc_value=bcv, point_sources=src, point_amps=amp))
    s.solve()
    p = meshes.fibonacci_sphere(60000, 1.0)
    pot, grad = s.project(p)
    om = oracle.OracleMesh(v, f, None, bcv)
    sel = slice(0, None, 300)
    q, g = oracle.project(om, oracle.OracleFreq(k, src, amp), *oracle.boundary_fields(om, s.solution()), p[sel])
    s.close()
    m.close()
    u = 2.0**-24
    assert (np.abs(pot[sel] - q) / np.abs(q)).mean() <= 12 * u
    assert (np.linalg.norm(grad[sel] - g, axis=1) / np.linalg.norm(g, axis=1)).mean() <= 12 * u
