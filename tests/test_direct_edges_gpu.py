"""The dense direct solver at the edges of its 32-column panels and 64 x 64
update tiles: sizes below, at and just above them, against the assembled
system itself.

Bar: the backward error |b - A x| / (|A| |x|) of an n x n elimination without
pivoting is at most 8 n u for these diagonally heavy matrices (growth factor
below 2; four real operations per complex one), u the unit roundoff of the
factors (2^-53 or 2^-24)."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,u", [(capi.PREC_FP64, 2.0 ** -53), (capi.PREC_MIXED, 2.0 ** -24)])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 130, 320])
def test_backward_error_at_panel_edges(n, prec, u):
    v, f = meshes.geodesic_sphere(4, 0.1)
    m = capi.Mesh(v, f[:n])
    s = capi.Solver(m, precision=prec)
    s.assemble(capi.Frequency(15.0, n, point_sources=[[1.0, 0.2, 0.1]], point_amps=[1.0]))
    A, b = s.system()
    s.solve_direct()
    x = s.solution()
    r = np.linalg.norm(b - A @ x) / (np.linalg.norm(A, 2) * np.linalg.norm(x))
    assert r <= 8 * n * u, (r, 8 * n * u)
    s.close()
    m.close()
