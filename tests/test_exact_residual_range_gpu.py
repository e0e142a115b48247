"""The first cycle's residual of shared right-hand sides near the end of the
float range, where a bias on the sums would not be finite: the unknowns reach
6e37, a stage's bound on its products more than 4e37.  Bar: test_exact_residual's, the reported
residual within 1e-9 of b - A x."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e39])
def test_reported_residual(scale):
    v, f = meshes.head_like(15)[:2]   # 4500 triangles
    n = len(f)
    m = capi.Mesh(v, f)
    k = 2 * np.pi * 4000 / 343
    fr = [capi.Frequency(k, n, point_sources=[meshes.surface_point_with_normal(v, f, 40 + r)], point_amps=[1e-4 * scale])
          for r in range(3)]
    s = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9, n_rhs=3)
    xs, _, _, infos = s.solve_multi(fr, np.zeros((0, 3)))
    one = capi.Solver(m, precision=capi.PREC_MIXED)
    for r in range(3):
        one.assemble(fr[r])
        A, b = one.system()
        true = np.linalg.norm(b / scale - A @ (xs[r] / scale)) / np.linalg.norm(b / scale)
        assert infos[r]["rel_residual"] <= 1e-9 and true <= infos[r]["rel_residual"] + 1e-9
    one.close()
    s.close()
    m.close()
