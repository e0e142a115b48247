"""The preconditioner's window correction for right-hand sides that share a
matrix (one read of the windows for up to eight): sizes whose last window is
one column, odd, or nearly full, and nine right-hand sides, eight of which
share.  A wrong correction costs iterations, so each right-hand side takes the
steps of its single solve (at most one more refinement cycle's, eight, or two
fewer, as for the shared products) and gives its solution to 1e-7."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1025, 1279, 2046])
@pytest.mark.parametrize("n_rhs", [2, 9])
def test_iterations_and_solutions(n, n_rhs):
    v, f = meshes.perturbed_ellipsoid(11, 7)   # 2420 triangles
    f = f[:n]
    m = capi.Mesh(v, f)
    fr = [workloads.frequency(capi, n, 5000.0, meshes.surface_point_with_normal(v, f, 60 + r)) for r in range(n_rhs)]
    pts = np.zeros((0, 3))
    s = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9, n_rhs=n_rhs)
    xs, _, _, infos = s.solve_multi(fr, pts)
    one = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9)
    for r in range(n_rhs):
        x0 = one.solve_frequency(fr[r], pts)[0]
        assert infos[r]["rel_residual"] <= 1e-9
        assert -2 <= infos[r]["iterations"] - one.info.iterations <= 8
        assert np.linalg.norm(xs[r] - x0) <= 1e-7 * np.linalg.norm(x0)
    s.close()
    one.close()
    m.close()
