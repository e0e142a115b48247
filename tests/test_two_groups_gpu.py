"""More right-hand sides than one shared-matrix group holds (eight): two groups
whose members end their cycles in different steps.  Smooth distant sources in
the first group converge sooner than sources at the surface in the second,
whose window corrections then run in the step that ends the first group's
cycle.

Iterations and solutions as a single solve's, with test_multi_rhs_gpu's
allowances; and no schedule of the blocks may show in a result, so repeated
solves agree bit for bit."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1025, 2420])
@pytest.mark.parametrize("n_rhs", [10, 12, 16])
def test_groups_end_apart(n_rhs, n):
    v, f = meshes.perturbed_ellipsoid(11, 7)   # 2420 triangles
    f = f[:n]
    m = capi.Mesh(v, f)
    far = [np.array([2.0, 0.3 * r, 0.1]) for r in range(8)]
    near = [meshes.surface_point_with_normal(v, f, 60 + r) for r in range(n_rhs - 8)]
    fr = [workloads.frequency(capi, n, 5000.0, p) for p in far + near]
    pts = np.zeros((0, 3))
    s = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9, n_rhs=n_rhs)
    xs, _, _, infos = s.solve_multi(fr, pts)
    xs = [np.array(x) for x in xs]
    its = [i["iterations"] for i in infos]
    for _ in range(3):
        again, _, _, infos2 = s.solve_multi(fr, pts)
        assert [i["iterations"] for i in infos2] == its
        assert all(np.array_equal(a, b) for a, b in zip(again, xs))
    one = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9)
    for r in range(n_rhs):
        x0 = one.solve_frequency(fr[r], pts)[0]
        assert infos[r]["rel_residual"] <= 1e-9
        assert -2 <= its[r] - one.info.iterations <= 8
        assert np.linalg.norm(xs[r] - x0) <= 1e-7 * np.linalg.norm(x0)
    assert len(set(its)) > 1   # not all in the same step
    s.close()
    one.close()
    m.close()
