"""The preconditioner's 128-row block inverses: on 128 unknowns the block is
the matrix, so GMRES ends in one step per cycle in FP64 (bar: 2 steps; the
inverse is good to about 1e-13 of the condition number) and in a few with the
fp16 copy of the matrix (a step leaves about 5e-4, so three cycles of at most
two steps reach 1e-9; bar: 8).  Pressure elements among velocity ones put the
largest entries of columns off the diagonal, so pivots leave it.  With a
second, partial block (129) and several blocks (384) a wrong block would cost
dozens of steps; bar there: FP64 and mixed within 4 steps a cycle."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 129, 384])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("k", [3.0, 40.0])
def test_steps_with_block_inverses(n, bc, k):
    v, f = meshes.geodesic_sphere(5, 0.1)   # 500 triangles
    f = f[:n]
    rng = np.random.default_rng(n)
    bct = np.where(rng.random(n) < 0.4, bc, 0).astype(np.int32)
    fr = capi.Frequency(k, n, bc_type=bct, point_sources=[[0.4, 0.3, 0.2]], point_amps=[1.0])
    m = capi.Mesh(v, f)
    steps = {}
    for prec in (capi.PREC_FP64, capi.PREC_MIXED):
        s = capi.Solver(m, precision=prec, tol=1e-9, precond="block-jacobi")
        x, _, _ = s.solve_frequency(fr, np.zeros((0, 3)))
        A, b = s.system()
        assert np.linalg.norm(b - A @ x) <= 3e-9 * np.linalg.norm(b)
        steps[prec] = (s.info.iterations, s.info.restarts)
        s.close()
    m.close()
    if n == 128:
        assert steps[capi.PREC_FP64][0] <= 2 and steps[capi.PREC_MIXED][0] <= 8
    else:
        assert steps[capi.PREC_MIXED][0] <= steps[capi.PREC_FP64][0] + 4 * steps[capi.PREC_MIXED][1]
