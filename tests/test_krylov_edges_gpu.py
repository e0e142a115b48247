"""GMRES at system sizes around the kernels' blocks (32-row groups, 128-row
preconditioner blocks, 256-row vector blocks, 1024-column chunks and windows):
the solution against a dense solve of the assembled system, both precisions,
and a batch whose row count makes an item take several row groups.

Bar: the relative residual target is 1e-10 and the systems' condition numbers
stay below 1e3, so the solution is within 1e-7 of the dense one."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


def _freq(n, k=15.0):
    return capi.Frequency(k, n, point_sources=[[0.5, 0.2, 0.1]], point_amps=[1e-2])


@pytest.mark.parametrize("prec", [capi.PREC_FP64, capi.PREC_MIXED])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 255, 257, 640, 1023, 1024, 1025, 1280])
def test_sizes_around_the_blocks(n, prec):
    v, f = meshes.geodesic_sphere(8, 0.1)
    m = capi.Mesh(v, f[:n])
    s = capi.Solver(m, precision=prec, tol=1e-10)
    s.assemble(_freq(n))
    A, b = s.system()
    s.solve()
    x = np.linalg.solve(A, b)
    assert s.info.rel_residual <= 1e-10
    assert np.linalg.norm(s.solution() - x) <= 1e-7 * np.linalg.norm(x)
    s.close()
    m.close()


def test_many_rows_in_a_batch_equal_single_solves():
    """Over 2432 row groups in the batch: items of four groups, bit for bit the
    single solves' results."""
    v, f = meshes.geodesic_sphere(16, 0.1)   # 5120 triangles
    n = len(f)
    m = capi.Mesh(v, f)
    ks = [8.0 + 2.0 * i for i in range(16)]
    ss = [capi.Solver(m, precision=capi.PREC_MIXED) for _ in ks]
    res = capi.solve_batch(ss, [_freq(n, k) for k in ks])
    for i in (0, 7, 15):
        one = capi.Solver(m, precision=capi.PREC_MIXED)
        x, _, _ = one.solve_frequency(_freq(n, ks[i]), np.zeros((0, 3)))
        assert np.array_equal(res[i][0], x), (i, np.abs(res[i][0] - x).max() / np.abs(x).max())
        one.close()
    for s in ss:
        s.close()
    m.close()
