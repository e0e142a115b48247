"""The right-hand side with and without boundary columns against the FP64
restatement of the reference, at row and column counts around the kernel's
64-row blocks, 8-row blocks and 32-column passes, on triangles and
quadrilaterals with a symmetry plane.  Bar: 1e-12 of the largest entry, the
plain path's."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 63, 64, 65, 129])
@pytest.mark.parametrize("cols", [0, 1, 31, 33, 64])
@pytest.mark.parametrize("quads", [False, True])
def test_rhs_rows_and_columns(quads, cols, rows):
    if quads:
        v, f = meshes.sphere_sector(10, 0.1, (1,))
        sym = (0, 1, 0)
    else:
        v, f = meshes.geodesic_sphere(3, 0.1)
        sym = (0, 0, 0)
    f = f[:rows]
    cols = min(cols, rows)
    rng = np.random.default_rng(rows + cols)
    bcv = np.zeros((rows, 4), complex)
    bcv[rng.permutation(rows)[:cols], : f.shape[1]] = rng.normal(size=(cols, f.shape[1])) + 0.5j
    src, amp, k = [[0.5, 0.3, 0.2]], [1.0 + 0.5j], 20.0
    _, b = oracle.assemble(oracle.OracleMesh(v, f, None, bcv, None, sym=sym), oracle.OracleFreq(k, src, amp))
    m = capi.Mesh(v, f, sym_planes=sym)
    s = capi.Solver(m, precision=capi.PREC_FP64)
    s.assemble(capi.Frequency(k, rows, bc_value=bcv, point_sources=src, point_amps=amp))
    _, b2 = s.system(with_matrix=False)
    assert np.abs(b2 - b).max() <= 1e-12 * np.abs(b).max()
    s.close()
    m.close()
