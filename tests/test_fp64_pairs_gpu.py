"""FP64 matrix entries of flat triangles against the FP64 restatement of the
reference, for every boundary condition and with a symmetry plane: far pairs
of every Gauss order (the sphere's near neighbours take the 7- and 13-point
rules) and high wave numbers (phases of tens of radians through the sine
table).  Bar: 1e-12 of the matrix scale, the plain path's."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2.0, 250.0])
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("half", [False, True])
def test_entries_by_boundary_condition(half, bc, k):
    if half:
        v, f = meshes.sphere_sector(6, 0.1, (1,), triangles=True)
        sym = (0, 2, 0)
    else:
        v, f = meshes.geodesic_sphere(3, 0.1)
        sym = (0, 0, 0)
    n = len(f)
    rng = np.random.default_rng(3)
    bct = np.where(rng.random(n) < 0.5, bc, 0).astype(np.int32)
    adm = np.where(bct == 2, (0.3 + 0.2j) * k, 0.0) * 1j
    src, amp = [[0.5, 0.3, 0.2]], [1.0 + 0.5j]
    A, b = oracle.assemble(oracle.OracleMesh(v, f, bct, None, adm, sym=sym), oracle.OracleFreq(k, src, amp))
    m = capi.Mesh(v, f, sym_planes=sym)
    s = capi.Solver(m, precision=capi.PREC_FP64)
    s.assemble(capi.Frequency(k, n, bc_type=bct, admittance=adm, point_sources=src, point_amps=amp))
    A2, b2 = s.system()
    assert np.abs(A2 - A).max() <= 1e-12 * np.abs(A).max()
    assert np.abs(b2 - b).max() <= 1e-12 * np.abs(b).max()
    s.close()
    m.close()
