"""The constants of the FP32 far pairs carry no rounding of their products: of two
neighbouring wave numbers, both floats, float(1 / k) k is 1 for one and rounds to
the float below 1 for the other, and the fitted scale of the matrices of pressure
elements (all pairs with k r above 20, where the product scales one of an
entry's two terms of like size) has to agree.

Bar: 2^-26, a quarter of the unit that the product was off by; the fit over
some 10^6 rounding errors of 10^-6 (the phases') scatters by 10^-9, and every other
constant's rounding cancels in the difference."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


def _scale(m, v, f, k):
    A, n = [], len(f)
    for prec in (capi.PREC_FP64, capi.PREC_MIXED):
        s = capi.Solver(m, precision=prec)
        s.assemble(capi.Frequency(k, n, bc_type=np.ones(n, np.int32), point_sources=[[0.5, 0.3, 0.2]], point_amps=[1.0]))
        A.append(s.system()[0])
        s.close()
    c = v[f].mean(axis=1)
    far = k * np.linalg.norm(c[:, None] - c[None], axis=2) > 20
    return (np.vdot(A[0][far], (A[1] - A[0])[far]) / np.vdot(A[0][far], A[0][far])).real


@pytest.mark.parametrize("triangles", [True, False])
def test_wave_numbers_agree(triangles):
    ks = 200.0 + 2.0**-16 * np.arange(2000)
    p = np.array([np.float32(1 / k) * np.float32(k) for k in ks])
    bad, good = ks[p < 1][0], ks[p == 1][0]
    v, f = meshes.geodesic_sphere(8, 0.1) if triangles else meshes.cube_sphere(14, 0.1)
    f = np.asarray(f)
    m = capi.Mesh(v, f)
    d = _scale(m, v, f, bad) - _scale(m, v, f, good)
    m.close()
    assert abs(d) <= 2.0**-26, d
