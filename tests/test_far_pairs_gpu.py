"""FP32 regular entries (two rows at a time, a warp's item of 2 .. 16 rows by
32 columns) against the FP64 restatement of the reference: triangles and
quadrilaterals, every boundary condition, symmetry images, element counts that
leave ragged rows and columns, small and large wave numbers.

Bar, per column condition, of the row's largest regular entry (the element's
and its image's magnitudes added: an antisymmetric pair cancels and keeps the
rounding of both): with u = 2^-24
a distance is good to 5 u (three squares, the reciprocal root, two products),
so the phase to 5 u k r; reduction, sine and cosine add 11 u and the some
twenty operations of the four points as much again.  Rounded up: u (64 + 8 k r)
with r the body's diameter."""
import ctypes as C

import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu


def _mixed():
    """A sphere whose upper faces are triangles and lower faces quadrilaterals,
    two of them halved: an odd number of elements."""
    v, f = meshes.cube_sphere(7, 0.1)
    out = []
    for q, e in enumerate(f):
        if q % 3 == 0:
            out += [[e[0], e[1], e[2], -1], [e[0], e[2], e[3], -1]]
        else:
            out.append(list(e))
    out = out if len(out) % 2 else out[:-1]   # an open surface is as good here
    return v, np.array(out, np.int32)


SHAPES = {
    "mixed": lambda: (*_mixed(), (0, 0, 0)),
    "quads": lambda: (*meshes.cube_sphere(5, 0.1), (0, 0, 0)),
    "half": lambda: (*meshes.sphere_sector(8, 0.1, (1,), triangles=True), (0, 2, 0)),
    "half_quads": lambda: (*meshes.sphere_sector(6, 0.1, (1,)), (0, 1, 0)),
    "sixteen_rows": lambda: (*meshes.geodesic_sphere(12, 0.1), (0, 0, 0)),
}


def _oracle_mesh(v, f, bct, adm, sym):
    om = oracle.OracleMesh(v, f, bct, None, adm, sym=sym)
    if f.shape[1] == 4:   # the wrapper takes four columns for quadrilaterals only
        om.nvert[f[:, 3] < 0] = 3
        p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in (om.centers, om.normals, om.areas)]
        oracle.lib().or_geometry(C.byref(om._s), *p)
    return om


@pytest.mark.parametrize("k", [2.0, 250.0])
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_entries(shape, bc, k):
    if shape == "sixteen_rows" and (bc, k) != (2, 250.0):
        pytest.skip("the large mesh runs once")
    v, f, sym = SHAPES[shape]()
    f = np.asarray(f)
    n = len(f)
    rng = np.random.default_rng(5)
    bct = np.where(rng.random(n) < 0.5, bc, 0).astype(np.int32)
    adm = np.where(bct == 2, (0.3 + 0.2j) * k, 0.0) * 1j
    src, amp = [[0.5, 0.3, 0.2]], [1.0 + 0.5j]
    A, _ = oracle.assemble(_oracle_mesh(v, f, bct, adm, sym), oracle.OracleFreq(k, src, amp))
    mag = np.abs(A)
    if any(sym):
        E, O = (oracle.assemble(_oracle_mesh(v, f, bct, adm, (0, q, 0)), oracle.OracleFreq(k, src, amp))[0] for q in (1, 2))
        mag = (np.abs(E + O) + np.abs(E - O)) / 2
    m = capi.Mesh(v, f, sym_planes=sym)
    s = capi.Solver(m, precision=capi.PREC_MIXED)
    s.assemble(capi.Frequency(k, n, bc_type=bct, admittance=adm, point_sources=src, point_amps=amp))
    A2, _ = s.system()
    s.close()
    m.close()
    # pairs well clear of the subdivided ones, for the images too
    c = np.array([v[[x for x in e if x >= 0]].mean(0) for e in f])
    size = np.sqrt(np.array([np.linalg.norm(np.cross(v[e[1]] - v[e[0]], v[e[2]] - v[e[0]])) for e in f]))
    far = np.ones((n, n), bool)
    for sg in ((1, -1) if any(sym) else (1,)):
        d = np.linalg.norm(c[:, None] - c[None] * np.array([1, sg, 1]), axis=2)
        far &= d > 2.5 * size[None]
    bar = 2.0 ** -24 * (64 + 8 * k * 0.2)
    for t in np.unique(bct):
        cols = far & (bct == t)[None]
        scale = np.where(cols, mag, 0).max(1, keepdims=True)
        assert (np.where(cols, np.abs(A2 - A), 0) <= bar * scale).all()
