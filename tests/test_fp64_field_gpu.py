"""The FP64 field of triangles, all pairs far, is as good as a plain evaluation
of the same rule in double precision: mean errors against extended precision
over two flattened heads and 1200 points each, where the phase's rounding
k r u is the error.

Bar: 1.1 times the plain evaluation's mean error (a mean of some 1200 points'
rounding errors scatters by a few percent)."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu
RULE = [(1 / 3, 1 / 3, -27 / 96), (0.2, 0.2, 25 / 96), (0.6, 0.2, 25 / 96), (0.2, 0.6, 25 / 96)]


def _field(T, v, f, phi, vel, k, pts):
    """The 4-point rule over every element, in real type T."""
    C = np.result_type(T, np.complex64).type
    p, pts, k = v[f].astype(T), pts.astype(T), T(k)
    phi, vel = phi.astype(C), vel.astype(C)
    a, b = p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]
    n = np.cross(a, b)
    J = np.sqrt((n * n).sum(1))
    n = n / J[:, None]
    out = np.zeros(len(pts), C)
    for s, t, w in RULE:
        s, t = T(s), T(t)
        y = s * p[:, 0] + t * p[:, 1] + (1 - s - t) * p[:, 2]
        d = y[None] - pts[:, None]
        r = np.sqrt((d * d).sum(-1))
        g = (np.cos(k * r) + C(1j) * np.sin(k * r)) * (T(w) * J / (4 * T(np.longdouble("3.14159265358979323846")) * r))
        dn = (d * n).sum(-1) / r
        out += (g * ((-1 / r + C(1j) * k) * dn * phi - vel)).sum(1)
    return out


@pytest.mark.parametrize("k", [73.0, 290.0])
def test_mean_error(k):
    err = np.zeros(2)
    for seed in (1, 2):
        v, f = meshes.geodesic_sphere(4, 0.1)   # 320 triangles
        v = v * [1, 1, 0.1 * seed]
        n = len(f)
        rng = np.random.default_rng(seed)
        bcv = np.zeros((n, 4), complex)
        bcv[: n // 8, :3] = (rng.normal(size=n // 8) + 1j * rng.normal(size=n // 8))[:, None] * 1e-2
        pts = rng.normal(size=(1200, 3))
        pts *= (rng.uniform(0.5, 1.6, 1200) / np.linalg.norm(pts, axis=1))[:, None]
        m = capi.Mesh(v, f)
        s = capi.Solver(m, precision=capi.PREC_FP64)
        # a source far too weak to be seen: the field is the body's alone
        s.assemble(capi.Frequency(k, n, bc_value=bcv, point_sources=[[5.0, 0.0, 0.0]], point_amps=[1e-40]))
        s.solve()
        x, (pot, _) = s.solution(), s.project(pts)
        s.close()
        m.close()
        exact = _field(np.longdouble, v, f, x, bcv[:, 0], k, pts)
        for i, q in enumerate((pot, _field(np.float64, v, f, x, bcv[:, 0], k, pts))):
            err[i] += (np.abs(q - exact) / np.abs(exact)).mean()
    assert err[0] <= 1.1 * err[1], err
