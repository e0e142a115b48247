"""Matrix entries where a far pair's quadrature point is much closer than
its centroid: a long thin triangle (1 : 500) whose distance ratio asks for the
4-point rule, collocation points 3e-4 and 3e-3 of its length beside two of the
rule's points, against the same rule in extended precision.

FP64, and mixed precision with a symmetry plane (far enough for the images to
be below the bar).  Bar: a point's vector d = y - x has an error of
3 u (|y| + |x|), u the unit roundoff, with both within the length of 1 (float
works with vectors from the centroid), so r and the products with the normals are good to
6 u / r of themselves; an entry's terms go with up to 1 / r^3, with a distance
and two products in them, and some forty operations more:
(8 * 6 u / r + 64 u) of the sum of the terms' sizes."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi

pytestmark = pytest.mark.gpu
L = np.longdouble
RULE = [(1 / 3, 1 / 3, -27 / 96), (0.2, 0.2, 25 / 96), (0.6, 0.2, 25 / 96), (0.2, 0.6, 25 / 96)]


def _mesh(rng):
    """A long triangle (element 0) about the origin and two small ones beside
    each of two points of its rule."""
    p = np.array([[0, 0, 0], [1, 0, 0], [rng.uniform(0.3, 0.7), 0.002, 0]]) - [0.5, 0, 0]
    p = p @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
    a, b = p[0] - p[2], p[1] - p[2]
    nrm = np.cross(a, b) / np.linalg.norm(np.cross(a, b))
    v, f = list(p), [[0, 1, 2]]
    for s, t, _ in RULE[2:]:
        for h in (3e-4, 3e-3):
            e = 2e-5 * rng.normal(size=(3, 3))
            f.append([len(v), len(v) + 1, len(v) + 2])
            v += list(p[2] + s * a + t * b + h * nrm + e - e.mean(0))
    return np.array(v), np.array(f, np.int32)


def _entry(p, x, nx, k, tau=1):
    a, b = p[0] - p[2], p[1] - p[2]
    n = np.cross(a, b)
    J = np.sqrt((n * n).sum())
    n = n / J
    z = size = L(0)
    for s, t, w in RULE:
        d = p[2] + L(s) * a + L(t) * b - x
        r = np.sqrt((d * d).sum())
        g = L(w) * J / (4 * L(np.pi) * r)
        re1, re2, nn = (d * n).sum() / r, -(d * nx).sum() / r, (n * nx).sum()
        z1 = -1 / r + 1j * k
        e = (3 / r**2 - k * k) * re1 * re2 + nn / r**2 - 1j * k / r * (3 * re1 * re2 + nn)
        z = z + (np.cos(k * r) + 1j * np.sin(k * r)) * g * (z1 * re1 + 1j / k * e)
        size = size + abs(g) * (8 / r + 8 / (k * r**2) + 8 * k)
    return z, size


@pytest.mark.parametrize("seed", [4, 5, 6])
@pytest.mark.parametrize("k", [2.0, 60.0])
@pytest.mark.parametrize("prec,sym,u", [(capi.PREC_FP64, (0, 0, 0), 2.0**-53), (capi.PREC_MIXED, (0, 1, 0), 2.0**-24)])
def test_entries(prec, sym, u, k, seed):
    v, f = _mesh(np.random.default_rng(seed))
    if any(sym):
        v = v + [0, 40.0, 0]
    m = capi.Mesh(v, f, sym_planes=sym)
    s = capi.Solver(m, precision=prec)
    s.assemble(capi.Frequency(k, len(f), point_sources=[[9.0, 9.0, 9.0]], point_amps=[1.0]))
    A, _ = s.system()
    s.close()
    m.close()
    p = v[f[0]].astype(L)
    a, b = p[0] - p[2], p[1] - p[2]
    for i in range(1, len(f)):
        q = v[f[i]]
        x = ((q[0] * (1 / 3) + q[1] * (1 / 3)) + q[2] * (1 - 1 / 3 - 1 / 3)).astype(L)
        n = np.cross(q[0] - q[2], q[1] - q[2])
        z, size = _entry(p, x, (n / np.linalg.norm(n)).astype(L), L(k))
        r = min(float(np.linalg.norm((p[2] + s_ * a + t * b - x).astype(float))) for s_, t, _ in RULE)
        bar = (48 * u / r + 64 * u) * size
        assert abs(L(A[i, 0].real) - z.real) <= bar and abs(L(A[i, 0].imag) - z.imag) <= bar, i
