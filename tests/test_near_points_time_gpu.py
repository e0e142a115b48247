"""A few hundred points near the surface among thousands on a small mesh must not
hold up the call: their subdivided and higher-order pairs are some 10^4 of 10^7 and
spread over the GPU, so the call takes at most three times as long as with all
points far.  (Best of several calls of each kind, in turn.)"""
import time

import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points", [(10, 10000), (13, 7000)])
def test_near_points_are_spread(n, points):
    v, f = meshes.head_like(n)[:2]
    rng = np.random.default_rng(2)
    far = meshes.fibonacci_sphere(points, 1.2)
    near = far.copy()
    t = v[f[rng.integers(len(f), size=500)]]
    nrm = np.cross(t[:, 0] - t[:, 2], t[:, 1] - t[:, 2])
    near[:500] = t.mean(1) + nrm / np.linalg.norm(nrm, axis=1)[:, None] * rng.uniform(0.003, 0.03, 500)[:, None]
    m = capi.Mesh(v, f)
    s = capi.Solver(m, precision=capi.PREC_MIXED)
    s.solve_frequency(capi.Frequency(30.0, len(f), point_sources=[[0.5, 0.3, 0.2]], point_amps=[1.0]), np.zeros((0, 3)))
    best = {}
    for _ in range(8):
        for name, p in (("far", far), ("near", near)):
            t0 = time.perf_counter()
            s.project(p)
            best[name] = min(best.get(name, 1e9), time.perf_counter() - t0)
    s.close()
    m.close()
    assert best["near"] <= 3 * best["far"], best
