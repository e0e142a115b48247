"""The first cycle's residual with error-free products: the residual that a
mixed solve reports against b - A x summed in 64 bits from the same complex64
matrix.  Several right-hand sides (the shared product, biased sums from 4096
unknowns on, two-sums below) and one (16 warps, two stages in flight); odd
element counts, so that the last column of a stage stands alone.

Bar: the reported residual is recursive after the first cycle, r -= A d with
|d| at most 3e-4 |x| and products good to 2^-22, so it differs from the true
one by 2^-22 * 3e-4 of |A| |x| (some ten times |b|) plus the first residual's
own error, below 1e-12 of it: 1e-9 over the reported value covers both."""
import numpy as np
import pytest

from mesh2hrtf_gb300 import capi, meshes, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rhs", [1, 3, 8])
@pytest.mark.parametrize("q,drop", [(14, 1), (15, 0), (15, 1)])
def test_reported_residual(q, drop, n_rhs):
    v, f = meshes.head_like(q)[:2]
    f = f[: len(f) - drop]
    n = len(f)
    m = capi.Mesh(v, f)
    fr = [workloads.frequency(capi, n, 4000.0, meshes.surface_point_with_normal(v, f, 40 + r)) for r in range(n_rhs)]
    one = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9)
    if n_rhs > 1:
        s = capi.Solver(m, precision=capi.PREC_MIXED, tol=1e-9, n_rhs=8)
        xs, _, _, infos = s.solve_multi(fr, np.zeros((0, 3)))
        s.close()
    for r in range(n_rhs):
        one.assemble(fr[r])
        A, b = one.system()
        if n_rhs > 1:
            x, rel = xs[r], infos[r]["rel_residual"]
        else:
            x = one.solve_frequency(fr[r], np.zeros((0, 3)))[0]
            rel = one.info.rel_residual
        true = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        assert rel <= 1e-9 and true <= rel + 1e-9
    one.close()
    m.close()
