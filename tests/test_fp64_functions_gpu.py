"""The FP64 path's own functions, as the kernels compile them.

Square root: over exponents of -300 .. 300 the root is the correctly rounded one
(its last step adds a fused residual good to 2^-51 of the correction, so a wrong
rounding needs a value that close to a tie), and the inverse is within 1.5 units
in the last place.

Sine and cosine: the table's two parts are good to 2^-64 or more, the angle sum's
corrections (below 2^-8) carry three roundings and the result one: half a unit in
the last place plus 2^-58, up to phases of 2^43; the library's two units beyond."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mesh2hrtf_gb300 import build, capi
from oracle import oracle_py as oracle

pytestmark = pytest.mark.gpu

CODE = r"""
#include "bem_common.cuh"
__global__ void k_root(int n, const double *x, double *root, double *inv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) inv[i] = bem::rsqrt_nr(x[i], root + i);
}
__global__ void k_sincos(int n, const double *x, double *s, double *c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) bem::sincos_t(x[i], s + i, c + i);
}
static double *up(int n, const double *h) {
    double *d = nullptr;
    cudaMalloc(&d, sizeof(double) * n);
    if (h) cudaMemcpy(d, h, sizeof(double) * n, cudaMemcpyHostToDevice);
    return d;
}
static void down(int n, double *d, double *h) {
    if (h) cudaMemcpy(h, d, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
}
extern "C" int run_root(int n, const double *x, double *root, double *inv) {
    double *a = up(n, x), *b = up(n, nullptr), *c = up(n, nullptr);
    k_root<<<(n + 255) / 256, 256>>>(n, a, b, c);
    down(n, a, nullptr); down(n, b, root); down(n, c, inv);
    return (int)cudaGetLastError();
}
extern "C" int run_sincos(int n, const double *x, double *s, double *c) {
    if (bem::init_sincos_table() != cudaSuccess) return 1;
    double *a = up(n, x), *b = up(n, nullptr), *d = up(n, nullptr);
    k_sincos<<<(n + 255) / 256, 256>>>(n, a, b, d);
    down(n, a, nullptr); down(n, b, s); down(n, d, c);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("functions")
    src, so = str(d / "functions.cu"), str(d / "functions.so")
    with open(src, "w") as f:
        f.write(CODE)
    subprocess.run([build.nvcc(), "-shared", "-o", so, src, "-O3", "-std=c++17", *build.ARCH, "-Xcompiler", "-fPIC",
                    "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include")], check=True)
    return ctypes.CDLL(so)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_square_root(lib):
    rng = np.random.default_rng(1)
    x = np.ldexp(rng.uniform(1.0, 2.0, 1 << 20), rng.integers(-300, 301, 1 << 20))
    x[:64] = np.ldexp(1.0, np.arange(64) - 32)
    root, inv = np.zeros_like(x), np.zeros_like(x)
    assert lib.run_root(len(x), _p(x), _p(root), _p(inv)) == 0
    assert np.array_equal(root, np.sqrt(x))
    e = inv.astype(np.longdouble) * np.sqrt(x.astype(np.longdouble)) - 1
    unit = np.ldexp(1.0, np.frexp(inv)[1] - 53).astype(np.longdouble) / inv
    assert (np.abs(e) <= 1.5 * unit).all()


@pytest.mark.parametrize("large", [False, True])
def test_sine_and_cosine(lib, large):
    rng = np.random.default_rng(2)
    n = 1 << 16
    lo, hi = (43, 200) if large else (-20, 43)
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
    if not large:
        q = rng.integers(-4000, 4000, n // 2)
        x[: n // 2] = (q + 0.5 * (q & 1)) * (2 * np.pi / 1024)   # cells' centres and borders
        x[0] = 0.0
    s, c = np.zeros(n), np.zeros(n)
    assert lib.run_sincos(n, _p(x), _p(s), _p(c)) == 0
    for got, f in ((s, np.sin), (c, np.cos)):
        e = np.abs(got - f(x.astype(np.longdouble)))
        unit = np.ldexp(1.0, np.frexp(got)[1] - 53)
        assert (e <= (2 * unit if large else 0.5 * unit + 2.0**-58)).all()


@pytest.mark.parametrize("quad", [False, True])
def test_distances_beyond_the_table(quad):
    """Phases of 1e18: in double precision all points of a small element are at
    the same distance of a point 5e14 away, so its entries and fields there have
    the oracle's sizes, whatever the phase."""
    shape = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]] if quad else [[0, 0, 0], [1, 0, 0], [0, 1, 0]], float)
    c = len(shape)
    row = np.array([3e14, 0, 4e14]) + 1e3 * (shape + shape[:, [1, 2, 0]])
    v, k = np.concatenate([1e-4 * shape, row]), 2000.0
    pts = np.array([[-3e14, 0, 4e14], [1e14, 2e14, -5e14]])
    weak = dict(point_sources=[[5.0, 0, 0]], point_amps=[1e-60])
    for n in (2, 1):
        f = np.arange(n * c, dtype=np.int32).reshape(n, c)
        bcv = np.zeros((n, 4), complex)
        bcv[0, :c] = 1.0
        om, of = oracle.OracleMesh(v[: n * c], f, None, bcv), oracle.OracleFreq(k, *weak.values())
        m = capi.Mesh(v[: n * c], f)
        s = capi.Solver(m, precision=capi.PREC_FP64)
        s.assemble(capi.Frequency(k, n, bc_value=bcv, **weak))
        if n == 2:
            A, want = s.system()[0], oracle.assemble(om, of)[0]
            assert abs(abs(A[1, 0]) - abs(want[1, 0])) <= 1e-9 * abs(want[1, 0])
        else:
            s.solve()
            pot, grad = s.project(pts)
            q, g = oracle.project(om, of, *oracle.boundary_fields(om, s.solution()), pts)
            assert (abs(abs(pot) - abs(q)) <= 1e-9 * abs(q)).all()
            assert (abs(abs(grad) - abs(g)) <= 1e-9 * abs(g).max(axis=1)[:, None]).all()
        s.close()
        m.close()
