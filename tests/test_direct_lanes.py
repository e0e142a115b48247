"""The factorisation of a diagonal block of the direct solver (factor_diag)
must not depend on the order in which its threads run between two barriers:
its source, compiled for the host, runs 256 coroutines that switch only at a
barrier, in ascending, descending and shuffled order, and gives L U of the
block in each.  Bar: n u of an n x n elimination, growth included 8 n u, as in
test_direct_edges_gpu."""
import ctypes
import pathlib
import re
import subprocess

import numpy as np
import pytest

SRC = pathlib.Path(__file__).parent.parent / "mesh2hrtf_gb300" / "csrc" / "bem_direct.cu"

HOST = r"""
#include <ucontext.h>
#include <algorithm>
#include <cmath>
#include <random>
#include <vector>
using std::fma;
using std::min;
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
struct double2 { double x, y; };
struct { int x; } threadIdx;
constexpr int kPanel = 32, kThreads = 256;
static ucontext_t main_ctx, ctx[kThreads];
static void atomicExch(int *p, int v) { *p = v; }
static void __syncthreads() { swapcontext(&ctx[threadIdx.x], &main_ctx); }
@@CODE@@
template <typename V> struct Job { static V (*D)[kPanel + 1]; static int kb, status, done; };
template <typename V> V (*Job<V>::D)[kPanel + 1];
template <typename V> int Job<V>::kb;
template <typename V> int Job<V>::status;
template <typename V> int Job<V>::done;
template <typename V> static void entry() {
    factor_diag<V>(Job<V>::D, Job<V>::kb, &Job<V>::status);
    ++Job<V>::done;
    swapcontext(&ctx[threadIdx.x], &main_ctx);
}
template <typename V> static int run(V *d, int kb, int order) {
    static std::vector<char> stacks((size_t)kThreads << 16);
    Job<V>::D = reinterpret_cast<V (*)[kPanel + 1]>(d);
    Job<V>::kb = kb;
    Job<V>::status = Job<V>::done = 0;
    std::vector<int> lanes(kThreads);
    std::mt19937 rng(order);
    for (int t = 0; t < kThreads; ++t) {
        lanes[t] = order == 1 ? kThreads - 1 - t : t;
        getcontext(&ctx[t]);
        ctx[t].uc_stack.ss_sp = &stacks[(size_t)t << 16];
        ctx[t].uc_stack.ss_size = 1 << 16;
        ctx[t].uc_link = nullptr;
        makecontext(&ctx[t], entry<V>, 0);
    }
    while (Job<V>::done < kThreads) {
        if (order > 1) std::shuffle(lanes.begin(), lanes.end(), rng);
        for (int t : lanes) {
            threadIdx.x = t;
            swapcontext(&main_ctx, &ctx[t]);
        }
    }
    return Job<V>::status;
}
extern "C" int factor_f(float2 *d, int kb, int order) { return run(d, kb, order); }
extern "C" int factor_d(double2 *d, int kb, int order) { return run(d, kb, order); }
"""


def _function(text, name):
    """The source of template function `name`, its template line included."""
    at = text.index(" " + name + "(")
    start = text.rindex("template <typename V>", 0, at)
    i, depth = text.index("{", at), 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[start : j + 1]
    raise ValueError(name)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    text = SRC.read_text()
    code = "\n".join(_function(text, f) for f in ("cdiv", "cnma", "factor_diag"))
    code = re.sub(r"#pragma unroll.*", "", code)
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(HOST.replace("@@CODE@@", code))
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(d / "lanes.so"), str(d / "lanes.cpp")],
                   check=True)
    return ctypes.CDLL(str(d / "lanes.so"))


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("kb", [1, 2, 31, 32])
@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
def test_order_of_threads(lib, dt, kb, order):
    rng = np.random.default_rng(kb)
    a = rng.normal(size=(kb, kb)) + 1j * rng.normal(size=(kb, kb)) + 3 * kb * np.eye(kb)
    a = a.astype(dt)
    D = np.zeros((32, 33), dt)
    D[:kb, :kb] = a
    f = lib.factor_f if dt == np.complex64 else lib.factor_d
    assert f(D.ctypes.data_as(ctypes.c_void_p), kb, order) == 0
    lu = D[:kb, :kb].astype(np.complex128)
    L, U = np.tril(lu, -1) + np.eye(kb), np.triu(lu)
    u = 2.0 ** -24 if dt == np.complex64 else 2.0 ** -53
    assert np.linalg.norm(L @ U - a) <= 8 * kb * u * np.linalg.norm(a, 2)


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
def test_an_update_rounds_once_at_the_entry(lib, dt):
    """a - l u with |l u| far below |a| is within half a unit of a, and three
    roundings of the product (two in it, one for a unit that the difference
    may drop to), of its value."""
    f = lib.factor_f if dt == np.complex64 else lib.factor_d
    u = 2.0 ** -24 if dt == np.complex64 else 2.0 ** -53
    rng = np.random.default_rng(8)
    for _ in range(300):
        D = np.zeros((32, 33), dt)
        off = 0.03 * (rng.normal(size=2) + 1j * rng.normal(size=2))
        a = np.array([[1 + 1j, off[0]], [off[1], 1.5 + 1.5j]]).astype(dt)
        D[:2, :2] = a
        assert f(D.ctypes.data_as(ctypes.c_void_p), 2, 0) == 0
        l, d = D[1, 0].astype(np.clongdouble), D[1, 1].astype(np.clongdouble)
        p = l * a[0, 1].astype(np.clongdouble)
        e = d - (a[1, 1].astype(np.clongdouble) - p)
        assert max(abs(e.real), abs(e.imag)) <= u + 3 * u * abs(p)   # half a unit in [1, 2)
