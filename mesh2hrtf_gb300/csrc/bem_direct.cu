// bem_direct.cu - dense direct solve of the assembled system: LU without
// pivoting in place, then forward and back substitution, as NumCalc does when
// NC.inp asks for Gaussian elimination (ISOLVER 4) or when CGS fails
// (Tfactor_usy / Tfbelim, NC_TypeDefinition.h:543-594, called from
// NC_IterativeSolverCGS, NC_CommonFunctions.cpp:1181-1191).
//
// Blocked right-looking factorisation A = L U (L unit lower, U upper) in the
// matrix's own precision (complex128 for FP64 solvers, complex64 for mixed
// ones), in panels of kPanel columns, two launches per panel:
//   k_lu_panel   L21 = A21 U11^-1 (8 lanes per row), U12 = L11^-1 A12 (8 lanes
//                per column), and the panel's step of the forward
//                substitution, from the factored diagonal block
//   k_lu_update  A22 -= L21 U12, 64 x 64 output tiles through shared memory,
//                and the right-hand sides' remaining rows; the block that
//                owns the next diagonal block factors it as soon as it is
//                updated, beside the other tiles
// The forward substitution rides along in FP64; the back substitution takes
// one launch per panel (k_bwd): every block solves the 32 x 32 triangle
// (a warp, lane per row) and updates its own rows, so no launch waits on a
// single-thread solve.  Like the reference, no pivoting: a zero pivot is
// reported, not worked around.
//
// What bounds it: the launch-to-launch chain of n / 32 panels below a few
// thousand unknowns, the update's FP32 (FP64) arithmetic above.  Before, a
// launch per pivot column (uncoalesced row walks) and one-thread diagonal
// solves took 88.8 ms at 2420 unknowns in complex64; this form takes
// 5.0 ms.
#include <cuda_runtime.h>

#include "../../include/bem_gb300.h"
#include "bem_solver.h"

namespace {

constexpr int kPanel = 32;
constexpr int kTile = 64;
// columns of L21 / rows of U12 staged at a time
template <typename V> constexpr int kChunk = sizeof(V) == 8 ? 32 : 16;
constexpr int kMaxB = bem::kMaxRhs;
constexpr int kRowsPerBwd = kPanel;    // k_bwd: rows per block, 8 lanes each

__device__ __forceinline__ double2 ld2(const double2 &v) { return v; }
__device__ __forceinline__ double2 ld2(const float2 &v) { return make_double2(v.x, v.y); }
template <typename V>
__device__ __forceinline__ V cmul(V a, V b) {
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <typename V>
__device__ __forceinline__ V csub(V a, V b) {
    V r;
    r.x = a.x - b.x;
    r.y = a.y - b.y;
    return r;
}
// a / b as the reference's Complex::operator/ forms it
template <typename V>
__device__ __forceinline__ V cdiv(V a, V b) {
    const auto t = b.x * b.x + b.y * b.y;
    V r;
    r.x = (a.x * b.x + a.y * b.y) / t;
    r.y = (a.y * b.x - a.x * b.y) / t;
    return r;
}

// a - b c, the product formed first: one rounding at the size of a, which on
// the heavy diagonal is far larger than the product (two fused updates of a
// round there twice: complex64, 130 unknowns, solutions 1.8e-7 .. 2.7e-7 from
// the exact ones against 1.3e-7 .. 1.6e-7; 2420 unknowns took 0.2 ms less)
template <typename V>
__device__ __forceinline__ V cnma(V a, V b, V c) {
    const auto re = fma(-b.y, c.y, b.x * c.x), im = fma(b.x, c.y, b.y * c.x);
    a.x -= re;
    a.y -= im;
    return a;
}

// Right-hand sides of the substitutions: y in (updated in place), z the
// forward result.
struct Rhs {
    int count;
    double2 *y[kMaxB], *z[kMaxB];
};

// Factor the kb x kb block D in shared memory (L below the diagonal, U on and
// above it), 256 threads: thread t holds row t / 8, columns t % 8 + 8 q in
// registers.  Step i needs row i and column i of the block as step i - 1 left
// them, which their owners publish in D; one barrier per step.
template <typename V>
__device__ void factor_diag(V (*D)[kPanel + 1], int kb, int *status) {
    const int r = threadIdx.x >> 3, c0 = threadIdx.x & 7;
    V a[kPanel / 8];
#pragma unroll
    for (int q = 0; q < kPanel / 8; ++q) a[q] = D[r][c0 + 8 * q];
#pragma unroll
    for (int p = 0; p < kPanel / 8; ++p) {
        // rolled: straight-line code for all 32 steps would be fetched once
        // per instruction from beyond the instruction cache
#pragma unroll 1
        for (int i = 8 * p; i < 8 * p + 8 && i < kb; ++i) {
            const V piv = D[i][i];
            if (threadIdx.x == 0 && piv.x == 0 && piv.y == 0) atomicExch(status, 1);
            if (r > i && r < kb) {
                const V l = cdiv(D[r][i], piv);
                if (c0 == (i & 7)) a[p] = l;
#pragma unroll
                for (int q = p; q < kPanel / 8; ++q) {
                    const int c = c0 + 8 * q;
                    if (c > i) {
                        a[q] = cnma(a[q], l, D[i][c]);
                        // only what step i + 1 reads: column i of row i + 1 is
                        // still being read by the row's other lanes
                        if (c == i + 1 || r == i + 1) D[r][c] = a[q];
                    }
                }
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int q = 0; q < kPanel / 8; ++q) D[r][c0 + 8 * q] = a[q];
    __syncthreads();
}

// the first diagonal block (later ones are factored by k_lu_update)
template <typename V>
__global__ void __launch_bounds__(256) k_lu_diag(V *A, size_t lda, int k0, int kb, int *status) {
    __shared__ V D[kPanel][kPanel + 1];
    for (int t = threadIdx.x; t < kb * kb; t += 256) D[t / kb][t % kb] = A[(size_t)(k0 + t / kb) * lda + k0 + t % kb];
    __syncthreads();
    factor_diag(D, kb, status);
    for (int t = threadIdx.x; t < kb * kb; t += 256) A[(size_t)(k0 + t / kb) * lda + k0 + t % kb] = D[t / kb][t % kb];
}

// Blocks [0, nt): 32 rows of L21 each; [nt, 2 nt): 32 columns of U12 each; the
// last block: z = L11^-1 y of every right-hand side (a warp each, FP64).  Eight
// lanes share a row (column): lane g holds entries g, g + 8, ... and the entry
// solved in a step goes round by shuffle, so no step needs a barrier and the
// loops stay short enough for the instruction cache (one thread per row with
// 32 unrolled steps took 50 us per launch, most of it instruction fetches).
template <typename V>
__device__ __forceinline__ V shfl8(V v, int src) {
    v.x = __shfl_sync(0xffffffffu, v.x, src, 8);
    v.y = __shfl_sync(0xffffffffu, v.y, src, 8);
    return v;
}

template <typename V>
__global__ void __launch_bounds__(256) k_lu_panel(V *A, size_t lda, int n, int k0, int kb, int nt, Rhs rhs) {
    __shared__ V D[kPanel][kPanel + 1], T[kPanel][kPanel + 1];
    constexpr int Q = kPanel / 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k1 = k0 + kb;
    const int blk = (int)blockIdx.x;
    const bool rows = blk < nt, ycol = blk == 2 * nt;
    const int j0 = k1 + (rows ? blk : blk - nt) * kPanel;   // first row or column of the block
    // the diagonal block and the block's own rows or columns, every load
    // issued before the first is used
    V d[Q], u[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int r = warp + 8 * q;
        d[q].x = d[q].y = u[q].x = u[q].y = 0;
        if (r < kb && lane < kb) d[q] = A[(size_t)(k0 + r) * lda + k0 + lane];
        if (rows) {
            if (j0 + r < n && lane < kb) u[q] = A[(size_t)(j0 + r) * lda + k0 + lane];
        } else if (!ycol) {
            if (r < kb && j0 + lane < n) u[q] = A[(size_t)(k0 + r) * lda + j0 + lane];
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        D[warp + 8 * q][lane] = d[q];
        T[warp + 8 * q][lane] = u[q];
    }
    __syncthreads();
    if (ycol) {
        for (int q = warp; q < rhs.count; q += 8) {
            double2 yv = lane < kb ? rhs.y[q][k0 + lane] : make_double2(0.0, 0.0);
#pragma unroll 4
            for (int i = 0; i < kPanel; ++i) {
                const double2 yi = make_double2(__shfl_sync(0xffffffffu, yv.x, i), __shfl_sync(0xffffffffu, yv.y, i));
                if (lane > i && lane < kb) yv = cnma(yv, ld2(D[lane][i]), yi);
            }
            if (lane < kb) rhs.z[q][k0 + lane] = yv;
        }
        return;
    }
    const int m = threadIdx.x >> 3, g = threadIdx.x & 7;   // row (column) of the tile, lane of its eight
    if (rows) {
#pragma unroll
        for (int q = 0; q < Q; ++q) u[q] = T[m][g + 8 * q];
#pragma unroll
        for (int p = 0; p < Q; ++p) {
#pragma unroll 1
            for (int i = 8 * p; i < 8 * p + 8 && i < kb; ++i) {
                const V l = cdiv(shfl8(u[p], i & 7), D[i][i]);
                if (g == (i & 7)) u[p] = l;
#pragma unroll
                for (int q = p; q < Q; ++q)
                    if (g + 8 * q > i) u[q] = cnma(u[q], l, D[i][g + 8 * q]);
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) T[m][g + 8 * q] = u[q];
    } else {
#pragma unroll
        for (int q = 0; q < Q; ++q) u[q] = T[g + 8 * q][m];
#pragma unroll
        for (int p = 0; p < Q; ++p) {
#pragma unroll 1
            for (int i = 8 * p; i < 8 * p + 8 && i < kb; ++i) {
                const V ui = shfl8(u[p], i & 7);
#pragma unroll
                for (int q = p; q < Q; ++q)
                    if (g + 8 * q > i) u[q] = cnma(u[q], D[g + 8 * q][i], ui);
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) T[g + 8 * q][m] = u[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int r = warp + 8 * q;
        if (rows) {
            if (j0 + r < n && lane < kb) A[(size_t)(j0 + r) * lda + k0 + lane] = T[r][lane];
        } else {
            if (r < kb && j0 + lane < n) A[(size_t)(k0 + r) * lda + j0 + lane] = T[r][lane];
        }
    }
}

// A22 -= L21 U12 over the trailing block [k1, n) x [k1, n), k1 = k0 + kb;
// 64 x 64 output tiles, 256 threads with 4 x 4 entries each (rows ty + 16 a,
// columns tx + 16 b: whole-segment global accesses, no bank conflicts).  The
// tile at (k1, k1) then factors the next panel's diagonal block; the tiles of
// the first column also update the right-hand sides' rows, y -= L21 z.
template <typename V>
__global__ void __launch_bounds__(256) k_lu_update(V *A, size_t lda, int n, int k0, int kb, Rhs rhs, int *status) {
    constexpr int CH = kChunk<V>;
    constexpr int kStage = CH * (2 * kTile + 1), kDiag = kPanel * (kPanel + 1);
    __shared__ __align__(16) unsigned char sm[sizeof(V) * (kStage > kDiag ? kStage : kDiag)];
    V (*Ls)[kTile + 1] = reinterpret_cast<V (*)[kTile + 1]>(sm);                                // [CH][row]
    V (*Us)[kTile] = reinterpret_cast<V (*)[kTile]>(sm + sizeof(V) * CH * (kTile + 1));      // [CH][column]
    const int k1 = k0 + kb;
    const int j0 = k1 + blockIdx.y * kTile, c0 = k1 + blockIdx.x * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    V acc[4][4], old[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            acc[a][b].x = acc[a][b].y = 0;
            const int j = j0 + ty + 16 * a, c = c0 + tx + 16 * b;
            old[a][b].x = old[a][b].y = 0;
            if (j < n && c < n) old[a][b] = A[(size_t)j * lda + c];
        }
    for (int kk = 0; kk < kb; kk += CH) {
#pragma unroll
        for (int t = threadIdx.x; t < kTile * CH; t += 256) {
            const int r = t / CH, q = t % CH;
            V v;
            v.x = v.y = 0;
            if (j0 + r < n && kk + q < kb) v = A[(size_t)(j0 + r) * lda + k0 + kk + q];
            Ls[q][r] = v;
        }
#pragma unroll
        for (int t = threadIdx.x; t < kTile * CH; t += 256) {
            const int q = t / kTile, r = t % kTile;
            V v;
            v.x = v.y = 0;
            if (c0 + r < n && kk + q < kb) v = A[(size_t)(k0 + kk + q) * lda + c0 + r];
            Us[q][r] = v;
        }
        __syncthreads();
#pragma unroll 4
        for (int q = 0; q < CH; ++q) {
            V lv[4], uv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) lv[a] = Ls[q][ty + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) uv[b] = Us[q][tx + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    acc[a][b].x = fma(lv[a].x, uv[b].x, acc[a][b].x);
                    acc[a][b].x = fma(-lv[a].y, uv[b].y, acc[a][b].x);
                    acc[a][b].y = fma(lv[a].x, uv[b].y, acc[a][b].y);
                    acc[a][b].y = fma(lv[a].y, uv[b].x, acc[a][b].y);
                }
        }
        __syncthreads();
    }
    const bool first = blockIdx.x == 0 && blockIdx.y == 0;
    const int nb = min(kPanel, n - k1);   // the next diagonal block
    V (*D)[kPanel + 1] = reinterpret_cast<V (*)[kPanel + 1]>(sm);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a, j = j0 + r;
        if (j >= n) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int q = tx + 16 * b, c = c0 + q;
            if (c >= n) continue;
            const V v = csub(old[a][b], acc[a][b]);
            if (first && r < nb && q < nb) D[r][q] = v;
            else A[(size_t)j * lda + c] = v;
        }
    }
    if (blockIdx.x == 0) {
        // y -= L21 z: 4 lanes per row, 8 columns each
        const int r = threadIdx.x >> 2, g = threadIdx.x & 3, j = j0 + r;
        for (int q = 0; q < rhs.count; ++q) {
            double2 s = make_double2(0.0, 0.0);
            if (j < n)
                for (int i = g; i < kb; i += 4) {
                    const double2 l = ld2(A[(size_t)j * lda + k0 + i]), z = rhs.z[q][k0 + i];
                    s.x += l.x * z.x - l.y * z.y;
                    s.y += l.x * z.y + l.y * z.x;
                }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            }
            if (g == 0 && j < n) rhs.y[q][j] = csub(rhs.y[q][j], s);
        }
    }
    if (first) {
        __syncthreads();
        factor_diag(D, nb, status);
        for (int t = threadIdx.x; t < nb * nb; t += 256) A[(size_t)(k1 + t / nb) * lda + k1 + t % nb] = D[t / nb][t % nb];
    }
}

// Back substitution of one panel: every block solves U11 x = z[k0 .. k0 + kb)
// (warp 0, lane per row; block 0 keeps the result) and takes x out of its own
// kRowsPerBwd rows above, 8 lanes per row with 4 columns each, whose entries
// of U are loaded before the triangle is solved.  blockIdx.y: right-hand side.
template <typename V>
__global__ void __launch_bounds__(8 * kRowsPerBwd) k_bwd(const V *A, size_t lda, int k0, int kb, Rhs rhs) {
    __shared__ V D[kPanel][kPanel + 1];
    __shared__ double2 xs[kPanel];
    double2 *z = rhs.z[blockIdx.y], *x = rhs.y[blockIdx.y];
    const int t = threadIdx.x, r = t >> 3, g = t & 7;
    const int j = blockIdx.x * kRowsPerBwd + r;
    const bool row = j < k0;
    V u[kPanel / 8];
#pragma unroll
    for (int q = 0; q < kPanel / 8; ++q) {
        u[q].x = u[q].y = 0;
        if (row && g + 8 * q < kb) u[q] = A[(size_t)j * lda + k0 + g + 8 * q];
    }
#pragma unroll
    for (int q = 0; q < kPanel / 8; ++q) {
        const int c = g + 8 * q;
        V v;
        v.x = v.y = 0;
        if (r < kb && c < kb) v = A[(size_t)(k0 + r) * lda + k0 + c];
        D[r][c] = v;
    }
    __syncthreads();
    if (t < 32) {
        // rows scaled by their pivots' inverses first, so that a step of the
        // solve is one fused update
        double2 v = t < kb ? z[k0 + t] : make_double2(0.0, 0.0);
        const double2 one = make_double2(1.0, 0.0);
        const double2 inv = t < kb ? cdiv(one, ld2(D[t][t])) : one;
        v = cmul(v, inv);
#pragma unroll 8
        for (int i = kPanel - 1; i >= 0; --i) {
            const double2 f = cmul(ld2(D[t][i]), inv);
            const double2 xi = make_double2(__shfl_sync(0xffffffffu, v.x, i), __shfl_sync(0xffffffffu, v.y, i));
            if (t < i && i < kb) v = cnma(v, f, xi);
        }
        if (t < kb) {
            xs[t] = v;
            if (blockIdx.x == 0) x[k0 + t] = v;
        }
    }
    __syncthreads();
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < kPanel / 8; ++q) {
        if (g + 8 * q >= kb) break;
        const double2 l = ld2(u[q]), xv = xs[g + 8 * q];
        s.x += l.x * xv.x - l.y * xv.y;
        s.y += l.x * xv.y + l.y * xv.x;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    if (g == 0 && row) z[j] = csub(z[j], s);
}

// A = L U in place and z = L^-1 y, then y = U^-1 z
template <typename V>
cudaError_t factor_and_solve(V *A, size_t lda, int n, const Rhs &rhs, int *status, cudaStream_t st) {
    long long launches = 1;
    k_lu_diag<V><<<1, 256, 0, st>>>(A, lda, 0, min(kPanel, n), status);
    for (int k0 = 0; k0 < n; k0 += kPanel) {
        const int kb = min(kPanel, n - k0), rest = n - k0 - kb;
        const int nt = (rest + kPanel - 1) / kPanel;
        k_lu_panel<V><<<2 * nt + 1, 256, 0, st>>>(A, lda, n, k0, kb, nt, rhs);
        ++launches;
        if (rest > 0) {
            const int t = (rest + kTile - 1) / kTile;
            k_lu_update<V><<<dim3(t, t), 256, 0, st>>>(A, lda, n, k0, kb, rhs, status);
            ++launches;
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    for (int k0 = ((n - 1) / kPanel) * kPanel; k0 >= 0; k0 -= kPanel) {
        const int kb = min(kPanel, n - k0);
        const dim3 grid(k0 > 0 ? (k0 + kRowsPerBwd - 1) / kRowsPerBwd : 1, rhs.count);
        k_bwd<V><<<grid, 8 * kRowsPerBwd, 0, st>>>(A, lda, k0, kb, rhs);
        ++launches;
    }
    bem::count_launches(launches);
    return cudaGetLastError();
}

}  // namespace

extern "C" bem_status bem_solve_direct(bem_solver_t s, bem_solve_info *info) {
    if (!s) return bem::fail(BEM_ERR_INVALID, "null solver");
    if (!s->have_freq) return bem::fail(BEM_ERR_INVALID, "bem_solve_direct before bem_assemble");
    if (s->factored) return bem::fail(BEM_ERR_INVALID, "bem_solve_direct: the matrix is already factored; assemble again");
    if (cudaSetDevice(s->mesh->device) != cudaSuccess) return bem::fail(BEM_ERR_CUDA, "cudaSetDevice failed");
    cudaStream_t st = s->st;
    const int n = s->n;
    BEM_CU(cudaMemsetAsync(s->d.status, 0, sizeof(int), st));
    BEM_CU(cudaEventRecord(s->ev[2], st));
    Rhs rhs{};
    rhs.count = s->n_rhs;
    for (int r = 0; r < s->n_rhs; ++r) {
        const bem::SolverBufs &d = s->buf(r);
        BEM_CU(cudaMemcpyAsync(d.x, d.b, sizeof(double2) * n, cudaMemcpyDeviceToDevice, st));
        rhs.y[r] = d.x;
        rhs.z[r] = d.r;   // the residual vector, idle here
    }
    if (s->prec == BEM_PREC_FP64) BEM_CU(factor_and_solve((double2 *)s->d.A, s->lda, n, rhs, s->d.status, st));
    else BEM_CU(factor_and_solve((float2 *)s->d.A, s->lda, n, rhs, s->d.status, st));
    BEM_CU(cudaEventRecord(s->ev[3], st));
    int zero_pivot = 0;
    BEM_CU(cudaMemcpyAsync(&zero_pivot, s->d.status, sizeof(int), cudaMemcpyDeviceToHost, st));
    BEM_CU(cudaStreamSynchronize(st));
    float ms = 0.f;
    BEM_CU(cudaEventElapsedTime(&ms, s->ev[2], s->ev[3]));
    s->factored = true;
    s->solved = true;
    s->info.iterations = 0;
    s->info.restarts = 0;
    s->info.rel_residual = 0.0;
    s->info.solve_ms = ms;
    s->info.matvec_ms = 0.0;
    s->info.n_matvec = 0;
    if (info) *info = s->info;
    if (zero_pivot) return bem::fail(BEM_ERR_INVALID, "bem_solve_direct: zero pivot (LU without pivoting)");
    return BEM_OK;
}
