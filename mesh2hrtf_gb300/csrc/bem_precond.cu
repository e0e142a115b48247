// bem_precond.cu - block-Jacobi preconditioner for the GMRES of bem_solve.
//
// The library numbers the unknowns along a Morton (Z-order) curve of the
// element centres, so consecutive unknowns are spatial neighbours and the
// diagonal blocks of A hold the strongest (near-field) couplings.  The
// preconditioner is the block diagonal of A with blocks of kBlock unknowns,
// inverted once per frequency; NumCalc's own preconditioner is a threshold
// ILU on the same near-field entries (NC_CommonFunctions.cpp:1357-1721).
// By default the Krylov kernels apply it with one correction step over
// windows of kPcWin unknowns, M = X (2 I - A_w X) (bem_gmres.cu), which
// needs no further set-up.
//
// Inversion: in-place Gauss-Jordan with partial pivoting, one block of kBlock
// rows per CTA or per cluster of CTAs that share its columns, entries in
// registers (gauss_jordan_one, gauss_jordan_cluster); the last, partial block of a system goes through shared
// memory or a global workspace (gauss_jordan).  Inverses are stored transposed
// so that the application (inside the Krylov kernels, bem_gmres.cu) reads them
// coalesced.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "bem_internal.h"

namespace bem {
namespace {

template <typename T> struct C2;
template <> struct C2<float> { using t = float2; };
template <> struct C2<double> { using t = double2; };

template <typename V> __device__ __forceinline__ V cmul2(V a, V b) {
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <typename V> __device__ __forceinline__ V cinv2(V a) {
    // 1/a, scaled to avoid overflow
    auto s = fabs(a.x) > fabs(a.y) ? fabs(a.x) : fabs(a.y);
    decltype(s) ar = a.x / s, ai = a.y / s, d = ar * ar + ai * ai;
    V r;
    r.x = ar / (d * s);
    r.y = -ai / (d * s);
    return r;
}

// The same with one division, for a chain that waits for it: scaled by a power
// of two (exact) instead of the larger component.
__device__ __forceinline__ float2 cinv_pow2(float2 a) {
    const int e = (int)((__float_as_uint(fmaxf(fabsf(a.x), fabsf(a.y))) >> 23) & 255u);   // biased exponent
    const float s = __uint_as_float((unsigned)min(max(254 - e, 1), 254) << 23);
    const float ar = a.x * s, ai = a.y * s, q = s / fmaf(ar, ar, ai * ai);
    return make_float2(ar * q, -ai * q);
}
__device__ __forceinline__ double2 cinv_pow2(double2 a) {
    const int e = (__double2hiint(fmax(fabs(a.x), fabs(a.y))) >> 20) & 2047;
    const double s = __hiloint2double(min(max(2046 - e, 1), 2046) << 20, 0);
    const double ar = a.x * s, ai = a.y * s, q = s / fma(ar, ar, ai * ai);
    return make_double2(ar * q, -ai * q);
}

// In-place Gauss-Jordan on the nb x nb block W (row-major, leading dim ld),
// executed by one CTA.  colk: nb scratch, piv: nb ints.
template <typename T>
__device__ void gauss_jordan(typename C2<T>::t *W, int ld, int nb, typename C2<T>::t *colk, int *piv,
                             int *pivrow, int *singular) {
    using V = typename C2<T>::t;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int k = 0; k < nb; ++k) {
        // pivot search by warp 0
        if (tid < 32) {
            T best = -1;
            int bi = k;
            for (int i = k + tid; i < nb; i += 32) {
                V a = W[(size_t)i * ld + k];
                T m = a.x * a.x + a.y * a.y;
                if (m > best) { best = m; bi = i; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                T ob = __shfl_down_sync(0xffffffffu, best, o);
                int oi = __shfl_down_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            if (tid == 0) {
                *pivrow = bi;
                piv[k] = bi;
                if (!(best > 0)) *singular = 1;
            }
        }
        __syncthreads();
        const int p = *pivrow;
        if (p != k)
            for (int j = tid; j < nb; j += nt) {
                V t = W[(size_t)k * ld + j];
                W[(size_t)k * ld + j] = W[(size_t)p * ld + j];
                W[(size_t)p * ld + j] = t;
            }
        __syncthreads();
        const V inv = cinv2(W[(size_t)k * ld + k]);
        for (int i = tid; i < nb; i += nt) colk[i] = W[(size_t)i * ld + k];
        __syncthreads();
        for (int j = tid; j < nb; j += nt) {
            V a = j == k ? V{1, 0} : W[(size_t)k * ld + j];
            W[(size_t)k * ld + j] = cmul2(a, inv);
        }
        __syncthreads();
        for (int e = tid; e < nb * nb; e += nt) {
            const int i = e / nb, j = e - i * nb;
            if (i == k) continue;
            const V f = colk[i];
            V a = j == k ? V{0, 0} : W[(size_t)i * ld + j];
            const V r = W[(size_t)k * ld + j];
            a.x -= f.x * r.x - f.y * r.y;
            a.y -= f.x * r.y + f.y * r.x;
            W[(size_t)i * ld + j] = a;
        }
        __syncthreads();
    }
    // undo the row interchanges as column interchanges, last first
    for (int k = nb - 1; k >= 0; --k) {
        const int p = piv[k];
        if (p != k)
            for (int i = tid; i < nb; i += nt) {
                V t = W[(size_t)i * ld + k];
                W[(size_t)i * ld + k] = W[(size_t)i * ld + p];
                W[(size_t)i * ld + p] = t;
            }
        __syncthreads();
    }
}

// The pivot of a column (v[q]: row lane + 32 q) by one warp: the largest |a|^2
// among the rows not in used, lowest row on ties; nothing comparable (zero or
// NaN) sets singular, and the lowest unused row serves.  Marks the row used.
template <typename V>
__device__ __forceinline__ int warp_pivot(const V (&v)[kBlock / 32], int lane, unsigned &used, int &singular) {
    decltype(v[0].x + v[0].x) best = -1;
    int p = kBlock;
#pragma unroll
    for (int q = 0; q < kBlock / 32; ++q) {
        const auto m = v[q].x * v[q].x + v[q].y * v[q].y;
        if (!((used >> q) & 1u) && m > best) {
            best = m;
            p = lane + 32 * q;
        }
    }
    if constexpr (sizeof(best) == 4) {
        // as whole numbers, in the same order: 0 for no candidate, else |a|^2's bits + 1
        const unsigned key = p < kBlock ? __float_as_uint(best) + 1u : 0u, top = __reduce_max_sync(0xffffffffu, key);
        p = (int)__reduce_min_sync(0xffffffffu, key == top ? (unsigned)p : (unsigned)kBlock);
        best = top > 0u ? __uint_as_float(top - 1u) : -1.f;
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const auto ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, p, o);
            if (ob > best || (ob == best && oi < p)) { best = ob; p = oi; }
        }
    }
    if (!(best > 0)) {
        if (lane == 0) singular = 1;
        if (p >= kBlock) {
            int cand = kBlock;
#pragma unroll
            for (int q = kBlock / 32 - 1; q >= 0; --q)
                if (!((used >> q) & 1u)) cand = lane + 32 * q;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cand = min(cand, __shfl_xor_sync(0xffffffffu, cand, o));
            p = cand;
        }
    }
    if (lane == (p & 31)) used |= 1u << (p >> 5);
    return p;
}

// a - f r, in the order of operations of every step
template <typename V> __device__ __forceinline__ V gj_update(V a, V f, V r) {
    a.x = fma(-f.x, r.x, a.x);
    a.x = fma(f.y, r.y, a.x);
    a.y = fma(-f.x, r.y, a.y);
    a.y = fma(-f.y, r.x, a.y);
    return a;
}

// The same on a full kBlock x kBlock block held in registers by one CTA: thread
// t of NT has columns t % C + c C (C = kBlock / NC) at rows kR (t / C) .. +
// kR - 1.  A step
// needs the pivot column, the pivot with its inverse, and the pivot row
// (published by the threads that hold it).  Rows are not interchanged: step k's
// pivot is the largest |a|^2 among the rows not used yet, lowest row on ties,
// and with p_k its row the inverse is Ainv[k][p_c] = W[p_k][c].
//
// Warp 0 looks a step ahead: while the others update, it forms the next column
// from its entries of the step before (published by their threads), finds its
// pivot and inverts it, which needed a barrier of its own.  The column's factors
// are loaded two rows at a time and serve NC columns: one column to a thread was
// bound by those loads.  complex64, up to 152 blocks: 204 us as below on one
// CTA, 199 with the look-ahead, 162 with two columns to a thread, 146 with the
// pivot found by whole-number reductions; 1280 blocks 1.83 -> 1.34 ms.  What is
// left is warp 0's chain.
template <typename T, int NT, int NC>
__device__ void gauss_jordan_one(const typename C2<T>::t *A, size_t lda, typename C2<T>::t *out, int *status) {
    using V = typename C2<T>::t;
    constexpr int C = kBlock / NC, G = NT / C, kR = kBlock / G;
    static_assert(G * kR == kBlock && C % 32 == 0 && kR % 2 == 0, "threads cover the block, a warp one row group");
    __shared__ __align__(16) V fcol[2][kBlock];   // the step's pivot column, by step parity
    __shared__ __align__(16) V prev[2][kBlock];   // the next column before the step
    __shared__ V rowb[kBlock], inv_s;
    __shared__ int piv[kBlock], singular_s;
    const int tid = threadIdx.x, lane = tid & 31, j = tid % C, i0 = tid / C * kR;
    V a[NC][kR];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < kR; ++q) a[c][q] = A[(size_t)(i0 + q) * lda + j + c * C];
    if (j < 2) {
#pragma unroll
        for (int q = 0; q < kR; ++q) (j == 0 ? fcol[0] : prev[1])[i0 + q] = a[0][q];
    }
    if (tid == 0) singular_s = 0;
    __syncthreads();
    unsigned used = 0;   // warp 0, bit q: row lane + 32 q has been a pivot row
    auto pivot = [&](int k, const V (&v)[kBlock / 32]) {
        const int p = warp_pivot(v, lane, used, singular_s);
        V b = v[0];
#pragma unroll
        for (int q = 1; q < kBlock / 32; ++q)
            if ((p >> 5) == q) b = v[q];
        if (lane == (p & 31)) {
            piv[k] = p;
            inv_s = cinv_pow2(b);
        }
    };
    if (tid < 32) {
        V v[kBlock / 32];
#pragma unroll
        for (int q = 0; q < kBlock / 32; ++q) v[q] = fcol[0][lane + 32 * q];
        pivot(0, v);
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < kBlock; ++k) {
        const V *f = fcol[k & 1];
        const int p = piv[k] - i0;   // the pivot row among this warp's rows
        // the pivot row, scaled (its own column: 1 / pivot)
        if (p >= 0 && p < kR) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                V r = a[c][0];
#pragma unroll
                for (int q = 1; q < kR; ++q)
                    if (p == q) r = a[c][q];
                if (j + c * C == k) { r.x = 1; r.y = 0; }
                rowb[j + c * C] = cmul2(r, inv_s);
            }
        }
        __syncthreads();
        if (tid < 32 && k + 1 < kBlock) {
            const V r = rowb[k + 1];
            V v[kBlock / 32];
#pragma unroll
            for (int q = 0; q < kBlock / 32; ++q) {
                const int i = lane + 32 * q;
                v[q] = gj_update(prev[(k + 1) & 1][i], f[i], r);
                if (i == piv[k]) v[q] = r;
                fcol[(k + 1) & 1][i] = v[q];
            }
            pivot(k + 1, v);
        }
        V r[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            r[c] = rowb[j + c * C];
            if (((j + c * C) >> 5) == (k >> 5)) {   // the warps with column k
                if (j + c * C == k) {
#pragma unroll
                    for (int q = 0; q < kR; ++q) a[c][q].x = a[c][q].y = 0;
                }
            }
        }
        const float4 *f2 = reinterpret_cast<const float4 *>(f + i0);   // two rows to a load
        static_assert(sizeof(V) == 8, "complex64");
#pragma unroll
        for (int q = 0; q < kR; q += 2) {
            const float4 ff = f2[q / 2];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                a[c][q] = gj_update(a[c][q], make_float2(ff.x, ff.y), r[c]);
                a[c][q + 1] = gj_update(a[c][q + 1], make_float2(ff.z, ff.w), r[c]);
            }
        }
        if (p >= 0 && p < kR) {
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int q = 0; q < kR; ++q)
                    if (p == q) a[c][q] = r[c];
        }
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (j + c * C == k + 2) {
#pragma unroll
                for (int q = 0; q < kR; ++q) prev[k & 1][i0 + q] = a[c][q];
            }
        __syncthreads();
    }
    // row i was the pivot of step inv_p(i), column j holds the inverse's column
    // p_j: Minv[c][r] (transposed) with r the step, c = piv[j]
    int *step = reinterpret_cast<int *>(rowb);
    if (tid < kBlock) step[piv[tid]] = tid;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < kR; ++q) out[(size_t)piv[j + c * C] * kBlock + step[i0 + q]] = a[c][q];
    if (tid == 0 && singular_s) atomicMax(status, 1);
}

// The same by CL CTAs of a cluster: CTA r has the columns r kBlock / CL .. .
// The pivot column is published by the threads that hold it as soon as the step
// before has updated it, in one of two buffers, and the other CTAs fetch it
// through distributed shared memory; every CTA finds the pivot for itself.
// For complex128, which an SM's narrow FP64 pipe bounds (4 FMA per entry and
// step): 40 blocks 3.9 ms in an L2 workspace, 1.24 ms over four SMs each.
template <typename T, int CL, int NT>
__device__ void gauss_jordan_cluster(const typename C2<T>::t *A, size_t lda, typename C2<T>::t *out, int *status) {
    using V = typename C2<T>::t;
    constexpr int C = kBlock / CL, G = NT / C, kR = kBlock / G;
    static_assert(G * kR == kBlock && C % 32 == 0, "threads cover the block, a warp one row group");
    __shared__ __align__(16) V colb[2][kBlock];       // pivot column, by step parity (own CTA's threads)
    __shared__ V col[kBlock];   // the pivot column fetched from its CTA
    __shared__ V rowb[C], inv_s;
    __shared__ int piv[kBlock], singular_s;
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int j = tid % C, i0 = tid / C * kR, jg = (int)rank * C + j;   // own column (in the CTA, in the block)
    V a[kR];
#pragma unroll
    for (int q = 0; q < kR; ++q) a[q] = A[(size_t)(i0 + q) * lda + jg];
    if (jg == 0) {
#pragma unroll
        for (int q = 0; q < kR; ++q) colb[0][i0 + q] = a[q];
    }
    unsigned used = 0;   // warp 0, bit q: row lane + 32 q has been a pivot row
    if (tid == 0) singular_s = 0;
#pragma unroll 1
    for (int k = 0; k < kBlock; ++k) {
        // the column is complete in its CTA, and the others are done with
        // the buffer of two steps ago
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
        if (tid < kBlock) {
            const unsigned src = (unsigned)__cvta_generic_to_shared(&colb[k & 1][tid]);
            unsigned rem;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rem) : "r"(src), "r"(k / C));
            V v;
            if constexpr (sizeof(V) == 16)
                asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(rem) : "memory");
            else
                asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(rem) : "memory");
            col[tid] = v;
        }
        __syncthreads();
        if (tid < 32) {
            V v[kBlock / 32];
#pragma unroll
            for (int q = 0; q < kBlock / 32; ++q) v[q] = col[lane + 32 * q];
            const int p = warp_pivot(v, lane, used, singular_s);
            if (lane == 0) {
                piv[k] = p;
                inv_s = cinv_pow2(col[p]);
            }
        }
        __syncthreads();
        const int p = piv[k] - i0;   // the pivot row among this warp's rows
        // the pivot row, scaled (its own column: 1 / pivot)
        if (p >= 0 && p < kR) {
            V r = a[0];
#pragma unroll
            for (int q = 1; q < kR; ++q)
                if (p == q) r = a[q];
            if (jg == k) { r.x = 1; r.y = 0; }
            rowb[j] = cmul2(r, inv_s);
        }
        __syncthreads();
        const V r = rowb[j];
        if ((jg >> 5) == (k >> 5)) {   // the warps with column k
            if (jg == k) {
#pragma unroll
                for (int q = 0; q < kR; ++q) a[q].x = a[q].y = 0;
            }
        }
#pragma unroll
        for (int q = 0; q < kR; ++q) {
            a[q] = gj_update(a[q], col[i0 + q], r);
        }
        if (p >= 0 && p < kR) {
#pragma unroll
            for (int q = 0; q < kR; ++q)
                if (p == q) a[q] = r;
        }
        if (jg == k + 1) {
#pragma unroll
            for (int q = 0; q < kR; ++q) colb[(k + 1) & 1][i0 + q] = a[q];
        }
    }
    __syncthreads();
    // row i was the pivot of step inv_p(i), column jg holds the inverse's column
    // p_jg: Minv[c][r] (transposed) with r the step, c = piv[jg]
    int *step = reinterpret_cast<int *>(rowb);   // C * sizeof(V) >= 4 kBlock
    static_assert(C * sizeof(V) >= kBlock * sizeof(int), "the steps fit the row buffer");
    if (tid < kBlock) step[piv[tid]] = tid;
    __syncthreads();
    const int c = piv[jg];
#pragma unroll
    for (int q = 0; q < kR; ++q) out[(size_t)c * kBlock + step[i0 + q]] = a[q];
    if (tid == 0 && rank == 0 && singular_s) atomicMax(status, 1);
    // no CTA leaves while another may still read its column buffer
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

__device__ __forceinline__ int find_blk(const int *off, int B, int item) {
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

constexpr int kBinv32Threads = 512, kBinv32Cols = 2;
constexpr int kBinv64Threads = 256, kBinv64Cluster = 4;

// The system's last, partial block by one CTA on the nb x nb work array w
// (leading dimension kBlock); the rest of the stored block is zero.
template <typename T>
__device__ void invert_partial(const PcSys &S, int r0, int nb, typename C2<T>::t *w, typename C2<T>::t *out) {
    using V = typename C2<T>::t;
    __shared__ V colk[kBlock];
    __shared__ int piv[kBlock];
    __shared__ int pivrow, singular;
    const V *A = (const V *)S.A;
    if (threadIdx.x == 0) singular = 0;
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
        const int i = e / nb, j = e - i * nb;
        w[i * kBlock + j] = A[(size_t)(r0 + i) * S.lda + r0 + j];
    }
    __syncthreads();
    gauss_jordan<T>(w, kBlock, nb, colk, piv, &pivrow, &singular);
    for (int e = threadIdx.x; e < kBlock * kBlock; e += blockDim.x) {
        const int c = e / kBlock, r = e - c * kBlock;
        V v;
        v.x = v.y = 0;
        if (r < nb && c < nb) v = w[r * kBlock + c];
        out[e] = v;
    }
    if (threadIdx.x == 0 && singular) atomicMax(S.status, 1);
}

// complex64: one CTA per block; a partial block's work array in shared memory
__global__ void __launch_bounds__(kBinv32Threads) k_binv32(const __grid_constant__ PcBatch tb) {
    extern __shared__ float2 smem[];
    const int sb = find_blk(tb.off, tb.B, blockIdx.x);
    const PcSys &S = tb.sys[sb];
    const int b = blockIdx.x - tb.off[sb], r0 = b * kBlock;
    const int nb = min(kBlock, S.n - r0);
    float2 *out = (float2 *)S.Minv + (size_t)b * kBlock * kBlock;
    if (nb == kBlock)
        gauss_jordan_one<float, kBinv32Threads, kBinv32Cols>((const float2 *)S.A + (size_t)r0 * S.lda + r0, S.lda, out, S.status);
    else
        invert_partial<float>(S, r0, nb, smem, out);
}

// complex128: a cluster of CTAs per block; a partial block by its first CTA,
// in the global workspace
__global__ void __cluster_dims__(kBinv64Cluster, 1, 1) __launch_bounds__(kBinv64Threads)
    k_binv64(const __grid_constant__ PcBatch tb) {
    const int item = blockIdx.x / kBinv64Cluster;
    const int sb = find_blk(tb.off, tb.B, item);
    const PcSys &S = tb.sys[sb];
    const int b = item - tb.off[sb], r0 = b * kBlock;
    const int nb = min(kBlock, S.n - r0);
    double2 *out = (double2 *)S.Minv + (size_t)b * kBlock * kBlock;
    if (nb == kBlock)
        gauss_jordan_cluster<double, kBinv64Cluster, kBinv64Threads>((const double2 *)S.A + (size_t)r0 * S.lda + r0, S.lda,
                                                                 out, S.status);
    else if (blockIdx.x % kBinv64Cluster == 0)
        invert_partial<double>(S, r0, nb, (double2 *)S.work + (size_t)b * kBlock * kBlock, out);
}

// fp16 copy of complex64 rows (SplitBatch): one warp per (row, column
// chunk of kMvChunk entries; with a block low-rank copy a block per (block
// row, chunk), only for the segments the copy reads).  The segment's largest component m sets the
// scale 2^(15 - e) with m < 2^e; every component is scaled (exactly) and
// rounded to nearest.  Power-of-two scales keep A16 * rs within one fp16
// rounding of A.  The warp holds its 8 KB segment in registers, so A is
// read once and no block-wide step is needed.
constexpr int kSplitThreads = 256;
constexpr int kSplitWarps = kSplitThreads / 32;

// One row segment (row i, chunk c) by one warp.
__device__ __forceinline__ void split_segment(const SplitSys &S, int i, int c, int lane) {
    const int n = S.n, nch = mv_chunks(n);
    const int c0 = c * kMvChunk, len = min(kMvChunk, n - c0), len2 = len >> 1;
    const float2 *seg = (const float2 *)S.A + (size_t)i * S.lda + c0;   // 8 KB aligned within the row
    const float4 *seg4 = reinterpret_cast<const float4 *>(seg);
    float4 v[kMvChunk / 64];
    float m = 0.f;
#pragma unroll
    for (int q = 0; q < kMvChunk / 64; ++q) {
        const int k = lane + 32 * q;
        v[q] = k < len2 ? __ldcs(seg4 + k) : make_float4(0.f, 0.f, 0.f, 0.f);   // A is streamed
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v[q].x), fabsf(v[q].y)), fmaxf(fabsf(v[q].z), fabsf(v[q].w))));
    }
    float2 last = make_float2(0.f, 0.f);
    if (len & 1) {
        last = seg[len - 1];
        m = fmaxf(m, fmaxf(fabsf(last.x), fabsf(last.y)));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    int e = 0;
    if (m > 0.f) frexpf(m, &e);   // m = f 2^e, 0.5 <= f < 1
    const float scale = ldexpf(1.f, 15 - e);
    if (lane == 0) S.rs[(size_t)i * nch + c] = ldexpf(1.f, e - 15);
    __half2 *h = (__half2 *)S.A16 + (size_t)i * S.lda + c0;
    uint2 *out = reinterpret_cast<uint2 *>(h);
#pragma unroll
    for (int q = 0; q < kMvChunk / 64; ++q) {
        const int k = lane + 32 * q;
        if (k < len2) {
            const __half2 h0 = __floats2half2_rn(v[q].x * scale, v[q].y * scale);
            const __half2 h1 = __floats2half2_rn(v[q].z * scale, v[q].w * scale);
            out[k] = make_uint2(*reinterpret_cast<const unsigned *>(&h0), *reinterpret_cast<const unsigned *>(&h1));
        }
    }
    if ((len & 1) && lane == 0) h[len - 1] = __floats2half2_rn(last.x * scale, last.y * scale);
}

__global__ void __launch_bounds__(kSplitThreads) k_split16(const __grid_constant__ SplitBatch tb) {
    const int sb = find_blk(tb.off, tb.B, blockIdx.x);
    const SplitSys &S = tb.sys[sb];
    const int n = S.n, nch = mv_chunks(n), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (S.blr_rank) {
        // block low-rank copy: a block per (block row I, chunk c), converted
        // only for the diagonal chunk (the preconditioner's window) and
        // chunks with a dense block of the block row; warp w takes rows w,
        // w + kSplitWarps, ...
        const int it = blockIdx.x - tb.off[sb], nb = S.blr_nb;
        const int I = it / nch, c = it - (it / nch) * nch;
        if (I >= nb) return;
        bool need = c == I * kBlrB / kMvChunk;
#pragma unroll
        for (int q = 0; q < kMvChunk / kBlrB; ++q) {
            const int J = c * (kMvChunk / kBlrB) + q;
            need |= J < nb && S.blr_rank[(size_t)I * nb + J] < 0;
        }
        if (!need) return;
        for (int r = warp; r < kBlrB; r += kSplitWarps) {
            const int i = I * kBlrB + r;
            if (i < n) split_segment(S, i, c, lane);
        }
        return;
    }
    const long long item = (long long)(blockIdx.x - tb.off[sb]) * kSplitWarps + warp;
    if (item >= (long long)n * nch) return;
    const int i = (int)(item / nch), c = (int)(item - (long long)i * nch);
    split_segment(S, i, c, lane);
}

}  // namespace

void split_batch_finish(SplitBatch &t) {
    t.off[0] = 0;
    for (int b = 0; b < t.B; ++b) {
        const SplitSys &q = t.sys[b];
        t.off[b + 1] = t.off[b] + (q.blr_rank ? q.blr_nb * mv_chunks(q.n)   // a block per (block row, chunk)
                                              : ceil_div((long long)q.n * mv_chunks(q.n), kSplitWarps));
    }
}

cudaError_t launch_split16(const SplitBatch &t, cudaStream_t st) {
    if (t.B <= 0 || t.off[t.B] == 0) return cudaSuccess;
    count_launches(1);
    k_split16<<<t.off[t.B], kSplitThreads, 0, st>>>(t);
    return cudaGetLastError();
}

// NumCalc's scaling preconditioner (NC_ComputeScalingVector,
// NC_CommonFunctions.cpp:1322-1351, TBEM branch): d_i = sqrt(N / sum_j
// |a_ij|^2), applied to the multiplier vector before every product
// (NC_MatrixVectorMultiplication, :1224-1232), i.e. on the right, and to the
// result at the end (:1193-1203).  Here it is the diagonal of M^{-1} in the
// block-Jacobi storage (the caller clears the blocks), so the Krylov kernels
// apply it unchanged.  Warp per row; row sums in the matrix's precision.
template <typename T>
__global__ void __launch_bounds__(256) k_pc_scaling(const PcSys S) {
    using C2 = typename std::conditional<std::is_same<T, double>::value, double2, float2>::type;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= S.n) return;
    const C2 *row = reinterpret_cast<const C2 *>(S.A) + (size_t)i * S.lda;
    T acc = 0;
    for (int j = lane; j < S.n; j += 32) {
        const C2 a = row[j];
        acc += a.x * a.x + a.y * a.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane != 0) return;
    if (!(acc > 0)) {
        atomicMax(S.status, 1);
        return;
    }
    const double d = sqrt((double)S.n / (double)acc);
    const int p = i / kBlock, r = i - p * kBlock;
    C2 *M = reinterpret_cast<C2 *>(S.Minv) + (size_t)p * kBlock * kBlock;
    C2 v;
    v.x = (T)d;
    v.y = 0;
    M[(size_t)r * kBlock + r] = v;
}

cudaError_t launch_pc_scaling(const PcSys &s, int prec, cudaStream_t st) {
    if (s.n <= 0) return cudaSuccess;
    const size_t bytes = (size_t)pc_blocks(s.n) * kBlock * kBlock * (prec == 0 ? 16 : 8);
    cudaError_t e = cudaMemsetAsync(s.Minv, 0, bytes, st);
    if (e != cudaSuccess) return e;
    count_launches(1);
    const int grid = (s.n + 7) / 8;
    if (prec == 0) k_pc_scaling<double><<<grid, 256, 0, st>>>(s);
    else k_pc_scaling<float><<<grid, 256, 0, st>>>(s);
    return cudaGetLastError();
}

size_t precond_bytes(int n, int prec) {
    const size_t nb = (size_t)pc_blocks(n);
    const size_t per = (size_t)kBlock * kBlock * (prec == 0 ? 16 : 8);
    return nb * per * (prec == 0 ? 2 : 1);   // FP64 needs the inversion workspace too
}

void pc_batch_finish(PcBatch &t) {
    t.off[0] = 0;
    for (int b = 0; b < t.B; ++b) t.off[b + 1] = t.off[b] + pc_blocks(t.sys[b].n);
}

cudaError_t launch_block_inverse(const PcBatch &t, int prec, cudaStream_t st) {
    if (t.B <= 0 || t.off[t.B] == 0) return cudaSuccess;
    count_launches(1);
    if (prec == 0) {
        k_binv64<<<t.off[t.B] * kBinv64Cluster, kBinv64Threads, 0, st>>>(t);
    } else {
        const int smem = kBlock * kBlock * sizeof(float2);
        cudaError_t e = cudaFuncSetAttribute(k_binv32, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        k_binv32<<<t.off[t.B], kBinv32Threads, smem, st>>>(t);
    }
    return cudaGetLastError();
}

}  // namespace bem
