// bem_kernels.cu - assembly, right-hand side and field-projection kernels.
//
// Every launch covers a batch of systems ((mesh, frequency) instances) whose
// table travels in kernel parameter space (__grid_constant__); a single solve
// is a batch of one.
//
// Regular pairs (k_far): the warps of a persistent grid take items of 32
// columns x 2 .. 16 rows, dealt in turn over all systems of the batch; each
// lane owns one column, so the column element's tables are loaded once per
// lane and reused for the rows, and the entries go out as coalesced row
// segments.  Pairs that NumCalc subdivides and the self pairs are skipped
// there and integrated by k_near: warps pull entries of the per-mesh near
// lists from a queue and integrate them cooperatively (warp_subdivide /
// warp_singular).
#include <algorithm>
#include <cmath>
#include <memory>
#include <type_traits>
#include <vector>

#include "bem_internal.h"
#include "bem_pair.cuh"

namespace bem {

namespace {

template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

__device__ __forceinline__ DevMesh to_dev(const DevMeshView &v) {
    DevMesh m;
    m.n = v.n; m.nvert = v.nvert; m.v64 = v.v64; m.c64 = v.c64; m.n64 = v.n64;
    m.area64 = v.area64; m.sqa64 = v.sqa64; m.chi = v.chi; m.clo = v.clo; m.t32 = v.t32;
    m.q32 = v.q32; m.isqa32 = v.isqa32; m.n32 = v.n32; m.row4 = v.row4;
    m.sym = v.sym;
    return m;
}

// Largest b with off[b] <= item (off ascending, off[0] = 0, item < off[B]).
__device__ __forceinline__ int find_sys(const int *off, int B, int item) {
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Persistent-grid exit: the last block to leave resets the queue counters
// (ctr[0] = items handed out, ctr[1] = blocks finished) for the next launch.
__device__ __forceinline__ void queue_exit(unsigned *ctr) {
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        if (atomicAdd(ctr + 1, 1u) == gridDim.x - 1) {
            ctr[0] = 0u;
            ctr[1] = 0u;
            __threadfence();
        }
    }
}

__device__ __forceinline__ cplx<double> ld_c(const double *p, int idx) {
    double2 v = reinterpret_cast<const double2 *>(p)[idx];
    return {v.x, v.y};
}

// Regular pair in precision T with a fixed Gauss order (no subdivision):
// the single-subelement case of NC_RegularIntegration.
template <typename T> struct FarPair;

template <> struct FarPair<double> {
    static __device__ __forceinline__ KVals<double> run(const Elem64 &e, const double x[3], const double nx[3],
                                                        int order, double k, double wr) {
        KVals<double> acc;
        acc.G = acc.H = acc.HT = acc.E = cmk(0.0, 0.0);
        const int np = e.nv == 3 ? tri_count(order) : quad_count(order);
        for (int g = 0; g < np; ++g) {
            double s, t, w;
            if (e.nv == 3) {
                const int o = tri_offset(order) + g;
                s = c_quad.tri[o][0]; t = c_quad.tri[o][1]; w = c_quad.tri[o][2];
            } else {
                const int a = g / order, b = g - a * order;
                s = c_quad.glx[order][a]; t = c_quad.glx[order][b];
                w = c_quad.glw[order][a] * c_quad.glw[order][b];
            }
            QPoint<double> q;
            map_point(e, s, t, x, w, q);
            KVals<double> v = kernel_values(q, nx, k, wr);
            acc.G += v.G; acc.H += v.H; acc.HT += v.HT; acc.E += v.E;
        }
        return acc;
    }
};

// Fused float evaluation of a regular pair's matrix entry.  The entry is
// linear in the kernel values, so each quadrature point contributes
// G * F with F built from the point's geometry and the column's boundary
// condition (NC_AssembleTBEM, NC_EquationSystem.cpp:165-207):
//   velocity:        H tau + E beta            -> F = tau z1 re1 + i b ze1
//   + admittance:    ... + (G + HT beta tau) Y -> F += Y (1 + i b tau z1 re2)
//   pressure:        -G tau - HT beta          -> F = -tau - i b z1 re2
// with z1 = -1/r + i wr, re1 = r^.n_y, re2 = -r^.n_x,
// ze1 = (3/r^2 - k^2) rq + n_x.n_y/r^2 - i wr/r (3 rq + n_x.n_y), rq = re1 re2,
// beta = i b.  One complex accumulator per entry instead of four.
struct FusedCol {
    int bc;
    float yr, yi;          // admittance (bc 2)
    float tau, b, k2, wr;  // tau, beta / i, k^2, time factor * k
};

__device__ __forceinline__ void fused_point(const FusedCol &c, float dny, float dnx, float nn, float r2, float w,
                                            float &acc_re, float &acc_im) {
    const float ir = rsqrt_approx(r2);
    const float r = r2 * ir;
    float sn, cs;
    phase_sincos(c.wr * r, &sn, &cs);
    const float amp = w * (float)(1.0 / kPI4) * ir;
    const float gr = cs * amp, gi = sn * amp;   // G
    const float re1 = dny * ir, re2 = -dnx * ir;
    float fr, fi;
    if (c.bc == 1) {
        // -tau - i b (-ir re2 + i wr re2) = (-tau + b wr re2, b ir re2)
        fr = fmaf(c.b * c.wr, re2, -c.tau);
        fi = c.b * ir * re2;
    } else {
        const float rq = re1 * re2, ir2 = ir * ir;
        const float e_re = fmaf(3.f * ir2 - c.k2, rq, nn * ir2);
        const float e_im = -c.wr * ir * fmaf(3.f, rq, nn);
        // tau z1 re1 + i b ze1
        fr = fmaf(-c.tau * ir, re1, -c.b * e_im);
        fi = fmaf(c.tau * c.wr, re1, c.b * e_re);
        if (c.bc == 2) {
            // Y (1 + i b tau z1 re2) = Y (1 - b tau wr re2, -b tau ir re2)
            const float pr = fmaf(-c.b * c.tau * c.wr, re2, 1.f), pi = -c.b * c.tau * ir * re2;
            fr += c.yr * pr - c.yi * pi;
            fi += c.yr * pi + c.yi * pr;
        }
    }
    acc_re = fmaf(gr, fr, fmaf(-gi, fi, acc_re));
    acc_im = fmaf(gr, fi, fmaf(gi, fr, acc_im));
}

// Points O0 .. O0+NP-1 of the triangle rules, unrolled so that the rule's
// constants are constant-bank operands (the order is uniform across most
// warps: neighbouring columns are neighbouring elements).
template <int NP, int O0>
__device__ __forceinline__ void tri_points(const Elem32 &e, float dny, float dnx0, float anx, float bnx, float nn,
                                           const FusedCol &c, float &ar, float &ai) {
#pragma unroll
    for (int g = 0; g < NP; ++g) {
        const float ss = c_trif[O0 + g][0] - (1.0f / 3.0f), tt = c_trif[O0 + g][1] - (1.0f / 3.0f);
        const float w = c_trif[O0 + g][2] * e.J;
        float d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = fmaf(tt, e.b[k], fmaf(ss, e.a[k], e.D[k]));
        const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        fused_point(c, dny, fmaf(tt, bnx, fmaf(ss, anx, dnx0)), nn, r2, w, ar, ai);
    }
}

// Matrix entry of a regular pair in float with a Gauss order above 2.  Flat
// triangles: n_y is constant and d.n_y = D.n_y at every point; d.n_x is
// affine in (s, t).
__device__ __forceinline__ float2 far_entry_f(const Elem32 &e, const float nx[3], int order, const FusedCol &c) {
    float ar = 0.f, ai = 0.f;
    if (e.nv == 3) {
        const float dny = e.D[0] * e.n[0] + e.D[1] * e.n[1] + e.D[2] * e.n[2];
        const float dnx0 = e.D[0] * nx[0] + e.D[1] * nx[1] + e.D[2] * nx[2];
        const float anx = e.a[0] * nx[0] + e.a[1] * nx[1] + e.a[2] * nx[2];
        const float bnx = e.b[0] * nx[0] + e.b[1] * nx[1] + e.b[2] * nx[2];
        const float nn = e.n[0] * nx[0] + e.n[1] * nx[1] + e.n[2] * nx[2];
        if (order == 3) tri_points<7, 4>(e, dny, dnx0, anx, bnx, nn, c, ar, ai);
        else tri_points<13, 11>(e, dny, dnx0, anx, bnx, nn, c, ar, ai);
    } else {
        const int np = quad_count(order);
        for (int g = 0; g < np; ++g) {
            const int a = g / order, b = g - a * order;
            QPoint<float> q;
            map_point(e, c_glxf[order][a], c_glxf[order][b], c_glwf[order][a] * c_glwf[order][b], q);
            const float dny = q.d[0] * q.ny[0] + q.d[1] * q.ny[1] + q.d[2] * q.ny[2];
            const float dnx = q.d[0] * nx[0] + q.d[1] * nx[1] + q.d[2] * nx[2];
            const float nn = q.ny[0] * nx[0] + q.ny[1] * nx[1] + q.ny[2] * nx[2];
            const float r2 = q.d[0] * q.d[0] + q.d[1] * q.d[1] + q.d[2] * q.d[2];
            fused_point(c, dny, dnx, nn, r2, q.wj, ar, ai);
        }
    }
    return make_float2(ar, ai);
}

// Order-2 far pairs on a flat triangle (the 4-point rule), two rows at a time
// in packed FP32, with the column element's data hoisted out of the row loop:
// point g's squared distance is |D|^2 + 2 s_g D.a + 2 t_g D.b + C_g with
// C_g = |s_g a + t_g b|^2 (at the order-2 ratio, |D| > 4 sqrt(area), the terms
// do not cancel on elements that are not long and thin; see far_tri2).  The distance, the phase and its reduction are rounded
// operation by operation (the phase's rounding is the entry's error); the
// kernel terms of fused_point are regrouped around u = 1/r as in far_tri64.
//
// Bound by the FMA pipe and the special-function unit together (27 packed and
// 2 scalar FP32 operations and 6 special functions per two evaluations, and
// about 45 per pair of entries); one entry at a time it was bound by
// instruction issue at 79 per evaluation.  20480-triangle head, 10 kHz: k_far
// 4.07 -> 3.33 ms, and 3.17 with the rows' data stored as pairs (18 moves a pair
// less); 1280 triangles 50 us as before, 3072 quadrilaterals and their images
// 690 -> 665.  Three blocks per SM with the column's data in shared memory
// instead of two with it in registers: 3.77 ms.
struct FarCol2 {
    F2 a[3], b[3], n[3];
    F2 C[3];       // |s_g a + t_g b|^2 of points 1 .. 3 (point 0 is the centroid)
    F2 wJ0, wJ1;   // weight J / (4 pi) of point 0 and of the others
};
static_assert(sizeof(FarCol2) == 14 * sizeof(F2), "28 registers");

__device__ __forceinline__ F2 dup2(float x) { return pk2(x, x); }

// Constants of the packed evaluation, each twice.
struct FarConst {
    ScConst<F2> sc;
    F2 m1, m3;       // -1, -3
    F2 p, q;         // the 4-point rule's s - 1/3: -2/15 and 4/15
};
__device__ __forceinline__ void far_const(FarConst &k) {
    k.sc.init();
    k.m1 = opaque2(-1.f);
    k.m3 = opaque2(-3.f);
    k.p = opaque2(c_far4[1][0]);
    k.q = opaque2(c_far4[2][0]);
}

__device__ __forceinline__ void far_col2(const DevMesh &m, int j, FarCol2 &e) {
    float a[3], b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = m.t32[k * m.n + j];
        b[k] = m.t32[(3 + k) * m.n + j];
        vdup(e.a[k], a[k]);
        vdup(e.b[k], b[k]);
        vdup(e.n[k], m.t32[(6 + k) * m.n + j]);
    }
    const float J4 = m.t32[9 * m.n + j] * (float)(1.0 / kPI4);
#pragma unroll
    for (int g = 1; g < 4; ++g) {
        float c = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float d = fmaf(c_far4[g][1], b[k], c_far4[g][0] * a[k]);
            c = fmaf(d, d, c);
        }
        vdup(e.C[g - 1], c);
    }
    vdup(e.wJ0, c_trif[0][2] * J4);
    vdup(e.wJ1, c_trif[1][2] * J4);
}

// Constants of a column, each twice.
struct FusedCol2 {
    F2 wr, b, bwr, k2, nt, tw;    // wr, beta / i, b wr, k^2, -tau, tau wr
    F2 yr, yi, nyi, bt, btw;      // admittance, -its imaginary part, b tau, b tau wr (BC 2)
};
// Sums of an entry pair: cos F_re, sin F_im (apart, so that no negation is
// needed) and the imaginary part.
struct FarSum2 { F2 rr, ri, ai; };

__device__ __forceinline__ F2 dot2(const F2 x[3], const F2 y[3]) {
    return vfma(x[2], y[2], vfma(x[0], y[0], vmul(x[1], y[1])));
}

// One quadrature point of two entries: squared distance, d.n_y, d.n_x, n_x.n_y,
// weight / (4 pi).  BC: the column's boundary condition (0 velocity, 1
// pressure, 2 velocity with admittance), fixed per instantiation so that the
// point has no branch.
template <int BC>
__device__ __forceinline__ void far_point2(const FarConst &k, const FusedCol2 &c, F2 r2, F2 dny, F2 dnx, F2 nn, F2 wj,
                                           FarSum2 &o) {
    F2 r, sn, cs, fr, fi, amp;
    const F2 u = vrsqrt(r2, &r);
    vsincos(k.sc, vmul(c.wr, r), sn, cs);
    if (BC == 1) {
        // -tau - i b z1 re2, z1 = -1/r + i wr, re2 = -d.n_x / r
        const F2 ndu = vmul(vmul(dnx, u), k.m1);
        fr = vfma(c.bwr, ndu, c.nt);
        fi = vmul(vmul(c.b, ndu), u);
        amp = vmul(wj, u);
    } else {
        // tau z1 re1 + i b ze1 (re1 = d.n_y / r), times r
        const F2 P = vmul(dny, dnx), u2 = vmul(u, u);
        const F2 E = vfma(vmul(P, u2), k.m3, nn);   // n_x.n_y - 3 P / r^2
        fr = vfma(c.bwr, E, vmul(vmul(c.nt, dny), u));
        fi = vfma(vmul(c.b, u), vfma(c.k2, P, E), vmul(c.tw, dny));
        amp = vmul(wj, u2);
        if (BC == 2) {
            // + Y (1 + i b tau z1 re2), times r
            const F2 pr = vfma(c.btw, dnx, r), pi = vmul(vmul(c.bt, u), dnx);
            fr = vfma(c.yr, pr, vfma(c.nyi, pi, fr));
            fi = vfma(c.yr, pi, vfma(c.yi, pr, fi));
        }
    }
    const F2 qr = vmul(amp, fr), qi = vmul(amp, fi);
    o.rr = vfma(cs, qr, o.rr);
    o.ri = vfma(sn, qi, o.ri);
    o.ai = vfma(cs, qi, vfma(sn, qr, o.ai));
}

// DIFF: the squared distance from the difference of the points, as every other
// pair's, for meshes with symmetry images.  Where a long thin triangle's point is
// closer than its centroid, the expanded sum loses (|D| / r)^2 units, and
// images come close at their plane.
template <int BC, bool DIFF>
__device__ __forceinline__ void far_tri2(const FarConst &k, const FarCol2 &e, const F2 D[3], F2 D2, const F2 nx[3],
                                         const FusedCol2 &c, FarSum2 &o) {
    const F2 dny = dot2(D, e.n), dnx = dot2(D, nx), nn = dot2(e.n, nx);
    const F2 anx = dot2(e.a, nx), bnx = dot2(e.b, nx);
    F2 Da, Db;
    if (!DIFF) {
        Da = dot2(D, e.a);
        Db = dot2(D, e.b);
        Da = vadd(Da, Da);   // exact: 2 s D.a = s (2 D.a)
        Db = vadd(Db, Db);
    }
    auto r2 = [&](F2 s, F2 t, F2 C) {
        if (!DIFF) return vfma(s, Da, vfma(t, Db, vadd(D2, C)));
        F2 d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) d[q] = vfma(t, e.b[q], vfma(s, e.a[q], D[q]));
        return dot2(d, d);
    };
    far_point2<BC>(k, c, D2, dny, dnx, nn, e.wJ0, o);
    far_point2<BC>(k, c, r2(k.p, k.p, e.C[0]), dny, vfma(k.p, bnx, vfma(k.p, anx, dnx)), nn, e.wJ1, o);
    far_point2<BC>(k, c, r2(k.q, k.p, e.C[1]), dny, vfma(k.p, bnx, vfma(k.q, anx, dnx)), nn, e.wJ1, o);
    far_point2<BC>(k, c, r2(k.p, k.q, e.C[2]), dny, vfma(k.q, bnx, vfma(k.p, anx, dnx)), nn, e.wJ1, o);
}

// The same for a quadrilateral column, whose four points (offset from the
// centre, normal, weight) were mapped once by far_quad_stage into the lane's
// column of shared memory.
constexpr int kQuadRows = 28;
__device__ __forceinline__ void far_quad_stage(const DevMesh &m, int j, float (*st)[32], int lane) {
    Elem32 e;
    const float zero[3] = {0.f, 0.f, 0.f};
    load_elem32(m, j, zero, zero, e);
    e.D[0] = e.D[1] = e.D[2] = 0.f;
#pragma unroll 1
    for (int g = 0; g < 4; ++g) {
        QPoint<float> q;
        map_point(e, c_glxf[2][g >> 1], c_glxf[2][g & 1], c_glwf[2][g >> 1] * c_glwf[2][g & 1], q);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            st[7 * g + k][lane] = q.d[k];
            st[7 * g + 3 + k][lane] = q.ny[k];
        }
        st[7 * g + 6][lane] = q.wj * (float)(1.0 / kPI4);
    }
}
template <int BC>
__device__ __forceinline__ void far_quad2(const FarConst &k, float (*st)[32], int lane, const F2 D[3], const F2 nx[3],
                                          const FusedCol2 &c, FarSum2 &o) {
#pragma unroll 1
    for (int g = 0; g < 4; ++g) {
        F2 d[3], ny[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            d[q] = vadd(D[q], dup2(st[7 * g + q][lane]));
            ny[q] = dup2(st[7 * g + 3 + q][lane]);
        }
        far_point2<BC>(k, c, dot2(d, d), dot2(d, ny), dot2(d, nx), dot2(ny, nx), dup2(st[7 * g + 6][lane]), o);
    }
}

// FP64 regular pair on a flat triangle, arranged for few FP64 instructions
// (the plain path is bound by GB300's narrow FP64 pipe): the column's edge
// vectors, normal, Jacobian and centroid, in two parts, are formed once per
// thread; a point's vector d is the difference D of the centroid's high part
// and x plus the point's offset, two roundings, D's exact for near pairs.  With
// P = (D.n_y)(d.n_x), u = 1/r, E = n_x.n_y - 3 P u^2 the velocity entry's factor is
//   u (b wr E - tau D.n_y u) + i u (b u (E + k^2 P) + tau wr D.n_y).
// 53 FP64 instructions per point (the general form through map_point and the
// library's square roots, divisions and sincos took about 250).  5120-triangle
// head, 5 kHz: k_far 33.0 -> 13.1 ms.  Mean errors against 80-bit entries, this
// and the general form, beyond a ratio of 4.5 and below 4, k = 73: head 1.35e-15
// and 1.50e-15, 8.6e-16 and 9.1e-16; sphere flattened to a tenth 8.4e-16 and
// 9.0e-16, 2.4e-16 and 3.0e-16.  |D|^2 + 2 s D.a + ... for the squared distance
// (7 instructions less) loses (|D| / r)^2 units where a long thin
// triangle's point comes close to x.
struct FarCol64 {
    double c[3], cl[3];  // centroid, high and low part
    double a[3], b[3], n[3];
    double cln;          // cl . n
    double J4;           // J / (4 pi)
    int far;             // the vertices' largest component (max_hi)
};
struct FusedCol64 {
    double yr, yi, tau, b, k2, wr;
};

__device__ __forceinline__ void far_col64(const DevMesh &m, int j, FarCol64 &e) {
    double n2 = 0.0;
    e.far = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double p2 = m.v64[(6 + k) * m.n + j];
        e.far = max(e.far, max_hi(m.v64[k * m.n + j], m.v64[(3 + k) * m.n + j], p2));
        e.a[k] = m.v64[k * m.n + j] - p2;
        e.b[k] = m.v64[(3 + k) * m.n + j] - p2;
        const double o = (e.a[k] + e.b[k]) * (1.0 / 3.0);
        e.c[k] = p2 + o;
        const double p = e.c[k] - o;   // the sum's error (Knuth)
        e.cl[k] = (p2 - p) + (o - (e.c[k] - p));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int p = (k + 1) % 3, q = (k + 2) % 3;
        e.n[k] = e.a[p] * e.b[q] - e.b[p] * e.a[q];
        n2 = fma(e.n[k], e.n[k], n2);
    }
    double len;
    const double il = rsqrt_nr(n2, &len);
#pragma unroll
    for (int k = 0; k < 3; ++k) e.n[k] *= il;
    e.cln = e.cl[0] * e.n[0] + e.cl[1] * e.n[1] + e.cl[2] * e.n[2];
    e.J4 = len * (1.0 / kPI4);
}

// Points o0 .. o0 + np - 1 of the triangle rules; D = centroid's high part - x.
template <int BC>
__device__ __forceinline__ cplx<double> far_tri64(const FarCol64 &e, const double D[3], const double nx[3], int o0,
                                                  int np, const FusedCol64 &c) {
    const double dny = fma(D[2], e.n[2], fma(D[1], e.n[1], fma(D[0], e.n[0], e.cln)));
    const double nn = e.n[0] * nx[0] + e.n[1] * nx[1] + e.n[2] * nx[2];
    const double ct = -c.tau * dny, cw = c.tau * c.wr * dny, bwr = c.b * c.wr;
    double ar = 0.0, ai = 0.0;
#pragma unroll 2
    for (int g = 0; g < np; ++g) {
        const double s = c_far64[o0 + g][0], t = c_far64[o0 + g][1], w = c_far64[o0 + g][2];
        double d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = D[k] + fma(t, e.b[k], fma(s, e.a[k], e.cl[k]));
        const double r2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
        const double dnx = fma(d[2], nx[2], fma(d[1], nx[1], d[0] * nx[0]));
        double r, sn, cs;
        const double u = rsqrt_nr(r2, &r), u2 = u * u;
        phase_sincos(c.wr * r, &sn, &cs);
        double fr, fi, amp;
        if (BC == 1) {
            const double du = dnx * u;
            fr = fma(-bwr, du, -c.tau);
            fi = -c.b * du * u;
            amp = w * e.J4 * u;
        } else {
            const double P = dny * dnx, E = fma(-3.0 * P, u2, nn);
            fr = fma(bwr, E, ct * u);
            fi = fma(c.b * u, fma(c.k2, P, E), cw);
            amp = w * e.J4 * u2;
            if (BC == 2) {
                // + Y (1 + i b tau z1 re2) / u
                const double bt = c.b * c.tau;
                const double pr = fma(bt * c.wr, dnx, r), pi = bt * u * dnx;
                fr += c.yr * pr - c.yi * pi;
                fi += c.yr * pi + c.yi * pr;
            }
        }
        ar = fma(amp, fma(cs, fr, -sn * fi), ar);
        ai = fma(amp, fma(cs, fi, sn * fr), ai);
    }
    return {ar, ai};
}

__device__ __forceinline__ cplx<double> far_entry_tri64(const FarCol64 &e, const double x[3], const double nx[3],
                                                        int order, int bc, const FusedCol64 &c) {
    const double D[3] = {e.c[0] - x[0], e.c[1] - x[1], e.c[2] - x[2]};
    const int o0 = tri_offset(order), np = tri_count(order);
    if (bc == 0) return far_tri64<0>(e, D, nx, o0, np, c);
    if (bc == 1) return far_tri64<1>(e, D, nx, o0, np, c);
    return far_tri64<2>(e, D, nx, o0, np, c);
}

template <typename T>
__device__ __forceinline__ cplx<T> col_adm(const DevFreq &f, int j, int bc) {
    if (bc != 2 || f.adm == nullptr) return {T(0), T(0)};
    cplx<double> a = ld_c(f.adm, j);
    return {(T)a.re, (T)a.im};
}

// ------------------------------------------------------------ symmetry images
// Image tables (DevSym): one thread per (image, element).  The vertices go
// through the reference's sequence of reflections (2 c - x per step, then the
// node swap, NC_ReflectElement, NC_3dFunctions.cpp:357-452), so that each
// image holds the coordinates the reference integrates over; the centre is
// the global point at the local centre, as NC_GenerateSubelements computes
// it for the level-0 test.
__global__ void __launch_bounds__(256) k_image_tables(DevMeshView mv, ImageTables out) {
    const DevMesh m = to_dev(mv);
    const int n = m.n;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)(m.sym.nref - 1) * n) return;
    const int k = (int)(t / n), j = (int)(t - (long long)k * n), kref = k + 1;
    Elem64 e;
    load_elem64(m, j, e);
    double nr[3] = {m.n64[j], m.n64[n + j], m.n64[2 * n + j]};
    for (int step = 1; step <= kref; ++step) {
        const int d = m.sym.rdir[step];
        const double c2 = 2.0 * m.sym.coord[d];
        for (int a = 0; a < e.nv; ++a) e.p[a][d] = __dsub_rn(c2, e.p[a][d]);
        nr[d] = -nr[d];
        for (int q = 0; q < (e.nv == 4 ? 2 : 1); ++q)
            for (int c = 0; c < 3; ++c) {
                const double tmp = e.p[2 * q][c];
                e.p[2 * q][c] = e.p[2 * q + 1][c];
                e.p[2 * q + 1][c] = tmp;
            }
    }
    const size_t nn = (size_t)n, ko = (size_t)k;
    double *v64 = out.v64 + ko * 12 * nn, *c64 = out.c64 + ko * 3 * nn;
    float *chi = out.chi + ko * 3 * nn, *clo = out.clo + ko * 3 * nn;
    float *t32 = out.t32 + ko * 10 * nn, *q32 = out.q32 + ko * 12 * nn;
    for (int a = 0; a < 4; ++a)
        for (int c = 0; c < 3; ++c) v64[(3 * a + c) * nn + j] = a < e.nv ? e.p[a][c] : 0.0;
    // local centre: (1 + 0 + 0) / 3 on triangles, 0 on quadrilaterals
    const double sc = e.nv == 3 ? 1.0 / 3.0 : 0.0;
    double cen[3];
    global_point_exact(e, sc, sc, cen);
    for (int c = 0; c < 3; ++c) {
        c64[c * nn + j] = cen[c];
        const float h = (float)cen[c];
        chi[c * nn + j] = h;
        clo[c * nn + j] = (float)(cen[c] - (double)h);
    }
    if (e.nv == 3) {
        for (int c = 0; c < 3; ++c) {
            t32[c * nn + j] = (float)(e.p[0][c] - e.p[2][c]);
            t32[(3 + c) * nn + j] = (float)(e.p[1][c] - e.p[2][c]);
            t32[(6 + c) * nn + j] = (float)nr[c];
        }
        t32[9 * nn + j] = m.t32[9 * nn + j];
        for (int r = 0; r < 12; ++r) q32[r * nn + j] = 0.f;
    } else {
        for (int r = 0; r < 10; ++r) t32[r * nn + j] = 0.f;
        for (int a = 0; a < 4; ++a)
            for (int c = 0; c < 3; ++c) q32[(3 * a + c) * nn + j] = (float)(e.p[a][c] - cen[c]);
    }
}

// ------------------------------------------------------------ near list
// Pairs (row i, column j) that NumCalc integrates with subdivision (level-0
// ratio distance/sqrt(area) < 1.3, exact FP64 test, for any image of j) plus
// the self pairs.  Depends on the geometry only, so it is built once per
// mesh.  Entries go to list[0, cap) in any order (warp-aggregated atomics);
// *count ends as the number of entries, which may exceed cap (the caller
// then runs again with a larger list).
//
// Bounding spheres of the column blocks (32 consecutive elements, Morton
// order) of every image, and each block's largest sqrt(area): warp per
// (image, block).  Radii are inflated past float rounding, so the block test
// of k_near_list never drops a pair the element test would keep.
__global__ void __launch_bounds__(256) k_block_spheres(DevMeshView mv, float4 *sph, float *bsq) {
    const DevMesh m = to_dev(mv);
    const int lane = threadIdx.x, n = m.n, nb = (n + 31) / 32;
    const int gw = blockIdx.x * 8 + threadIdx.y;
    if (gw >= nb * m.sym.nref) return;
    const int kref = gw / nb, b = gw - kref * nb;
    const DevMesh mk = image_mesh(m, kref);
    const int j = b * 32 + lane, jj = j < n ? j : b * 32;   // idle lanes repeat the block's first element
    float c[3], lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c[k] = mk.chi[k * n + jj] + mk.clo[k * n + jj];
        lo[k] = c[k];
        hi[k] = c[k];
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    }
    const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
    float r = sqrtf((c[0] - cx) * (c[0] - cx) + (c[1] - cy) * (c[1] - cy) + (c[2] - cz) * (c[2] - cz));
    float sq = (float)m.sqa64[jj];
    for (int o = 16; o > 0; o >>= 1) {
        r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
        sq = fmaxf(sq, __shfl_xor_sync(0xffffffffu, sq, o));
    }
    if (lane == 0) {
        const float cmax = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz)));
        sph[gw] = make_float4(cx, cy, cz, r * (1.f + 1e-5f) + 1e-6f * cmax);
        if (kref == 0) bsq[b] = sq * (1.f + 1e-5f);
    }
}

// Near list: warp per row, lanes over 32 column blocks at a time.  A block
// whose sphere (of any image) lies farther from the row's centre than 1.31
// times its largest sqrt(area) holds no pair below the subdivision threshold
// 1.3 (the element test below keeps pairs up to 1.3 (1 + 1e-4) for the exact
// decision); the other blocks get the element test, image by image as the
// reference loops them, with one entry per (row, column) carrying the mask of
// near images (the self pair always).
__global__ void __launch_bounds__(256) k_near_list(DevMeshView mv, const float4 *sph, const float *bsq, int2 *list,
                                                   unsigned long long *count, unsigned long long cap) {
    const DevMesh m = to_dev(mv);
    const int lane = threadIdx.x, n = m.n, nb = (n + 31) / 32, nref = m.sym.nref;
    const int i = blockIdx.x * 8 + threadIdx.y;
    if (i >= n) return;
    const float ci[3] = {m.chi[i] + m.clo[i], m.chi[n + i] + m.clo[n + i], m.chi[2 * n + i] + m.clo[2 * n + i]};
    const float cn = fmaxf(fabsf(ci[0]), fmaxf(fabsf(ci[1]), fabsf(ci[2])));
    for (int cb0 = 0; cb0 < nb; cb0 += 32) {
        const int cb = cb0 + lane;
        bool cand = false;
        if (cb < nb) {
            const float thr = 1.31f * bsq[cb];
            for (int kref = 0; kref < nref; ++kref) {
                const float4 sp = sph[kref * nb + cb];
                const float d0 = ci[0] - sp.x, d1 = ci[1] - sp.y, d2 = ci[2] - sp.z;
                const float slack = 1e-6f * (cn + fmaxf(fabsf(sp.x), fmaxf(fabsf(sp.y), fabsf(sp.z))));
                if (sqrtf(d0 * d0 + d1 * d1 + d2 * d2) - sp.w <= thr + slack) cand = true;
            }
        }
        unsigned cm = __ballot_sync(0xffffffffu, cand);
        while (cm) {
            const int bl = __ffs(cm) - 1;
            cm &= cm - 1;
            const int j = (cb0 + bl) * 32 + lane;
            unsigned imask = 0;
            if (j < n) {
                for (int kref = 0; kref < nref; ++kref) {
                    if (kref == 0 && j == i) { imask |= 1u; continue; }
                    const DevMesh mk = image_mesh(m, kref);
                    const float d0 = (mk.chi[j] - m.chi[i]) + (mk.clo[j] - m.clo[i]);
                    const float d1 = (mk.chi[n + j] - m.chi[n + i]) + (mk.clo[n + j] - m.clo[n + i]);
                    const float d2 = (mk.chi[2 * n + j] - m.chi[2 * n + i]) + (mk.clo[2 * n + j] - m.clo[2 * n + i]);
                    const float rf = sqrtf(d0 * d0 + d1 * d1 + d2 * d2) * m.isqa32[j];
                    if (rf <= 1.3f * (1.0f + 1e-4f)) {
                        const double x[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
                        if (ratio0_exact(mk, j, x) < kTolf) imask |= 1u << kref;
                    }
                }
            }
            const bool near = imask != 0;
            const unsigned mask = __ballot_sync(0xffffffffu, near);
            if (!mask) continue;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(mask));
            base = __shfl_sync(0xffffffffu, base, 0);
            const unsigned long long idx = base + __popc(mask & ((1u << lane) - 1u));
            if (near && list && idx < cap) list[idx] = make_int2(i, j | (int)(imask << kNearColBits));
        }
    }
}

// ------------------------------------------------------------ regular pairs
// Regular (not subdivided) pairs: a warp takes 32 columns, one per lane, and
// some rows.  The column element is loaded once per lane and reused for its
// rows; entries go out as coalesced row segments.  Near and self pairs are
// zero here; k_near adds their integrals.
//
// Rows per item (an item is one warp's 32 columns x far_rows rows): the more,
// the further the column's preparation is spread; small systems take fewer so
// that the 2432 warps of the grid (two blocks of eight on each of 152 SMs) get
// about six items or more each (with one or two the last round would leave most
// of them idle).  The host and the kernel both form it, so it goes by the
// number and not by the device; entries do not depend on it.
__host__ __device__ inline int far_rows(int n) {
    const long long e = (long long)n * n / (32 * 6 * 2432);   // rows for six items per warp
    return e >= 16 ? 16 : e >= 8 ? 8 : e >= 4 ? 4 : 2;
}

// Out-of-line parts of the float tile, taken by few pairs: keeping them out
// of the row loop keeps the mesh pointers they read out of its registers.
// Exact (FP64) decision for a pair within the float test's margin of a
// threshold: 0 for a near pair, else the Gauss order.
__device__ __noinline__ int far_order_exact(const DevMeshView *mv, int kref, int i, int j) {
    const DevMesh m = to_dev(*mv);
    const int n = m.n;
    const double x64[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
    const double rd = ratio0_exact(image_mesh(m, kref), j, x64);
    return rd < kTolf ? 0 : gauss_order(rd);
}
// Entry of a Gauss order above 2.
__device__ __noinline__ float2 far_entry_general(const DevMeshView *mv, int kref, int j, float D0, float D1, float D2,
                                                 float nx0, float nx1, float nx2, int order, FusedCol fc) {
    const DevMesh m = image_mesh(to_dev(*mv), kref);
    Elem32 e;
    const float zero[3] = {0.f, 0.f, 0.f};
    load_elem32(m, j, zero, zero, e);
    e.D[0] = D0; e.D[1] = D1; e.D[2] = D2;
    const float nx[3] = {nx0, nx1, nx2};
    return far_entry_f(e, nx, order, fc);
}

// One warp's item of image kref of the columns: rows from i0, column block tx.
// st: the warp's shared memory for quadrilateral columns.
// kref = 0 writes the entries; the images add theirs (reflection factor
// applied, NC_AssembleTBEM, NC_EquationSystem.cpp:181-206) in image order.
// Near images and the self pair contribute zero here; k_near adds them.
template <typename T, bool IMG>
__device__ __forceinline__ void far_tile(const DevMeshView &mv, const DevFreq &f,
                                         typename Vec2<T>::type *__restrict__ A, size_t lda, int tx, int i0, int kref,
                                         const FarConst &fk, float (*st)[32]) {
    const DevMesh m = to_dev(mv);
    const DevMesh mk = image_mesh(m, kref);
    const int lane = threadIdx.x, n = m.n, rpt = far_rows(n);
    const int j = tx * 32 + lane;
    if (j >= n) return;
    Phys<T> PT;
    if constexpr (std::is_same<T, double>::value) PT = {f.k, f.wr, f.tao, f.beta_im};
    else PT = {f.kf, f.wrf, f.taof, f.beta_imf};
    const int bcj = f.bc_type ? f.bc_type[j] : 0;
    const cplx<T> admj = col_adm<T>(f, j, bcj);
    const bool neg = image_negated(m, kref);
    const bool tri = m.nvert[j] == 3;
    const float cjh[3] = {mk.chi[j], mk.chi[n + j], mk.chi[2 * n + j]};
    const float cjl[3] = {mk.clo[j], mk.clo[n + j], mk.clo[2 * n + j]};
    const float isq2 = m.isqa32[j] * m.isqa32[j];
    auto put = [&](int i, T re, T im) {
        typename Vec2<T>::type *p = A + (size_t)i * lda + j, o;
        if (kref > 0) {
            o = *p;
            o.x += neg ? -re : re;
            o.y += neg ? -im : im;
        } else {
            o.x = re;
            o.y = im;
        }
        *p = o;
    };
    if constexpr (std::is_same<T, double>::value) {
        FarCol64 e4;
        if (tri) far_col64(mk, j, e4);
        const FusedCol64 fc = {admj.re, admj.im, f.tao, f.beta_im, f.k * f.k, f.wr};
        const int reach = phase_reach(f.wr);
        const bool fits = tri && e4.far < reach;
#pragma unroll 1
        for (int r = 0; r < rpt; ++r) {
            const int i = i0 + r;
            if (i >= n) break;
            cplx<double> val = {0.0, 0.0};
            if (i != j || kref > 0) {
                // the quadrature decision from the float distance, the exact
                // FP64 one (a square root and a division) only near a threshold
                const float *nr = reinterpret_cast<const float *>(m.row4 + 5 * (size_t)(i >> 1)) + (i & 1);   // -centre
                const float d0 = (cjh[0] + nr[0]) + (cjl[0] + nr[6]), d1 = (cjh[1] + nr[2]) + (cjl[1] + nr[8]),
                            d2 = (cjh[2] + nr[4]) + (cjl[2] + nr[10]);
                const float q2 = (d0 * d0 + d1 * d1 + d2 * d2) * isq2;
                bool near = false;
                int order = 2;
                if (q2 <= c_quad.far2_sq && !classify_fast(sqrtf(q2), near, order)) {
                    order = far_order_exact(&mv, kref, i, j);
                    near = order == 0;
                }
                if (!near) {
                    const double x64[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
                    const double nx64[3] = {m.n64[i], m.n64[n + i], m.n64[2 * n + i]};
                    if (fits && max_hi(x64[0], x64[1], x64[2]) < reach) {
                        val = far_entry_tri64(e4, x64, nx64, order, bcj, fc);
                    } else {
                        Elem64 e;
                        load_elem64(mk, j, e);
                        val = combine_entry(FarPair<double>::run(e, x64, nx64, order, f.k, f.wr), bcj, admj, PT);
                    }
                }
            }
            put(i, val.re, val.im);
        }
    } else {
        FarCol2 e2;
        if (tri) far_col2(mk, j, e2);
        else far_quad_stage(mk, j, st, lane);
        FusedCol fc;
        fc.bc = bcj;
        fc.yr = admj.re;
        fc.yi = admj.im;
        fc.tau = PT.tao;
        fc.b = PT.beta_im;
        fc.k2 = PT.k * PT.k;
        fc.wr = PT.wr;
        const FusedCol2 f2 = {dup2(fc.wr), dup2(fc.b), dup2(f.bwrf), dup2(f.k2f), dup2(-fc.tau),
                              dup2(f.twrf), dup2(fc.yr), dup2(fc.yi), dup2(-fc.yi), dup2(f.btf), dup2(f.btwf)};
#pragma unroll 1
        for (int r = 0; r < rpt; r += 2) {
            const int i = i0 + r;
            if (i >= n) break;
            // the two rows' data (the same for the warp's 32 columns)
            const float4 *row = m.row4 + 5 * (size_t)(i >> 1);   // items start at even rows
            const float4 v0 = row[0], v1 = row[1], v2 = row[2], v3 = row[3];
            const float2 v4 = *reinterpret_cast<const float2 *>(row + 4);
            const F2 D[3] = {vadd(vadd(dup2(cjh[0]), pk2(v0.x, v0.y)), vadd(dup2(cjl[0]), pk2(v1.z, v1.w))),
                             vadd(vadd(dup2(cjh[1]), pk2(v0.z, v0.w)), vadd(dup2(cjl[1]), pk2(v2.x, v2.y))),
                             vadd(vadd(dup2(cjh[2]), pk2(v1.x, v1.y)), vadd(dup2(cjl[2]), pk2(v2.z, v2.w)))};
            const F2 D2 = vfma(D[2], D[2], vfma(D[0], D[0], vmul(D[1], D[1])));
            const F2 nx[3] = {pk2(v3.x, v3.y), pk2(v3.z, v3.w), pk2(v4.x, v4.y)};
            float q2[2];
            unpk2(vmul(D2, dup2(isq2)), q2[0], q2[1]);
            // quadrature orders; 0: near or self
            int ord[2] = {2, 2};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (q2[h] <= c_quad.far2_sq) {
                    bool near = false;
                    if (i + h == j && kref == 0) near = true;
                    else if (!classify_fast(sqrtf(q2[h]), near, ord[h])) {
                        ord[h] = far_order_exact(&mv, kref, i + h < n ? i + h : i, j);
                        near = ord[h] == 0;
                    }
                    if (near) ord[h] = 0;
                }
            }
            FarSum2 o = {dup2(0.f), dup2(0.f), dup2(0.f)};
            if (ord[0] == 2 || ord[1] == 2) {
                if (tri) {
                    auto points = [&](auto diff) {
                        constexpr bool kDiff = decltype(diff)::value;
                        if (bcj == 0) far_tri2<0, kDiff>(fk, e2, D, D2, nx, f2, o);
                        else if (bcj == 1) far_tri2<1, kDiff>(fk, e2, D, D2, nx, f2, o);
                        else far_tri2<2, kDiff>(fk, e2, D, D2, nx, f2, o);
                    };
                    if (IMG && m.sym.nref > 1) points(std::true_type());
                    else points(std::false_type());
                } else {
                    if (bcj == 0) far_quad2<0>(fk, st, lane, D, nx, f2, o);
                    else if (bcj == 1) far_quad2<1>(fk, st, lane, D, nx, f2, o);
                    else far_quad2<2>(fk, st, lane, D, nx, f2, o);
                }
            }
            float er[2], ei[2], d[3][2];
            unpk2(vfma(o.ri, fk.m1, o.rr), er[0], er[1]);
            unpk2(o.ai, ei[0], ei[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (ord[h] == 0) er[h] = ei[h] = 0.f;
                else if (ord[h] > 2) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) unpk2(D[c], d[c][0], d[c][1]);
                    const float2 v = far_entry_general(&mv, kref, j, d[0][h], d[1][h], d[2][h], h ? v3.y : v3.x,
                                                       h ? v3.w : v3.z, h ? v4.y : v4.x, ord[h], fc);
                    er[h] = v.x;
                    ei[h] = v.y;
                }
            }
            put(i, er[0], ei[0]);
            if (i + 1 < n) put(i + 1, er[1], ei[1]);
        }
    }
}

constexpr int kRhsRows = 64;   // k_rhs without boundary columns: rows per block, a thread each
constexpr int kFarPerSm = kFarPerSmMax;   // resident k_far blocks per SM allowed by the launch bounds

// The grid's warps take the items in turn.  A queue of eight-warp tiles in place
// of that: 20480 triangles 3.23 against 3.33 ms, but 66 against 50 us at 1280,
// where its last tiles leave most SMs idle.
// ONE: the batch holds a single system, whose table then stays in constant
// operands instead of registers.  IMG: some mesh of the batch has symmetry
// images.
template <typename T, bool ONE, bool IMG>
__global__ void __launch_bounds__(256, kFarPerSm) k_far(const __grid_constant__ AsmBatch tb) {
    __shared__ float st[std::is_same<T, float>::value ? 8 : 1][kQuadRows][32];
    const int total = tb.far_off[tb.B];
    FarConst fk;
    if constexpr (std::is_same<T, float>::value) far_const(fk);
    for (int item = blockIdx.x * 8 + threadIdx.y; item < total; item += gridDim.x * 8) {
        const int b = ONE ? 0 : find_sys(tb.far_off, tb.B, item);
        const AsmSys &S = tb.sys[ONE ? 0 : b];
        const int local = item - tb.far_off[b];
        const int ntx = (S.m.n + 31) / 32;
        const int nref = IMG ? S.m.sym.nref : 1;
        for (int kref = 0; kref < nref; ++kref)
            far_tile<T, IMG>(S.m, S.f, (typename Vec2<T>::type *)S.A, S.lda, local % ntx, local / ntx * far_rows(S.m.n), kref,
                        fk, st[std::is_same<T, float>::value ? threadIdx.y : 0]);
    }
}

// ------------------------------------------------------------ near pairs
// One warp per entry of the near list: the self pair by warp_singular (FP64;
// warp_singular_f in FP32 for complex64 systems) plus NumCalc's free term,
// subdivided pairs by warp_subdivide with the
// kernel arithmetic in T; with symmetry planes every image of the entry's
// mask in image order.  The sum is added to the entry k_far wrote (its far
// images, or zero).
template <typename T>
__device__ __forceinline__ void near_pair(const DevMeshView &mv, const DevFreq &f, int2 ij,
                                          typename Vec2<T>::type *__restrict__ A, size_t lda, int *status,
                                          WarpScratch &ws) {
    const DevMesh m = to_dev(mv);
    const int lane = threadIdx.x, n = m.n;
    const int i = ij.x, j = ij.y & kMaxElements;
    const unsigned imask = (unsigned)ij.y >> kNearColBits;
    const double x64[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
    const double nx64[3] = {m.n64[i], m.n64[n + i], m.n64[2 * n + i]};
    Phys<double> P{f.k, f.wr, f.tao, f.beta_im};
    Phys<T> PT{(T)f.k, (T)f.wr, (T)f.tao, (T)f.beta_im};
    const int bcj = f.bc_type ? f.bc_type[j] : 0;
    cplx<T> sum = {T(0), T(0)};
    int err = kDevOk;
    for (int kref = 0; kref < 8; ++kref) {
        if (!((imask >> kref) & 1u)) continue;
        const DevMesh mk = image_mesh(m, kref);
        Elem64 e;
        load_elem64(mk, j, e);
        cplx<T> entry;
        if (kref == 0 && i == j) {
            KVals<double> sv;
            if constexpr (std::is_same<T, float>::value) {
                // FP32 rule on the vertices relative to the collocation point
                float pl[4][3];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int k = 0; k < 3; ++k) pl[a][k] = a < e.nv ? (float)(e.p[a][k] - x64[k]) : 0.f;
                const float nxf[3] = {(float)nx64[0], (float)nx64[1], (float)nx64[2]};
                const KVals<float> vf = warp_singular_f(e.nv, pl, nxf, f.kf, f.wrf);
                sv.G = {vf.G.re, vf.G.im};
                sv.H = {vf.H.re, vf.H.im};
                sv.HT = {vf.HT.re, vf.HT.im};
                sv.E = {vf.E.re, vf.E.im};
            } else {
                sv = warp_singular(e, x64, nx64, P, 0, nullptr).v;
            }
            cplx<double> a = combine_entry(sv, bcj, col_adm<double>(f, j, bcj), P);
            // free term, NC_EquationSystem.cpp:220-231
            const cplx<double> beta = {0.0, P.beta_im};
            if (bcj == 1) a += beta * (-(0.5 * P.tao));
            else a += (col_adm<double>(f, j, bcj) * beta - cplx<double>{1.0, 0.0}) * 0.5;
            entry = {(T)a.re, (T)a.im};
        } else if constexpr (std::is_same<T, double>::value) {
            // float tables only for the subdivision's fast decisions
            const float xhi[3] = {m.chi[i], m.chi[n + i], m.chi[2 * n + i]};
            const float xlo[3] = {m.clo[i], m.clo[n + i], m.clo[2 * n + i]};
            Elem32 ef;
            load_elem32(mk, j, xhi, xlo, ef);
            AsmSink<double> sink;
            sink.e = &e; sink.x = x64; sink.nx = nx64; sink.k = f.k; sink.wr = f.wr;
            sink.init();
            const int rc = warp_subdivide(e, m.area64[j], x64, ws, sink, &ef, m.isqa32[j]);
            if (rc != kDevOk) err = rc;
            KVals<double> v = sink.reduce();
            entry = combine_entry(v, bcj, col_adm<double>(f, j, bcj), PT);
        } else {
            const float xhi[3] = {m.chi[i], m.chi[n + i], m.chi[2 * n + i]};
            const float xlo[3] = {m.clo[i], m.clo[n + i], m.clo[2 * n + i]};
            const float nx32[3] = {(float)nx64[0], (float)nx64[1], (float)nx64[2]};
            Elem32 e32;
            load_elem32(mk, j, xhi, xlo, e32);
            AsmSink<float> sink;
            sink.e = &e32; sink.nx = nx32; sink.k = PT.k; sink.wr = PT.wr;
            sink.init();
            const int rc = warp_subdivide(e, m.area64[j], x64, ws, sink, &e32, m.isqa32[j]);
            if (rc != kDevOk) err = rc;
            KVals<float> v = sink.reduce();
            entry = combine_entry(v, bcj, col_adm<float>(f, j, bcj), PT);
        }
        if (image_negated(m, kref)) entry = entry * T(-1);
        sum += entry;
    }
    if (lane == 0) {
        typename Vec2<T>::type o = A[(size_t)i * lda + j];
        o.x += sum.re;
        o.y += sum.im;
        A[(size_t)i * lda + j] = o;
        if (err != kDevOk) atomicMax(status, err);
    }
}

// Bound by latency (each pair is a chain of subdivision levels, and the code is
// long), so the float form takes four blocks per SM at 64 registers: 61440 pairs
// 400 -> 280 us, 3840 pairs 30 -> 27 (three blocks 313, five 291).  The FP64 form
// keeps two: its pipe is the limit.
template <typename T>
__global__ void __launch_bounds__(256, std::is_same<T, float>::value ? 4 : 2) k_near(const __grid_constant__ AsmBatch tb, unsigned *ctr) {
    __shared__ WarpScratch ws_all[8];
    WarpScratch &ws = ws_all[threadIdx.y];
    const int total = tb.near_off[tb.B];
    while (true) {
        int item = 0;
        if (threadIdx.x == 0) item = (int)atomicAdd(ctr, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        const int b = find_sys(tb.near_off, tb.B, item);
        const AsmSys &S = tb.sys[b];
        const int2 ij = S.near[item - tb.near_off[b]];
        near_pair<T>(S.m, S.f, ij, (typename Vec2<T>::type *)S.A, S.lda, S.status, ws);
        __syncwarp();
    }
    queue_exit(ctr);
}

// Images of the incident waves in the symmetry planes: step kref reflects a
// plane-wave direction (negates one component) or a point source (2 c - x)
// across the plane normal to axis rdir[kref]; the reflection factor of image
// kref is the element images' (NC_ReflectPointVector, NC_3dFunctions.cpp:181-242).
__device__ __forceinline__ void reflect_source(const DevSym &sy, int kref, double v[3], bool point) {
    const int d = sy.rdir[kref];
    if (point) v[d] = __dsub_rn(2.0 * sy.coord[d], v[d]);
    else v[d] = -v[d];
}

// Plane waves take their phase at x minus the positions of the planes
// present (NC_EquationSystem.cpp:1743-1748, NC_PostProcessing.cpp:794-799).
__device__ __forceinline__ void plane_wave_origin(const DevSym &sy, const double x[3], double xs[3]) {
    for (int k = 0; k < 3; ++k) xs[k] = ((sy.axes >> k) & 1u) ? x[k] - sy.coord[k] : x[k];
}

// Incident waves at a collocation point (NC_IncidentWaveRHS,
// NC_EquationSystem.cpp:1731-1812), with their symmetry-plane images.
__device__ cplx<double> incident_rhs(const DevSym &sy, const DevFreq &f, const double x[3], const double nx[3]) {
    cplx<double> zrc = {0.0, 0.0};
    const cplx<double> bt = {0.0, f.beta_im * f.tao};
    double xs[3];
    plane_wave_origin(sy, x, xs);
    for (int s = 0; s < f.n_plane; ++s) {
        double d[3] = {f.pw_dir[3 * s], f.pw_dir[3 * s + 1], f.pw_dir[3 * s + 2]};
        const cplx<double> amp = ld_c(f.pw_amp, s);
        for (int kref = 0; kref < sy.nref; ++kref) {
            if (kref > 0) reflect_source(sy, kref, d, false);
            const double rf = ((sy.rneg >> kref) & 1u) ? -1.0 : 1.0;
            const double ph = (d[0] * xs[0] + d[1] * xs[1] + d[2] * xs[2]) * f.wr;
            double sn, cs;
            sincos(ph, &sn, &cs);
            const cplx<double> zg = cplx<double>{cs * rf, sn * rf} * amp;
            const double re1 = f.wr * (d[0] * nx[0] + d[1] * nx[1] + d[2] * nx[2]);
            const cplx<double> zv = {-zg.im * re1, zg.re * re1};
            zrc -= zg + zv * bt;
        }
    }
    for (int s = 0; s < f.n_point; ++s) {
        double p[3] = {f.ps_xyz[3 * s], f.ps_xyz[3 * s + 1], f.ps_xyz[3 * s + 2]};
        const cplx<double> amp = ld_c(f.ps_amp, s);
        for (int kref = 0; kref < sy.nref; ++kref) {
            if (kref > 0) reflect_source(sy, kref, p, true);
            const double rf = ((sy.rneg >> kref) & 1u) ? -1.0 : 1.0;
            double d[3] = {x[0] - p[0], x[1] - p[1], x[2] - p[2]};
            const double r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
            d[0] /= r; d[1] /= r; d[2] /= r;
            double sn, cs;
            sincos(f.wr * r, &sn, &cs);
            const double re2 = rf / kPI4 / r;
            const cplx<double> zg = cplx<double>{cs * re2, sn * re2} * amp;
            const double re1 = d[0] * nx[0] + d[1] * nx[1] + d[2] * nx[2];
            const cplx<double> zv = cplx<double>{-re1 / r, f.wr * re1} * zg;
            zrc -= zg + zv * bt;
        }
    }
    return zrc;
}

// Free term of the prescribed value (NC_EquationSystem.cpp:233-244) and
// incident waves of row i.
__device__ cplx<double> rhs_row(const DevMesh &m, const DevFreq &f, int i, const double x[3], const double nx[3]) {
    const int n = m.n, nv = m.nvert[i];
    const int bci = f.bc_type ? f.bc_type[i] : 0;
    cplx<double> z0 = {0.0, 0.0}, zbvi = {0.0, 0.0};
    if (f.bc_val)
        for (int a = 0; a < nv; ++a) zbvi += ld_c(f.bc_val, a * n + i);
    zbvi = {zbvi.re / (double)nv, zbvi.im / (double)nv};
    const cplx<double> beta = {0.0, f.beta_im};
    if (bci != 1) z0 += ((zbvi * beta) * f.tao) * 0.5;
    else z0 += (zbvi * f.tao) * 0.5;
    if (f.n_plane + f.n_point > 0) z0 += incident_rhs(m.sym, f, x, nx);
    return z0;
}

// Right-hand side (FP64): the row's own terms (rhs_row) and the columns whose
// prescribed values are nonzero (Zrsintel[4], NC_EquationSystem.cpp:188-198),
// each with all its images: nodal values in the image's node order, velocity
// values negated with the reflection factor, no factor on the term itself
// (NC_ReflectElement, NC_3dFunctions.cpp:410-415; NC_AssembleTBEM).
//
// Bound by the FP64 pipe, which issues whole warps, so the lanes have to be
// full.  Without such columns a thread takes a row (kRhsRows per block, two
// warps, so that small systems still spread over the SMs): 19 us for 20480
// rows and one source, 194 us with a warp per row and one lane at work.  With columns a warp takes a row and its lanes
// the columns: far columns are integrated whole in their lane, subdivided ones
// and the self pair by the warp, one at a time.  Integrating every column with
// the warp left 28 of 32 lanes idle on the 4-point rule: 3072 quadrilaterals with
// one image and 48 such columns 8.2 -> 1.5 ms.  The rows beside those columns
// subdivide many of them and are neighbours in the element order, so a block
// takes rows that lie far apart: 1.49 -> 1.39 ms; two blocks per SM at 128
// registers instead of one at 255: 1.23.  Staging the columns' points in shared
// memory (1.57 from 1.39) or dealing them to a cluster (1.83) cost more in
// waits than they saved.
__global__ void __launch_bounds__(256, 2) k_rhs(const __grid_constant__ AsmBatch tb) {
    __shared__ WarpScratch ws_all[8];
    const int sb = find_sys(tb.rhs_off, tb.B, blockIdx.x);
    const AsmSys &S = tb.sys[sb];
    const DevMesh m = to_dev(S.m);
    const DevFreq &f = S.f;
    double2 *b = (double2 *)S.b;
    const int lane = threadIdx.x, w = threadIdx.y;
    const int n = m.n, blk = blockIdx.x - tb.rhs_off[sb];
    if (f.n_bc_cols == 0) {
        const int t = w * 32 + lane, i = blk * kRhsRows + t;
        if (t >= kRhsRows || i >= n) return;
        const double x[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
        const double nx[3] = {m.n64[i], m.n64[n + i], m.n64[2 * n + i]};
        const cplx<double> z = rhs_row(m, f, i, x, nx);
        b[i] = make_double2(z.re, z.im);
        return;
    }
    const int i = w * (tb.rhs_off[sb + 1] - tb.rhs_off[sb]) + blk;   // neighbours in different blocks
    if (i >= n) return;
    WarpScratch &ws = ws_all[w];
    const double x[3] = {m.c64[i], m.c64[n + i], m.c64[2 * n + i]};
    const double nx[3] = {m.n64[i], m.n64[n + i], m.n64[2 * n + i]};
    const Phys<double> P{f.k, f.wr, f.tao, f.beta_im};
    cplx<double> zw = {0.0, 0.0};   // the warp's terms (same on every lane)
    int err = kDevOk;
    RhsSink sink;   // the lane's far columns
    sink.x = x; sink.nx = nx; sink.P = P;
    sink.init();
    for (int kref = 0; kref < m.sym.nref; ++kref) {
        const DevMesh mk = image_mesh(m, kref);
        const bool neg = image_negated(m, kref);
        auto values = [&](int jc, int bcj, cplx<double> bc[4]) {
            const double vs = (bcj != 1 && neg) ? -1.0 : 1.0;
            const int nvj = m.nvert[jc];
            for (int a = 0; a < 4; ++a)
                bc[a] = a < nvj ? ld_c(f.bc_val, image_node(a, kref, nvj) * n + jc) * vs : cplx<double>{0.0, 0.0};
        };
        for (int base = 0; base < f.n_bc_cols; base += 32) {
            const bool valid = base + lane < f.n_bc_cols;
            bool whole = false;   // taken by the whole warp
            if (valid) {
                const int jc = f.bc_cols[base + lane];
                const double rd = ratio0_exact(mk, jc, x);
                whole = rd < kTolf || (kref == 0 && jc == i);
                if (!whole) {
                    const int order = gauss_order(rd), bcj = f.bc_type ? f.bc_type[jc] : 0;
                    Elem64 e;
                    load_elem64(mk, jc, e);
                    cplx<double> bc[4];
                    values(jc, bcj, bc);
                    sink.e = &e; sink.bc = bc; sink.bctype = bcj == 1 ? 1 : 0;
                    const int np = sub_npts(e.nv, order);
                    for (int g = 0; g < np; ++g) {
                        double s, t, wq;
                        sub_point(e.nv, order, g, 0.0, 0.0, 1.0, s, t, wq);
                        sink.add(s, t, wq);
                    }
                }
            }
            unsigned todo = __ballot_sync(0xffffffffu, whole);
            while (todo) {
                const int jc = f.bc_cols[base + __ffs(todo) - 1];
                todo &= todo - 1;
                const int bcj = f.bc_type ? f.bc_type[jc] : 0;
                Elem64 e;
                load_elem64(mk, jc, e);
                cplx<double> bc[4];
                values(jc, bcj, bc);
                if (kref == 0 && jc == i) {
                    zw += warp_singular(e, x, nx, P, bcj == 1 ? 2 : 1, bc).rhs;
                } else {
                    RhsSink ns;
                    ns.e = &e; ns.x = x; ns.nx = nx; ns.bc = bc; ns.bctype = bcj == 1 ? 1 : 0; ns.P = P;
                    ns.init();
                    // float tables for the subdivision's fast decisions
                    const float xhi[3] = {m.chi[i], m.chi[n + i], m.chi[2 * n + i]};
                    const float xlo[3] = {m.clo[i], m.clo[n + i], m.clo[2 * n + i]};
                    Elem32 ef;
                    load_elem32(mk, jc, xhi, xlo, ef);
                    const int rc = warp_subdivide(e, m.area64[jc], x, ws, ns, &ef, m.isqa32[jc]);
                    if (rc != kDevOk) err = rc;
                    zw += ns.reduce();
                }
            }
        }
    }
    const cplx<double> zf = sink.reduce();
    if (lane == 0) {
        const cplx<double> z = rhs_row(m, f, i, x, nx) + zw + zf;
        b[i] = make_double2(z.re, z.im);
        if (err != kDevOk) atomicMax(S.status, err);
    }
}

// Element potentials and nodal normal velocities after the solve
// (NC_WriteResultsObjectMesh, NC_PostProcessing.cpp:389-410).
__global__ void __launch_bounds__(256) k_fields(const __grid_constant__ ProjBatch tb) {
    const int sb = find_sys(tb.fld_off, tb.B, blockIdx.x);
    const ProjSys &S = tb.sys[sb];
    const DevMeshView &mv = S.m;
    const DevFreq &f = S.f;
    const double2 *x = (const double2 *)S.x;
    double2 *phi = (double2 *)S.phi, *vel = (double2 *)S.vel;
    int *ivi = S.ivi;
    const int j = (blockIdx.x - tb.fld_off[sb]) * blockDim.x + threadIdx.x;
    const int n = mv.n;
    if (j >= n) return;
    const int bc = f.bc_type ? f.bc_type[j] : 0;
    const int nv = mv.nvert[j];
    const cplx<double> xj = {x[j].x, x[j].y};
    cplx<double> p, v[4];
    for (int a = 0; a < 4; ++a)
        v[a] = (f.bc_val && a < nv) ? ld_c(f.bc_val, a * n + j) : cplx<double>{0.0, 0.0};
    if (bc == 1) {
        p = v[0];
        for (int a = 0; a < 4; ++a) v[a] = a < nv ? xj : cplx<double>{0.0, 0.0};
    } else {
        p = xj;
        if (bc == 2 && f.adm) {
            const cplx<double> z1 = (xj * ld_c(f.adm, j)) * f.tao;
            for (int a = 0; a < nv; ++a) v[a] -= z1;
        }
    }
    int any = 0;
    for (int a = 0; a < nv; ++a)
        if (sqrt(v[a].re * v[a].re + v[a].im * v[a].im) > kEPSY) any = 1;
    phi[j] = make_double2(p.re, p.im);
    for (int a = 0; a < 4; ++a) vel[a * n + j] = make_double2(v[a].re, v[a].im);
    float2 *phi32 = (float2 *)S.phi32, *vel32 = (float2 *)S.vel32;
    phi32[j] = make_float2((float)p.re, (float)p.im);
    for (int a = 0; a < 4; ++a) vel32[a * n + j] = make_float2((float)v[a].re, (float)v[a].im);
    ivi[j] = any;
}

// Far-pair projection of a flat triangle without velocity terms, fused
// (NC_IntegrationTBEM, NC_PostProcessing.cpp:1217-1322, with phi factored out
// of the quadrature sum): per point Gw = w J e^{i wr r}/(4 pi r), Gi =
// Gw (-1/r + i wr), r^.n_y = (D.n_y)/r (constant numerator on a flat
// element);
//   P  += Gi (r^.n_y)
//   U  += Gw [(r^.n_y)(k^2 - 3/r^2) + i 3 wr (r^.n_y)/r] / r * (y - x)
//   T  -= Gi / r
// and the element adds phi P to the potential and phi (U + T n_y) to the
// gradient.
template <int NP, int O0>
__device__ __forceinline__ void proj_tri_points(const Elem32 &e, float dny, float k2, float wr, float2 &P,
                                                float2 (&U)[3], float2 &T) {
#pragma unroll
    for (int g = 0; g < NP; ++g) {
        const float ss = c_trif[O0 + g][0] - (1.0f / 3.0f), tt = c_trif[O0 + g][1] - (1.0f / 3.0f);
        const float wj = c_trif[O0 + g][2] * e.J * (float)(1.0 / kPI4);
        float d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = fmaf(tt, e.b[k], fmaf(ss, e.a[k], e.D[k]));
        const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const float ir = rsqrt_approx(r2), r = r2 * ir;
        float sn, cs;
        phase_sincos(wr * r, &sn, &cs);
        const float amp = wj * ir;
        const float gr = cs * amp, gi = sn * amp;                              // Gw
        const float hr = fmaf(-gr, ir, -gi * wr), hi = fmaf(gr, wr, -gi * ir);   // Gi
        const float dn = dny * ir;                                           // r^.n_y
        P.x = fmaf(hr, dn, P.x);
        P.y = fmaf(hi, dn, P.y);
        const float ir2 = ir * ir;
        const float f1r = dn * (k2 - 3.0f * ir2), f1i = 3.0f * wr * dn * ir;
        const float ur = (gr * f1r - gi * f1i) * ir, ui = (gr * f1i + gi * f1r) * ir;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            U[k].x = fmaf(ur, d[k], U[k].x);
            U[k].y = fmaf(ui, d[k], U[k].y);
        }
        T.x = fmaf(-hr, ir, T.x);
        T.y = fmaf(-hi, ir, T.y);
    }
}

// Element data of image kref for the projection: potential and nodal
// velocities times the reflection factor, velocities in the image's node
// order (NC_ContributionTBEM, NC_PostProcessing.cpp:925-940).
template <typename T>
__device__ __forceinline__ void proj_elem_data(const double2 *phi, const double2 *vel, const float2 *phi32,
                                               const float2 *vel32, int n, int j, int nv, bool iv, int kref,
                                               bool neg, cplx<T> &ph, cplx<T> vl[4]) {
    const T sg = neg ? T(-1) : T(1);
    if constexpr (std::is_same<T, double>::value) {
        ph = cplx<T>{phi[j].x, phi[j].y} * sg;
        for (int a = 0; a < 4; ++a) {
            const int src = image_node(a, kref, nv);
            vl[a] = (iv && a < nv) ? cplx<T>{vel[src * n + j].x, vel[src * n + j].y} * sg : cplx<T>{0, 0};
        }
    } else {
        const float2 p2 = phi32[j];
        ph = cplx<T>{p2.x, p2.y} * sg;
        for (int a = 0; a < 4; ++a) {
            const float2 v2 = (iv && a < nv) ? vel32[image_node(a, kref, nv) * n + j] : make_float2(0.f, 0.f);
            vl[a] = cplx<T>{v2.x, v2.y} * sg;
        }
    }
}

// Potential and gradient of point p from the element sums (FP64): the tau
// factor, then the incident field with its images (NC_ContributionIncidentWaves,
// NC_PostProcessing.cpp:776-866).
__device__ void project_finish(const DevMesh &m, const DevFreq &f, const double x64[3], int p, cplx<double> sp,
                               cplx<double> sg[3], double2 *pot, double2 *grad) {
    if (f.tao != 1.0) {
        sp = sp * f.tao;
        for (int kk = 0; kk < 3; ++kk) sg[kk] = sg[kk] * f.tao;
    }
    if (f.n_plane || f.n_point) {
        const DevSym &sy = m.sym;
        double xs[3];
        plane_wave_origin(sy, x64, xs);
        for (int s = 0; s < f.n_plane; ++s) {
            double d[3] = {f.pw_dir[3 * s], f.pw_dir[3 * s + 1], f.pw_dir[3 * s + 2]};
            const cplx<double> amp = ld_c(f.pw_amp, s);
            for (int kref = 0; kref < sy.nref; ++kref) {
                if (kref > 0) reflect_source(sy, kref, d, false);
                const double rf = ((sy.rneg >> kref) & 1u) ? -1.0 : 1.0;
                double sn, cs;
                sincos((d[0] * xs[0] + d[1] * xs[1] + d[2] * xs[2]) * f.wr, &sn, &cs);
                const cplx<double> zg = cplx<double>{cs * rf, sn * rf} * amp;
                sp += zg;
                const cplx<double> zv = {-zg.im * f.wr, zg.re * f.wr};
                for (int kk = 0; kk < 3; ++kk) sg[kk] += zv * d[kk];
            }
        }
        for (int s = 0; s < f.n_point; ++s) {
            double q[3] = {f.ps_xyz[3 * s], f.ps_xyz[3 * s + 1], f.ps_xyz[3 * s + 2]};
            const cplx<double> amp = ld_c(f.ps_amp, s);
            for (int kref = 0; kref < sy.nref; ++kref) {
                if (kref > 0) reflect_source(sy, kref, q, true);
                const double rf = ((sy.rneg >> kref) & 1u) ? -1.0 : 1.0;
                double d[3] = {x64[0] - q[0], x64[1] - q[1], x64[2] - q[2]};
                const double r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
                d[0] /= r; d[1] /= r; d[2] /= r;
                double sn, cs;
                sincos(f.wr * r, &sn, &cs);
                const double re2 = rf / kPI4 / r;
                const cplx<double> zg = cplx<double>{cs * re2, sn * re2} * amp;
                sp += zg;
                const cplx<double> zv = cplx<double>{-1.0 / r, f.wr} * zg;
                for (int kk = 0; kk < 3; ++kk) sg[kk] += zv * d[kk];
            }
        }
    }
    pot[p] = make_double2(sp.re, sp.im);
    if (grad)
        for (int kk = 0; kk < 3; ++kk) grad[3 * p + kk] = make_double2(sg[kk].re, sg[kk].im);
}

// Field projection, one warp per point: lanes sweep the elements (and their
// symmetry images) 32 at a time; regular pairs in the lane, subdivided pairs
// by the whole warp.
template <typename T>
__global__ void __launch_bounds__(256, 2) k_project(const __grid_constant__ ProjBatch tb) {
    __shared__ WarpScratch ws_all[8];
    const int sb = find_sys(tb.pt_off, tb.B, blockIdx.x);
    const ProjSys &S = tb.sys[sb];
    const DevMesh m = to_dev(S.m);
    const DevFreq &f = S.f;
    const double2 *phi = (const double2 *)S.phi, *vel = (const double2 *)S.vel;
    const float2 *phi32 = (const float2 *)S.phi32, *vel32 = (const float2 *)S.vel32;
    const int *ivi = S.ivi;
    const int npts = S.npts;
    const double *pts = S.pts;
    double2 *pot = (double2 *)S.pot, *grad = (double2 *)S.grad;
    int *status = S.status;
    const int lane = threadIdx.x, w = threadIdx.y;
    const int n = m.n;
    const int p = (blockIdx.x - tb.pt_off[sb]) * 8 + w;
    if (p >= npts) return;
    WarpScratch &ws = ws_all[w];
    const double x64[3] = {pts[3 * p], pts[3 * p + 1], pts[3 * p + 2]};
    float xhi[3], xlo[3];
    for (int k = 0; k < 3; ++k) {
        xhi[k] = (float)x64[k];
        xlo[k] = (float)(x64[k] - (double)xhi[k]);
    }
    ProjAcc<T> acc;
    acc.p = acc.g[0] = acc.g[1] = acc.g[2] = cmk(T(0), T(0));
    const T k = (T)f.k, wr = (T)f.wr;
    int err = kDevOk;
    for (int kref = 0; kref < m.sym.nref; ++kref) {
        const DevMesh mk = image_mesh(m, kref);
        const bool neg = image_negated(m, kref);
        for (int base = 0; base < n; base += 32) {
            const int j = base + lane;
            const bool valid = j < n;
            bool near = false;
            int order = 2;
            if (valid) {
                // element data in T (float copies for the float path: no FP64 conversions)
                const bool iv = ivi[j] != 0;
                const int nv = m.nvert[j];
                cplx<T> ph, vl[4];
                proj_elem_data<T>(phi, vel, phi32, vel32, n, j, nv, iv, kref, neg, ph, vl);
                if constexpr (std::is_same<T, double>::value) {
                    const double rd = ratio0_exact(mk, j, x64);
                    near = rd < kTolf;
                    if (!near) {
                        order = gauss_order(rd);
                        Elem64 e;
                        load_elem64(mk, j, e);
                        const int np = e.nv == 3 ? tri_count(order) : quad_count(order);
                        for (int g = 0; g < np; ++g) {
                            double s, t, wq;
                            sub_point(e.nv, order, g, 0.0, 0.0, 1.0, s, t, wq);
                            QPoint<double> q;
                            map_point(e, s, t, x64, wq, q);
                            proj_point(q, ph, vl, e.nv, iv, k, wr, acc);
                        }
                    }
                } else {
                    Elem32 e;
                    load_elem32(mk, j, xhi, xlo, e);
                    const float q2 = (e.D[0] * e.D[0] + e.D[1] * e.D[1] + e.D[2] * e.D[2]) * (m.isqa32[j] * m.isqa32[j]);
                    if (q2 <= c_quad.far2_sq && !classify_fast(sqrtf(q2), near, order)) {
                        const double rd = ratio0_exact(mk, j, x64);
                        near = rd < kTolf;
                        if (!near) order = gauss_order(rd);
                    }
                    if (!near && e.nv == 3 && !iv) {
                        // fused flat-triangle path (no velocity terms)
                        float2 P = make_float2(0.f, 0.f), U[3], Tn = make_float2(0.f, 0.f);
                        U[0] = U[1] = U[2] = make_float2(0.f, 0.f);
                        const float dny = e.D[0] * e.n[0] + e.D[1] * e.n[1] + e.D[2] * e.n[2];
                        const float k2 = (float)k * (float)k;
                        if (order <= 2) proj_tri_points<4, 0>(e, dny, k2, (float)wr, P, U, Tn);
                        else if (order == 3) proj_tri_points<7, 4>(e, dny, k2, (float)wr, P, U, Tn);
                        else proj_tri_points<13, 11>(e, dny, k2, (float)wr, P, U, Tn);
                        const cplx<float> pp = ph * cplx<float>{P.x, P.y};
                        acc.p.re += pp.re;
                        acc.p.im += pp.im;
#pragma unroll
                        for (int kk = 0; kk < 3; ++kk) {
                            const cplx<float> gg = ph * cplx<float>{fmaf(Tn.x, e.n[kk], U[kk].x), fmaf(Tn.y, e.n[kk], U[kk].y)};
                            acc.g[kk].re += gg.re;
                            acc.g[kk].im += gg.im;
                        }
                    } else if (!near) {
                        const int np = e.nv == 3 ? tri_count(order) : quad_count(order);
                        for (int g = 0; g < np; ++g) {
                            float s, t, wq;
                            if (e.nv == 3) {
                                const int o = tri_offset(order) + g;
                                s = c_trif[o][0]; t = c_trif[o][1]; wq = c_trif[o][2];
                            } else {
                                const int a = g / order, b = g - a * order;
                                s = c_glxf[order][a]; t = c_glxf[order][b];
                                wq = c_glwf[order][a] * c_glwf[order][b];
                            }
                            QPoint<float> q;
                            map_point(e, s, t, wq, q);
                            proj_point(q, ph, vl, e.nv, iv, k, wr, acc);
                        }
                    }
                }
            }
            unsigned todo = __ballot_sync(0xffffffffu, valid && near);
            while (todo) {
                const int L = __ffs(todo) - 1;
                todo &= todo - 1;
                const int jl = base + L;
                Elem64 e;
                load_elem64(mk, jl, e);
                const bool iv = ivi[jl] != 0;
                cplx<T> ph, vl[4];
                proj_elem_data<T>(phi, vel, phi32, vel32, n, jl, e.nv, true, kref, neg, ph, vl);
                ProjAcc<T> r;
                int rc;
                if constexpr (std::is_same<T, double>::value) {
                    ProjSink<double> sink;
                    sink.e = &e; sink.x = x64; sink.phi = ph; sink.vel = vl; sink.ivi = iv; sink.k = k; sink.wr = wr;
                    sink.init();
                    rc = warp_subdivide(e, m.area64[jl], x64, ws, sink);
                    r = sink.reduce();
                } else {
                    Elem32 e32;   // float tables: the arithmetic and the fast decisions
                    load_elem32(mk, jl, xhi, xlo, e32);
                    ProjSink<float> sink;
                    sink.e = &e32; sink.phi = ph; sink.vel = vl; sink.ivi = iv; sink.k = k; sink.wr = wr;
                    sink.init();
                    rc = warp_subdivide(e, m.area64[jl], x64, ws, sink, &e32, m.isqa32[jl]);
                    r = sink.reduce();
                }
                if (rc != kDevOk) err = rc;
                if (lane == 0) {
                    acc.p += r.p;
                    for (int kk = 0; kk < 3; ++kk) acc.g[kk] += r.g[kk];
                }
            }
        }
    }
    // FP64 cross-lane reduction
    cplx<double> sp = warp_sum(cplx<double>{(double)acc.p.re, (double)acc.p.im});
    cplx<double> sg[3];
    for (int kk = 0; kk < 3; ++kk) sg[kk] = warp_sum(cplx<double>{(double)acc.g[kk].re, (double)acc.g[kk].im});
    if (lane == 0) {
        project_finish(m, f, x64, p, sp, sg, pot, grad);
        if (err != kDevOk) atomicMax(status, err);
    }
}

// Projection with lanes = evaluation points.  A block takes some groups of
// points (32 lanes x kP points per lane) and a slice of the elements, which it
// stages proj_chunk at a time in shared memory; its 8 warps are pgb point
// groups x 8 / pgb element parts (proj_batch_finish).  An element's data is
// the same for all lanes: one broadcast read serves 32 kP points.
//
// In float a lane holds two points and the 4-point rule runs in packed
// arithmetic: the kernel was bound by instruction issue (about 62 FP32
// instructions per evaluation), now by the FMA pipe.  The distance, the
// phase k r and its reduction are rounded operation by operation as in
// map_point / phase_sincos: at k r of hundreds of radians their rounding is
// the result's error.  The rest is regrouped: with G = w u e^{i wr r}, u = 1/r
// and alpha = u^2 - i wr u, an element's sums over its points
//   P0 = -sum (d.n_y) G alpha
//   G0 = sum n_y G alpha + (d.n_y) u^2 (k^2 G - 3 G alpha) d
// do not depend on the unknowns: the element adds W P0 to the potential and
// W G0 to the gradient, W = phi J / 4 pi (NC_IntegrationTBEM,
// NC_PostProcessing.cpp:1217-1322, for H = G (-u + i wr) (r^.n_y)).  So the
// right-hand sides of one matrix (NR > 1) share them.  Elements with nodal
// velocities add V G and V G alpha d per point, V = -(velocity at the point)
// J / 4 pi.  d.n_y is constant on a flat triangle, so its normal terms wait
// for the element's sum.  A right-hand side's sums are formed by the same
// operations in the same order whatever NR is.
//
// Points of higher order and subdivided pairs take proj_whole and
// warp_subdivide.  Partial sums go to ProjSys::part per (slice, point);
// k_project_sum adds the slices (FP64) and finishes the point.  In float, 11950
// points on 20480 elements 3.87 -> 2.14 ms (41 instructions per evaluation,
// FMA pipe 64 % active on a smaller case), 64 points on 5120 elements 225 ->
// 17 us (40 warps swept the elements before), 3072 quadrilaterals with an
// image and velocities, 1730 points 1.63 -> 0.19 ms; FP64, 1730 points on 5120
// elements 17.1 -> 4.3 ms.
constexpr int kProjSlice = 256;   // most elements per slice
constexpr int kProjStep = 16;     // fewest elements per slice
// Elements of a slice whose terms are added one by one, each with two roundings at
// the sum's size; the runs are then added up.  One sum over a slice (476 elements
// where the scratch holds 43 slices) left gradients near the surface up to a fifth
// further from 64-bit ones than single roundings had; runs of 64 leave them 0.6 ..
// 0.9 of that, in the same time.
constexpr int kProjRun = 64;
// elements staged at a time (the stage and the subdivision scratch share 48 KB)
__host__ __device__ constexpr int proj_chunk(int nr) { return nr <= 2 ? 16 : 8; }
// Resident blocks, 2 on each of 152 SMs: a number and not the device's own, since
// the split decides the order of a field's sums and a result should not depend
// on the device.
constexpr int kProjSlots = 304;

template <typename T> struct ProjLane;
template <> struct ProjLane<float> { using R = F2; static constexpr int kP = 2, kPart = 2; };
template <> struct ProjLane<double> { using R = double; static constexpr int kP = 1, kPart = 4; };

// A staged element.  Float triangles: v[0..2] centre, high parts, v[3..5] low
// parts, 6 a, 9 b, 12 n.  Else, per point g: 6 + 3 g position (float: offset
// from the centre, staged as above), 18 + 3 g normal (FP64 triangles: 18 n),
// 30 + g weight (quadrilaterals).  FP64 subtracts positions, as map_point does:
// an offset from the centroid leaves the rounding of the centroid and of the
// difference in all points of the element (scattered fields 1 m away at k = 73
// up to 1.4 times as far from 80-bit ones).  Per right-hand side W (re, im, -im,
// -re) and, where some right-hand side has nodal velocities, V of the points.
template <typename T, int NR> struct ProjElem {
    typename ProjLane<T>::R v[34], W[NR][4], V[NR][4][3];
    float hi[3], lo[3], isq2;
    int nv, iv, far;   // far: the vertices' largest component (FP64; max_hi)
};

template <typename T>
__device__ __forceinline__ void proj_put(typename ProjLane<T>::R *v, cplx<T> z) {
    vdup(v[0], z.re);
    vdup(v[1], z.im);
    vdup(v[2], -z.im);
}

// Thread g (0..3) of element j's four: its part of the staged element.  sys:
// the right-hand sides' systems (nr of them).
template <typename T, int NR>
__device__ void proj_stage(const ProjSys *sys, int nr, const DevMesh &m, const DevMesh &mk, int kref, bool neg, int j,
                           int g, ProjElem<T, NR> &o) {
    const int n = m.n, nv = m.nvert[j];
    const T i4pi = T(1.0 / kPI4);
    T fac = i4pi, sh[4];   // J / 4 pi (1 / 4 pi on quadrilaterals); shape functions at point g
    if (nv == 3) {
        sh[0] = (T)c_quad.tri[g][0];
        sh[1] = (T)c_quad.tri[g][1];
        sh[2] = T(1) - sh[0] - sh[1];
        sh[3] = T(0);
        T J;
        if constexpr (std::is_same<T, float>::value) {
            J = mk.t32[9 * n + j];
            if (g < 3) {   // one of a, b, n each
                for (int k = 0; k < 3; ++k) vdup(o.v[6 + 3 * g + k], mk.t32[(3 * g + k) * n + j]);
            }
        } else {
            FarCol64 f;
            far_col64(mk, j, f);
            J = f.J4 * kPI4;
            for (int k = 0; k < 3; ++k) {
                o.v[6 + 3 * g + k] = f.c[k] + fma(c_far64[g][1], f.b[k], fma(c_far64[g][0], f.a[k], f.cl[k]));
                if (g == 0) o.v[18 + k] = f.n[k];
            }
        }
        fac = J * i4pi;
    } else {
        QPoint<T> q;
        if constexpr (std::is_same<T, float>::value) {
            Elem32 e;
            const float zero[3] = {0.f, 0.f, 0.f};
            load_elem32(mk, j, zero, zero, e);
            e.D[0] = e.D[1] = e.D[2] = 0.f;
            map_point(e, c_glxf[2][g >> 1], c_glxf[2][g & 1], c_glwf[2][g >> 1] * c_glwf[2][g & 1], q);
        } else {
            Elem64 e;
            load_elem64(mk, j, e);
            const double zero[3] = {0.0, 0.0, 0.0};
            map_point(e, c_quad.glx[2][g >> 1], c_quad.glx[2][g & 1], zero,
                      c_quad.glw[2][g >> 1] * c_quad.glw[2][g & 1], q);
        }
        for (int k = 0; k < 3; ++k) {
            vdup(o.v[6 + 3 * g + k], q.d[k]);
            vdup(o.v[18 + 3 * g + k], q.ny[k]);
        }
        vdup(o.v[30 + g], q.wj);
        for (int a = 0; a < 4; ++a) sh[a] = q.sh[a];
    }
    if (g == 0) {
        o.nv = nv;
        const float q = m.isqa32[j];
        o.isq2 = q * q;
        for (int k = 0; k < 3; ++k) {
            o.hi[k] = mk.chi[k * n + j];
            o.lo[k] = mk.clo[k * n + j];
            if constexpr (std::is_same<T, float>::value) {
                vdup(o.v[k], o.hi[k]);
                vdup(o.v[3 + k], o.lo[k]);
            }
        }
        o.far = 0;
        if constexpr (std::is_same<T, double>::value) {
            for (int a = 0; a < nv; ++a)
                o.far = max(o.far, max_hi(mk.v64[3 * a * n + j], mk.v64[(3 * a + 1) * n + j], mk.v64[(3 * a + 2) * n + j]));
        }
    }
    bool any = false;
#pragma unroll 1
    for (int r = 0; r < nr; ++r) any |= sys[r].ivi[j] != 0;
    if (g == 0) o.iv = any;
#pragma unroll 1
    for (int r = 0; r < nr; ++r) {
        const ProjSys &S = sys[r];
        const bool iv = S.ivi[j] != 0;
        cplx<T> ph, vl[4];
        proj_elem_data<T>((const double2 *)S.phi, (const double2 *)S.vel, (const float2 *)S.phi32,
                          (const float2 *)S.vel32, n, j, nv, iv, kref, neg, ph, vl);
        if (g == 0) {
            proj_put<T>(o.W[r], ph * fac);
            vdup(o.W[r][3], -(ph.re * fac));
        }
        if (any) {
            cplx<T> z = {T(0), T(0)};
            for (int a = 0; a < 4; ++a) z += vl[a] * sh[a];
            proj_put<T>(o.V[r][g], z * -fac);
        }
    }
}

template <typename R> struct RAcc { R pr, pi, gr[3], gi[3]; };
template <typename R> __device__ __forceinline__ void racc_zero(RAcc<R> &a) {
    vdup(a.pr, 0);
    a.pi = a.pr;
#pragma unroll
    for (int k = 0; k < 3; ++k) a.gr[k] = a.gi[k] = a.pr;
}
template <typename R> __device__ __forceinline__ void racc_sum(RAcc<R> &a, const RAcc<R> &b) {
    a.pr = vadd(a.pr, b.pr);
    a.pi = vadd(a.pi, b.pi);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a.gr[k] = vadd(a.gr[k], b.gr[k]);
        a.gi[k] = vadd(a.gi[k], b.gi[k]);
    }
}

// The 4-point rule of a staged element at the lane's points, for the points
// with their bit in mask, added to the right-hand sides' sums.
template <typename T, int NR, bool TRI, bool VEL>
__device__ __forceinline__ void proj_far(const ProjElem<T, NR> &e, int nr, const typename ProjLane<T>::R (&D)[3],
                                         unsigned mask, typename ProjLane<T>::R wr, typename ProjLane<T>::R nwr,
                                         typename ProjLane<T>::R k2, typename ProjLane<T>::R m3,
                                         const ScConst<typename ProjLane<T>::R> &sc,
                                         RAcc<typename ProjLane<T>::R> (&acc)[NR]) {
    using R = typename ProjLane<T>::R;
    R dny, Tr, Ti, P0r, P0i, G0r[3], G0i[3];
    vdup(Tr, 0);
    Ti = P0r = P0i = Tr;
#pragma unroll
    for (int k = 0; k < 3; ++k) G0r[k] = G0i[k] = Tr;
    constexpr bool kFlat = TRI && std::is_same<T, float>::value;   // offsets from the centroid
    constexpr int kN = kFlat ? 12 : 18;
    if (TRI) {
        R c[3];   // the centroid (FP64: the rule's first point) - x
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if constexpr (kFlat) c[k] = D[k];
            else c[k] = vadd(D[k], e.v[6 + k]);
        }
        dny = vfma(c[2], e.v[kN + 2], vfma(c[0], e.v[kN], vmul(c[1], e.v[kN + 1])));
    }
    constexpr int kUnroll = std::is_same<T, float>::value ? 4 : 1;   // FP64: pipe bound, registers short
#pragma unroll kUnroll
    for (int g = 0; g < 4; ++g) {
        R d[3], w;
        if constexpr (kFlat) {
            const float2 s2 = c_far4d[g][0], t2 = c_far4d[g][1], w2 = c_far4d[g][2];
            const R ss = pk2(s2.x, s2.y), tt = pk2(t2.x, t2.y);
            w = pk2(w2.x, w2.y);
#pragma unroll
            for (int k = 0; k < 3; ++k) d[k] = vfma(tt, e.v[9 + k], vfma(ss, e.v[6 + k], D[k]));
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) d[k] = vadd(D[k], e.v[6 + 3 * g + k]);
            if constexpr (TRI) {
                w = c_far64[g][2];
            } else {
                dny = vfma(d[2], e.v[18 + 3 * g + 2], vfma(d[0], e.v[18 + 3 * g], vmul(d[1], e.v[18 + 3 * g + 1])));
                w = e.v[30 + g];
            }
        }
        const R r2 = vfma(d[2], d[2], vfma(d[0], d[0], vmul(d[1], d[1])));
        // points out of the mask: zero distance, before anything is formed from
        // it (such a point may lie on this rule's, or beyond phase_sincos)
        R r, sn, cs, u;
        if constexpr (std::is_same<T, float>::value) {
            float lo, hi;
            unpk2(r2, lo, hi);
            u = pk2((mask & 1u) ? rsqrt_approx(lo) : 0.f, (mask & 2u) ? rsqrt_approx(hi) : 0.f);
            r = vmul(r2, u);
        } else {
            u = rsqrt_nr(r2, &r);
            if (!mask) u = r = 0.0;
        }
        vsincos(sc, vmul(wr, r), sn, cs);
        const R A = vmul(u, u), B = vmul(wr, u), nB = vmul(nwr, u), p = vmul(w, u);
        const R Gr = vmul(p, cs), Gi = vmul(p, sn);
        const R hr = vfma(Gi, B, vmul(Gr, A)), hi = vfma(Gr, nB, vmul(Gi, A));   // G alpha
        const R Ad = vmul(A, dny);
        const R vr = vmul(Ad, vfma(m3, hr, vmul(k2, Gr))), vi = vmul(Ad, vfma(m3, hi, vmul(k2, Gi)));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            G0r[k] = vfma(vr, d[k], G0r[k]);
            G0i[k] = vfma(vi, d[k], G0i[k]);
        }
        if (TRI) {
            Tr = vadd(Tr, hr);
            Ti = vadd(Ti, hi);
        } else {
            P0r = vfma(dny, hr, P0r);   // -P0 until the end
            P0i = vfma(dny, hi, P0i);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                G0r[k] = vfma(hr, e.v[18 + 3 * g + k], G0r[k]);
                G0i[k] = vfma(hi, e.v[18 + 3 * g + k], G0i[k]);
            }
        }
        if (VEL) {
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                if (r >= nr) break;
                const R *V = e.V[r][g];
                acc[r].pr = vfma(V[0], Gr, vfma(V[2], Gi, acc[r].pr));
                acc[r].pi = vfma(V[0], Gi, vfma(V[1], Gr, acc[r].pi));
                const R zr = vfma(V[2], hi, vmul(V[0], hr)), zi = vfma(V[1], hr, vmul(V[0], hi));
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    acc[r].gr[k] = vfma(zr, d[k], acc[r].gr[k]);
                    acc[r].gi[k] = vfma(zi, d[k], acc[r].gi[k]);
                }
            }
        }
    }
    if (TRI) {
        P0r = vmul(dny, Tr);
        P0i = vmul(dny, Ti);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            G0r[k] = vfma(Tr, e.v[kN + k], G0r[k]);
            G0i[k] = vfma(Ti, e.v[kN + k], G0i[k]);
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (r >= nr) break;
        const R Wr = e.W[r][0], Wi = e.W[r][1], nWi = e.W[r][2], nWr = e.W[r][3];
        acc[r].pr = vfma(nWr, P0r, vfma(Wi, P0i, acc[r].pr));
        acc[r].pi = vfma(nWr, P0i, vfma(nWi, P0r, acc[r].pi));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            acc[r].gr[k] = vfma(Wr, G0r[k], vfma(nWi, G0i[k], acc[r].gr[k]));
            acc[r].gi[k] = vfma(Wr, G0i[k], vfma(Wi, G0r[k], acc[r].gi[k]));
        }
    }
}

// A not subdivided pair of a higher Gauss order, or of a phase beyond
// phase_sincos's range, by one lane.
template <typename T>
__device__ __noinline__ ProjAcc<T> proj_whole(const ProjSys *Sp, int kref, int j, int order, int p) {
    const ProjSys &S = *Sp;
    const DevMesh m = to_dev(S.m);
    const DevMesh mk = image_mesh(m, kref);
    const int n = m.n, nv = m.nvert[j];
    const bool iv = S.ivi[j] != 0;
    const double x[3] = {S.pts[3 * p], S.pts[3 * p + 1], S.pts[3 * p + 2]};
    cplx<T> ph, vl[4];
    proj_elem_data<T>((const double2 *)S.phi, (const double2 *)S.vel, (const float2 *)S.phi32,
                      (const float2 *)S.vel32, n, j, nv, iv, kref, image_negated(m, kref), ph, vl);
    ProjAcc<T> acc;
    acc.p = acc.g[0] = acc.g[1] = acc.g[2] = cmk(T(0), T(0));
    const T k = (T)S.f.k, wr = (T)S.f.wr;
    const int np = sub_npts(nv, order);
    if constexpr (std::is_same<T, double>::value) {
        Elem64 e;
        load_elem64(mk, j, e);
        for (int g = 0; g < np; ++g) {
            double s, t, w;
            sub_point(nv, order, g, 0.0, 0.0, 1.0, s, t, w);
            QPoint<double> q;
            map_point(e, s, t, x, w, q);
            proj_point(q, ph, vl, nv, iv, k, wr, acc);
        }
    } else {
        float xhi[3], xlo[3];
        for (int c = 0; c < 3; ++c) {
            xhi[c] = (float)x[c];
            xlo[c] = (float)(x[c] - (double)xhi[c]);
        }
        Elem32 e;
        load_elem32(mk, j, xhi, xlo, e);
        if (nv == 3 && !iv) {   // the unknown once per pair, the points' constants in the code
            float2 P = make_float2(0.f, 0.f), U[3] = {P, P, P}, Tn = P;
            const float dny = e.D[0] * e.n[0] + e.D[1] * e.n[1] + e.D[2] * e.n[2];
            if (order == 3) proj_tri_points<7, 4>(e, dny, k * k, wr, P, U, Tn);
            else proj_tri_points<13, 11>(e, dny, k * k, wr, P, U, Tn);
            acc.p = ph * cplx<float>{P.x, P.y};
            for (int q = 0; q < 3; ++q) acc.g[q] = ph * cplx<float>{fmaf(Tn.x, e.n[q], U[q].x), fmaf(Tn.y, e.n[q], U[q].y)};
            return acc;
        }
        for (int g = 0; g < np; ++g) {
            float s, t, w;
            sub_point_f(nv, order, g, 0.f, 0.f, 1.f, s, t, w);
            QPoint<float> q;
            map_point(e, s, t, w, q);
            proj_point(q, ph, vl, nv, iv, k, wr, acc);
        }
    }
    return acc;
}

// A subdivided pair, by the whole warp; the reduced sum on every lane.
template <typename T>
__device__ __noinline__ ProjAcc<T> proj_near(const ProjSys *Sp, int kref, int j, int p, WarpScratch *ws, int *err) {
    const ProjSys &S = *Sp;
    const DevMesh m = to_dev(S.m);
    const DevMesh mk = image_mesh(m, kref);
    const int n = m.n;
    const double x[3] = {S.pts[3 * p], S.pts[3 * p + 1], S.pts[3 * p + 2]};   // a uniform load
    float xhi[3], xlo[3];
    for (int c = 0; c < 3; ++c) {
        xhi[c] = (float)x[c];
        xlo[c] = (float)(x[c] - (double)xhi[c]);
    }
    Elem64 e;
    load_elem64(mk, j, e);
    Elem32 e32;   // float arithmetic, and the subdivision's fast decisions
    load_elem32(mk, j, xhi, xlo, e32);
    cplx<T> ph, vl[4];
    proj_elem_data<T>((const double2 *)S.phi, (const double2 *)S.vel, (const float2 *)S.phi32,
                      (const float2 *)S.vel32, n, j, e.nv, true, kref, image_negated(m, kref), ph, vl);
    ProjSink<T> sink;
    if constexpr (std::is_same<T, double>::value) { sink.e = &e; sink.x = x; }
    else sink.e = &e32;
    sink.phi = ph; sink.vel = vl; sink.ivi = S.ivi[j] != 0; sink.k = (T)S.f.k; sink.wr = (T)S.f.wr;
    sink.init();
    const int rc = warp_subdivide(e, m.area64[j], x, *ws, sink, &e32, m.isqa32[j]);
    if (rc != kDevOk) *err = rc;
    return sink.reduce();
}

__device__ __forceinline__ void racc_add(RAcc<double> &a, int, const ProjAcc<double> &b) {
    a.pr += b.p.re;
    a.pi += b.p.im;
    for (int k = 0; k < 3; ++k) { a.gr[k] += b.g[k].re; a.gi[k] += b.g[k].im; }
}
__device__ __forceinline__ void half_add(F2 &a, int h, float x) { a = vadd(a, h ? pk2(0.f, x) : pk2(x, 0.f)); }
__device__ __forceinline__ void racc_add(RAcc<F2> &a, int h, const ProjAcc<float> &b) {
    half_add(a.pr, h, b.p.re);
    half_add(a.pi, h, b.p.im);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        half_add(a.gr[k], h, b.g[k].re);
        half_add(a.gi[k], h, b.g[k].im);
    }
}

// acc[r] += b for the lane's point h, with every index known at compile time
// (a runtime index would put the sums in local memory)
template <typename T, int NR>
__device__ __forceinline__ void racc_at(RAcc<typename ProjLane<T>::R> (&acc)[NR], int r, int h, const ProjAcc<T> &b) {
#pragma unroll
    for (int q = 0; q < NR; ++q)
        if (q == r) racc_add(acc[q], h, b);
}

// NR = 1: the batch's systems, one after the other.  NR > 1: systems 0 .. nr - 1
// are right-hand sides of one matrix (same mesh, points and split).
template <typename T, int NR>
__global__ void __launch_bounds__(256, NR <= 2 ? 2 : 1) k_project_pts(const __grid_constant__ ProjBatch tb, int nr) {
    using R = typename ProjLane<T>::R;
    constexpr int P = ProjLane<T>::kP, kChunk = proj_chunk(NR);
    __shared__ WarpScratch ws_all[8];
    __shared__ ProjElem<T, NR> el[kChunk];
    static_assert(sizeof(ws_all) >= 256 * 8 * sizeof(R), "the warps' sums fit the subdivision scratch");
    const int sb = NR > 1 ? 0 : find_sys(tb.lp_off, tb.B, blockIdx.x);
    const ProjSys &S = tb.sys[sb];
    const DevMesh m = to_dev(S.m);
    const DevFreq &f = S.f;
    const int lane = threadIdx.x, w = threadIdx.y, tid = w * 32 + lane, n = m.n, npts = S.npts;
    const int nsl = S.nslice, pgb = S.pgb, ewb = 8 / pgb;
    const int item = blockIdx.x - tb.lp_off[sb];
    const int sl = item % nsl, gb = item / nsl;
    const int ew = w / pgb;                                   // element part
    const int p0 = (gb * pgb + w % pgb) * 32 * P + lane;     // the lane's points: p0, p0 + 32
    const int j0 = sl * S.per, j1 = min(n, j0 + S.per);
    const bool group = p0 - lane < npts;                      // the warp has points
    // The points, as float hi/lo pairs for the distances of the quadrature
    // decision and (float) the arithmetic; made opaque to the compiler: under
    // register pressure it otherwise recomputes them from the FP64 values,
    // and GB300 issues those conversions on its narrow FP64 pipe.  Idle
    // points repeat the group's first.
    float xh[P][3], xl[P][3];
    R X[6];   // float: packed high and low parts, negated; FP64: the point
#pragma unroll
    for (int h = 0; h < P; ++h) {
        const int p = p0 + 32 * h < npts ? p0 + 32 * h : (group ? p0 - lane : 0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double xv = S.pts[3 * p + c];
            xh[h][c] = (float)xv;
            xl[h][c] = (float)(xv - (double)xh[h][c]);
            asm volatile("" : "+f"(xh[h][c]), "+f"(xl[h][c]));
            if constexpr (P == 1) X[c] = xv;
        }
    }
    if constexpr (P == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            X[c] = pk2(-xh[0][c], -xh[P - 1][c]);
            X[3 + c] = pk2(-xl[0][c], -xl[P - 1][c]);
        }
    }
    T k = (T)f.k, wrs = (T)f.wr;
    if constexpr (P == 2) asm volatile("" : "+f"(k), "+f"(wrs));
    R wr, nwr, k2, m3;
    vdup(wr, wrs);
    vdup(nwr, -wrs);
    vdup(k2, k * k);
    m3 = opaque2(T(-3));
    ScConst<R> sc;
    sc.init();
    // sums of up to kProjRun elements; of those before them, in local memory,
    // which the compiler is to leave there (in registers they push the loop's
    // own values out)
    RAcc<R> acc[NR], sum_s[NR], *sum = sum_s;
    asm volatile("" : "+l"(sum)::"memory");
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        racc_zero(acc[r]);
        racc_zero(sum[r]);
    }
    auto flush = [&]() {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            racc_sum(sum[r], acc[r]);
            racc_zero(acc[r]);
        }
    };
    if (NR == 1) nr = 1;
    int reach = 0;   // FP64: phases of elements within it fit phase_sincos
    if constexpr (P == 1) {
        reach = phase_reach(wrs);
        if (max_hi(X[0], X[1], X[2]) >= reach) reach = 0;
    }
    int err = kDevOk;
    for (int kref = 0; kref < m.sym.nref; ++kref) {
        const DevMesh mk = image_mesh(m, kref);
        const bool neg = image_negated(m, kref);
        for (int base = j0; base < j1; base += kChunk) {
            const int cnt = min(kChunk, j1 - base);
            __syncthreads();   // the previous chunk has been read
            if (tid < 4 * kChunk && (tid >> 2) < cnt)
                proj_stage<T, NR>(&S, nr, m, mk, kref, neg, base + (tid >> 2), tid & 3, el[tid >> 2]);
            __syncthreads();
            if (!group) continue;
            for (int q = ew; q < cnt; q += ewb) {
                const ProjElem<T, NR> &e = el[q];
                const bool tri = e.nv == 3;
                // distances and quadrature orders of the lane's points
                R D[3];
                float q2[P];
                if constexpr (P == 2) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) D[c] = vadd(vadd(e.v[c], X[c]), vadd(e.v[3 + c], X[3 + c]));   // X holds -x
                    const F2 d2 = vfma(D[2], D[2], vfma(D[0], D[0], vmul(D[1], D[1])));
                    unpk2(vmul(d2, pk2(e.isq2, e.isq2)), q2[0], q2[P - 1]);
                } else {
                    float d[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        D[c] = -X[c];
                        d[c] = (e.hi[c] - xh[0][c]) + (e.lo[c] - xl[0][c]);
                    }
                    q2[0] = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) * e.isq2;
                }
                unsigned far = 0;
                int ord[P];   // 0: subdivided
#pragma unroll
                for (int h = 0; h < P; ++h) {
                    bool near = false;
                    ord[h] = 2;
                    if (q2[h] <= c_quad.far2_sq) {
                        if (!classify_fast(sqrtf(q2[h]), near, ord[h])) {
                            const int p = p0 + 32 * h < npts ? p0 + 32 * h : p0 - lane;
                            const double xp[3] = {S.pts[3 * p], S.pts[3 * p + 1], S.pts[3 * p + 2]};
                            const double rd = ratio0_exact(mk, base + q, xp);
                            near = rd < kTolf;
                            if (!near) ord[h] = gauss_order(rd);
                        }
                        if (near) ord[h] = 0;
                    }
                    if (ord[h] == 2 && (P == 2 || e.far < reach)) far |= 1u << h;
                }
                if (__any_sync(0xffffffffu, far != 0)) {
                    if (tri) {
                        if (!e.iv) proj_far<T, NR, true, false>(e, nr, D, far, wr, nwr, k2, m3, sc, acc);
                        else proj_far<T, NR, true, true>(e, nr, D, far, wr, nwr, k2, m3, sc, acc);
                    } else {
                        if (!e.iv) proj_far<T, NR, false, false>(e, nr, D, far, wr, nwr, k2, m3, sc, acc);
                        else proj_far<T, NR, false, true>(e, nr, D, far, wr, nwr, k2, m3, sc, acc);
                    }
                }
                if (__all_sync(0xffffffffu, far == (1u << P) - 1u)) continue;
#pragma unroll
                for (int h = 0; h < P; ++h) {
                    const bool pv = p0 + 32 * h < npts;
                    if (pv && ord[h] != 0 && !((far >> h) & 1u))
#pragma unroll 1
                        for (int r = 0; r < nr; ++r)
                            racc_at<T, NR>(acc, r, h, proj_whole<T>(&tb.sys[sb + r], kref, base + q, ord[h], p0 + 32 * h));
                    unsigned todo = __ballot_sync(0xffffffffu, pv && ord[h] == 0);
                    while (todo) {
                        const int L = __ffs(todo) - 1;
                        todo &= todo - 1;
#pragma unroll 1
                        for (int r = 0; r < nr; ++r) {
                            const ProjAcc<T> z = proj_near<T>(&tb.sys[sb + r], kref, base + q, p0 - lane + 32 * h + L,
                                                              &ws_all[w], &err);
                            if (lane == L) racc_at<T, NR>(acc, r, h, z);
                        }
                    }
                }
            }
            if ((base + kChunk - j0) % kProjRun == 0) flush();
        }
    }
    flush();
    if (err != kDevOk && lane == 0) atomicMax(S.status, err);
    // the element parts of a point group meet in shared memory, in order
    R *red = reinterpret_cast<R *>(ws_all);   // [warp][8][lane]
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (r >= nr) break;
        RAcc<R> a = sum[r];
        if (ewb > 1) {
            __syncthreads();
            if (ew > 0) {
                R *o = red + (size_t)w * 8 * 32 + lane;
                o[0] = a.pr;
                o[32] = a.pi;
#pragma unroll
                for (int c = 0; c < 3; ++c) { o[(2 + 2 * c) * 32] = a.gr[c]; o[(3 + 2 * c) * 32] = a.gi[c]; }
            }
            __syncthreads();
            for (int q = 1; q < ewb && ew == 0; ++q) {
                const R *o = red + (size_t)(w + q * pgb) * 8 * 32 + lane;
                a.pr = vadd(a.pr, o[0]);
                a.pi = vadd(a.pi, o[32]);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    a.gr[c] = vadd(a.gr[c], o[(2 + 2 * c) * 32]);
                    a.gi[c] = vadd(a.gi[c], o[(3 + 2 * c) * 32]);
                }
            }
        }
        if (ew > 0 || !group) continue;
        float4 *part = tb.sys[sb + r].part;
        if constexpr (P == 2) {
            float v[2][8];
            unpk2(a.pr, v[0][0], v[1][0]);
            unpk2(a.pi, v[0][1], v[1][1]);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                unpk2(a.gr[c], v[0][2 + 2 * c], v[1][2 + 2 * c]);
                unpk2(a.gi[c], v[0][3 + 2 * c], v[1][3 + 2 * c]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 *out = part + 2 * ((size_t)sl * S.pstride + p0 + 32 * h);
                out[0] = make_float4(v[h][0], v[h][1], v[h][2], v[h][3]);
                out[1] = make_float4(v[h][4], v[h][5], v[h][6], v[h][7]);
            }
        } else {
            double2 *out = reinterpret_cast<double2 *>(part) + 4 * ((size_t)sl * S.pstride + p0);
            out[0] = make_double2(a.pr, a.pi);
#pragma unroll
            for (int c = 0; c < 3; ++c) out[1 + c] = make_double2(a.gr[c], a.gi[c]);
        }
    }
}

// Sums of the slices (FP64) and the finish of a point (tau factor, incident
// field).  A block of 256 threads takes PT points, 256 / PT threads each adding
// every (256 / PT)th slice; the threads' sums are added in order by the thread
// that finishes the point.  The additions and conversions run on an SM's
// narrow FP64 pipe, so few points (up to kSumSpread) go 4 to a block to reach
// more SMs: 64 points x 320 slices on 2 SMs took 56 us, on 16 they take 15.
// (4 blocks on each of 152 SMs, as a number for the reason given at kProjSlots)
constexpr int kSumSpread = 2432;
__host__ __device__ inline int sum_points(int npts) { return npts <= kSumSpread ? 4 : 32; }

template <typename T>
__global__ void __launch_bounds__(256) k_project_sum(const __grid_constant__ ProjBatch tb) {
    __shared__ double red[256][8];   // [slice thread][point][component]
    const int sb = find_sys(tb.ps_off, tb.B, blockIdx.x);
    const ProjSys &S = tb.sys[sb];
    const int PT = sum_points(S.npts), per = 256 / PT;
    const int pi = threadIdx.x % PT, w = threadIdx.x / PT;
    const int p = (blockIdx.x - tb.ps_off[sb]) * PT + pi;
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = 0.0;
    if (p < S.npts) {
#pragma unroll 4
        for (int sl = w; sl < S.nslice; sl += per) {
            if constexpr (std::is_same<T, float>::value) {
                const float4 *in = S.part + 2 * ((size_t)sl * S.pstride + p);
                const float4 u = in[0], v = in[1];
                a[0] += (double)u.x; a[1] += (double)u.y; a[2] += (double)u.z; a[3] += (double)u.w;
                a[4] += (double)v.x; a[5] += (double)v.y; a[6] += (double)v.z; a[7] += (double)v.w;
            } else {
                const double2 *in = reinterpret_cast<const double2 *>(S.part) + 4 * ((size_t)sl * S.pstride + p);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double2 u = in[q];
                    a[2 * q] += u.x;
                    a[2 * q + 1] += u.y;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) red[threadIdx.x][q] = a[q];
    __syncthreads();
    // 8 PT threads: component c of point e
    if (threadIdx.x < 8 * PT) {
        const int e = threadIdx.x >> 3, c = threadIdx.x & 7, top = min(per, S.nslice);
        double t = red[e][c];
        for (int u = 1; u < top; ++u) t += red[u * PT + e][c];
        red[e][c] = t;
    }
    __syncthreads();
    if (w != 0 || p >= S.npts) return;
    const double *t = red[pi];
    cplx<double> sg[3] = {{t[2], t[3]}, {t[4], t[5]}, {t[6], t[7]}};
    const DevMesh m = to_dev(S.m);
    const double x64[3] = {S.pts[3 * p], S.pts[3 * p + 1], S.pts[3 * p + 2]};
    project_finish(m, S.f, x64, p, {t[0], t[1]}, sg, (double2 *)S.pot, (double2 *)S.grad);
}

// ---------------------------------------------------------------- tables
// Published Gauss-Legendre and triangle rules at the precision NumCalc
// tabulates them (NC_IntegrationConstants.h:26-49,3729-3865).
const double kGLPos[7][3][2] = {
    {{0, 0}},
    {{0.0, 2.0}},
    {{0.577350269189626, 1.0}},
    {{0.0, 0.888888888888889}, {0.774596669241483, 0.555555555555556}},
    {{0.339981043584856, 0.652145154862546}, {0.861136311594053, 0.347854845137454}},
    {{0.0, 0.568888888888889}, {0.538469310105683, 0.478628670499366}, {0.906179845938664, 0.236926885056189}},
    {{0.238619186083197, 0.467913934572691}, {0.661209386466265, 0.360761573048139}, {0.932469514203152, 0.171324492379170}},
};

const double kTri[24][3] = {
    // Strang-Fix 4 points
    {1.0 / 3.0, 1.0 / 3.0, -27.0 / 96.0}, {0.2, 0.2, 25.0 / 96.0}, {0.6, 0.2, 25.0 / 96.0}, {0.2, 0.6, 25.0 / 96.0},
    // Radon 7 points
    {0.1012865073235, 0.1012865073235, 0.1259391805448 / 2.0},
    {0.7974269853531, 0.1012865073235, 0.1259391805448 / 2.0},
    {0.1012865073235, 0.7974269853531, 0.1259391805448 / 2.0},
    {0.4701420641051, 0.0597158717898, 0.1323941527885 / 2.0},
    {0.4701420641051, 0.4701420641051, 0.1323941527885 / 2.0},
    {0.0597158717898, 0.4701420641051, 0.1323941527885 / 2.0},
    {0.3333333333333, 0.3333333333333, 0.225 / 2.0},
    // 13 points, degree 7
    {0.0651301029022, 0.0651301029022, 0.0533472356088 / 2.0},
    {0.8697397941956, 0.0651301029022, 0.0533472356088 / 2.0},
    {0.0651301029022, 0.8697397941956, 0.0533472356088 / 2.0},
    {0.3128654960049, 0.0486903154253, 0.0771137608903 / 2.0},
    {0.6384441885698, 0.3128654960049, 0.0771137608903 / 2.0},
    {0.0486903154253, 0.6384441885698, 0.0771137608903 / 2.0},
    {0.6384441885698, 0.0486903154253, 0.0771137608903 / 2.0},
    {0.3128654960049, 0.6384441885698, 0.0771137608903 / 2.0},
    {0.0486903154253, 0.3128654960049, 0.0771137608903 / 2.0},
    {0.2603459660790, 0.2603459660790, 0.1756152574332 / 2.0},
    {0.4793080678419, 0.2603459660790, 0.1756152574332 / 2.0},
    {0.2603459660790, 0.4793080678419, 0.1756152574332 / 2.0},
    {0.3333333333333, 0.3333333333333, -0.1495700444677 / 2.0},
};

// Host copy of NumCalc's order test (NC_Macros.h:44-50) for the thresholds.
bool order_ok_host(int m, double ratdis) {
    const double disfac = 0.5 / ratdis;
    double eg = 32.0, eh = 64.0 * (2.0 * (double)m + 1.0), ee = 128.0 * ((double)m + 1.0) * (2.0 * (double)m + 1.0);
    for (int q = 0; q < 2 * m + 1; ++q) eg *= disfac;
    for (int q = 0; q < 2 * m + 2; ++q) eh *= disfac;
    for (int q = 0; q < 2 * m + 3; ++q) ee *= disfac;
    return ee < 0.001 && eh < 0.001 && eg < 0.001;
}

double order_threshold(int m) {
    // bisection over the ordered bit patterns of positive doubles
    double lo = 0.5, hi = 1000.0;  // order_ok false at lo, true at hi
    uint64_t a, b;
    memcpy(&a, &lo, 8);
    memcpy(&b, &hi, 8);
    while (b - a > 1) {
        uint64_t c = a + (b - a) / 2;
        double mid;
        memcpy(&mid, &c, 8);
        if (order_ok_host(m, mid)) b = c; else a = c;
    }
    double t;
    memcpy(&t, &b, 8);
    return t;
}

}  // namespace

cudaError_t init_device_tables() {
    QuadTables q;
    memset(&q, 0, sizeof(q));
    float trif[24][3], glxf[7][6], glwf[7][6];
    for (int i = 0; i < 24; ++i)
        for (int k = 0; k < 3; ++k) { q.tri[i][k] = kTri[i][k]; trif[i][k] = (float)kTri[i][k]; }
    for (int n = 1; n <= 6; ++n) {
        const int h = n / 2;
        double x[6] = {0}, w[6] = {0};
        if (n % 2) {
            x[h] = kGLPos[n][0][0]; w[h] = kGLPos[n][0][1];
            for (int i = 1; i <= h; ++i) {
                x[h + i] = kGLPos[n][i][0]; x[h - i] = -kGLPos[n][i][0];
                w[h + i] = w[h - i] = kGLPos[n][i][1];
            }
        } else {
            for (int i = 0; i < h; ++i) {
                x[h + i] = kGLPos[n][i][0]; x[h - 1 - i] = -kGLPos[n][i][0];
                w[h + i] = w[h - 1 - i] = kGLPos[n][i][1];
            }
        }
        for (int i = 0; i < 6; ++i) {
            q.glx[n][i] = x[i]; q.glw[n][i] = w[i];
            glxf[n][i] = (float)x[i]; glwf[n][i] = (float)w[i];
        }
    }
    for (int i = 0; i < 6; ++i) { glxf[0][i] = glwf[0][i] = 0.f; }
    for (int m = 2; m <= 5; ++m) {
        q.order_thr[m] = order_threshold(m);
        q.order_thrf[m] = (float)q.order_thr[m];
    }
    q.far2_sq = (float)((q.order_thr[2] * (1.0 + 3e-5)) * (q.order_thr[2] * (1.0 + 3e-5)));
    cudaError_t e = cudaMemcpyToSymbol(c_quad, &q, sizeof(q));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_trif, trif, sizeof(trif));
    float far4[4][2];
    for (int g = 0; g < 4; ++g) {
        far4[g][0] = trif[g][0] - (1.0f / 3.0f);
        far4[g][1] = trif[g][1] - (1.0f / 3.0f);
    }
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_far4, far4, sizeof(far4));
    float2 far4d[4][3];
    for (int g = 0; g < 4; ++g) {
        far4d[g][0] = make_float2(far4[g][0], far4[g][0]);
        far4d[g][1] = make_float2(far4[g][1], far4[g][1]);
        far4d[g][2] = make_float2(trif[g][2], trif[g][2]);
    }
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_far4d, far4d, sizeof(far4d));
    double far64[24][4];
    for (int g = 0; g < 24; ++g) {
        far64[g][0] = kTri[g][0] - 1.0 / 3.0;
        far64[g][1] = kTri[g][1] - 1.0 / 3.0;
        far64[g][2] = kTri[g][2];
        far64[g][3] = 0.0;
    }
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_far64, far64, sizeof(far64));
    if (e == cudaSuccess) e = init_sincos_table();
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_glxf, glxf, sizeof(glxf));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_glwf, glwf, sizeof(glwf));
    return e;
}

cudaError_t launch_image_tables(const DevMeshView &m, const ImageTables &out, cudaStream_t st) {
    const long long total = (long long)(m.sym.nref - 1) * m.n;
    if (total <= 0) return cudaSuccess;
    count_launches(1);
    k_image_tables<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(m, out);
    return cudaGetLastError();
}

size_t near_list_scratch_bytes(int n, int nref) {
    const size_t nb = (size_t)(n + 31) / 32;
    return nb * (size_t)nref * sizeof(float4) + nb * sizeof(float);
}

cudaError_t launch_near_list(const DevMeshView &m, void *scratch, int2 *list, unsigned long long cap,
                             unsigned long long *count, cudaStream_t st) {
    const int nb = (m.n + 31) / 32;
    float4 *sph = (float4 *)scratch;
    float *bsq = (float *)(sph + (size_t)nb * m.sym.nref);
    dim3 block(32, 8);
    count_launches(2);
    k_block_spheres<<<(nb * m.sym.nref + 7) / 8, block, 0, st>>>(m, sph, bsq);
    k_near_list<<<(m.n + 7) / 8, block, 0, st>>>(m, sph, bsq, list, count, cap);
    return cudaGetLastError();
}

void asm_batch_finish(AsmBatch &t) {
    t.far_off[0] = t.near_off[0] = t.rhs_off[0] = 0;
    t.img = 0;
    for (int b = 0; b < t.B; ++b) {
        if (t.sys[b].m.sym.nref > 1) t.img = 1;
        const int n = t.sys[b].m.n;
        const int nt = (n + 31) / 32;
        t.far_off[b + 1] = t.far_off[b] + nt * ceil_div(n, far_rows(n));
        t.near_off[b + 1] = t.near_off[b] + (int)t.sys[b].n_near;
        const int rows = t.sys[b].f.n_bc_cols > 0 ? 8 : kRhsRows;   // k_rhs: a warp or a thread per row
        t.rhs_off[b + 1] = t.rhs_off[b] + (n + rows - 1) / rows;
    }
}

// Work split of the projection, from the system's own sizes only (a system's
// result does not depend on the rest of its batch).  Point groups per block:
// the most, up to 8, that pad the groups by less than a fourteenth (a wide
// block stages its elements for more points; 28 groups of 1730 points go in
// fours).  Slices: of at most kProjSlice elements (the length of an FP32 sum),
// more where that leaves SMs idle, down to kProjStep elements; the number of
// blocks is then rounded down to whole rounds of the resident ones (2 per SM
// of 152; 26 slices of 24 blocks ran a third round for 16 of them: 11950 points
// on 20480 elements 2.43 ms, with whole rounds 2.15), and the scratch may hold
// fewer.  Where it leaves less than two rounds of blocks, as for many points on a
// small mesh, blocks take fewer groups, whose elements their warps then share:
// points near the surface, with their subdivided pairs and higher orders, often
// follow one another and would hold up a few blocks (2000 triangles, 10550
// points of which 500 are near: 4.8 -> 0.73 ms; 4000 points along the surface
// of 5120 triangles 1.6 -> 0.63 ms, with one round 0.84).  It costs up to 8 % where all
// points are far (1730 points on 5120 triangles 166 -> 180 us).
void proj_batch_finish(ProjBatch &t, int prec) {
    t.fld_off[0] = t.pt_off[0] = t.lp_off[0] = t.ps_off[0] = 0;
    const int gpts = 32 * (prec == 0 ? ProjLane<double>::kP : ProjLane<float>::kP);
    const int part = prec == 0 ? ProjLane<double>::kPart : ProjLane<float>::kPart;
    for (int b = 0; b < t.B; ++b) {
        ProjSys &S = t.sys[b];
        t.fld_off[b + 1] = t.fld_off[b] + (S.m.n + 255) / 256;
        t.pt_off[b + 1] = t.pt_off[b] + (S.npts + 7) / 8;
        const int G = ceil_div(S.npts, gpts);
        S.pgb = 8;
        while (S.pgb > 1 && 14 * (ceil_div(G, S.pgb) * S.pgb - G) >= G) S.pgb /= 2;
        int GB = G > 0 ? ceil_div(G, S.pgb) : 1;
        S.pstride = G * gpts;
        const long long fit = G > 0 && S.part ? S.part_cap / ((long long)part * S.pstride) : 0;
        const long long least = ceil_div(S.m.n, kProjSlice), most = ceil_div(S.m.n, kProjStep);
        auto slices = [&]() {
            const long long nsl = std::max(least, std::min<long long>(most, ceil_div(4 * kProjSlots, GB)));
            return std::min(nsl, fit);
        };
        long long nsl = slices();
        while (S.pgb > 1 && nsl * GB < 2 * kProjSlots) {
            S.pgb /= 2;
            GB = ceil_div(G, S.pgb);
            nsl = slices();
        }
        const long long rounds = nsl * GB / kProjSlots;
        if (rounds > 0 && rounds <= 4) nsl = std::max(std::min(least, fit), rounds * kProjSlots / GB);
        S.per = nsl > 0 ? ceil_div(S.m.n, nsl) : 0;
        S.nslice = nsl > 0 ? ceil_div(S.m.n, S.per) : 0;
        t.lp_off[b + 1] = t.lp_off[b] + (G > 0 ? GB * S.nslice : 0);
        t.ps_off[b + 1] = t.ps_off[b] + ceil_div(S.npts, sum_points(S.npts));
    }
}

namespace {
int g_sms = 0;
int sm_count() {
    if (g_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 1;
    }
    return g_sms;
}
}  // namespace

cudaError_t launch_assemble(const AsmBatch &t, int prec, unsigned *ctr, cudaStream_t st, AsmShape shape) {
    if (t.B <= 0) return cudaSuccess;
    dim3 block(32, 8);
    const int far_items = t.far_off[t.B], near_items = t.near_off[t.B];
    // persistent grids: far_per_sm resident blocks of k_far per SM (launch
    // bounds allow kFarPerSm), near_per_sm of k_near, twice that for complex64 (its
    // launch bounds allow 2 and 4)
    const int fps = std::max(1, std::min(shape.far_per_sm, kFarPerSm));
    const int nps = std::max(1, std::min(shape.near_per_sm, 2)) * (prec == 0 ? 1 : 2);
    const int gfar = std::max(1, std::min((far_items + 7) / 8, fps * sm_count()));
    const int gnear = std::max(1, std::min((near_items + 7) / 8, nps * sm_count()));
    // Systems that fill the GPU on their own take one single-system launch
    // each: the single-system kernel keeps the table in constant operands
    // (fewer registers, no spills), which beat one launch over the batch.
    bool split = t.B > 1;
    for (int b = 0; b < t.B && split; ++b)
        if (t.far_off[b + 1] - t.far_off[b] < 8 * fps * sm_count()) split = false;
    std::unique_ptr<AsmBatch> one_sys;
    if (split) one_sys.reset(new AsmBatch());
    count_launches((split ? t.B : 1) + (near_items ? 1 : 0));
    auto far = [&](const AsmBatch &a, int grid) {
        const bool one = a.B == 1;
        if (prec == 0) {
            if (a.img) {
                if (one) k_far<double, true, true><<<grid, block, 0, st>>>(a);
                else k_far<double, false, true><<<grid, block, 0, st>>>(a);
            } else {
                if (one) k_far<double, true, false><<<grid, block, 0, st>>>(a);
                else k_far<double, false, false><<<grid, block, 0, st>>>(a);
            }
        } else {
            if (a.img) {
                if (one) k_far<float, true, true><<<grid, block, 0, st>>>(a);
                else k_far<float, false, true><<<grid, block, 0, st>>>(a);
            } else {
                if (one) k_far<float, true, false><<<grid, block, 0, st>>>(a);
                else k_far<float, false, false><<<grid, block, 0, st>>>(a);
            }
        }
    };
    if (split) {
        for (int b = 0; b < t.B; ++b) {
            one_sys->B = 1;
            one_sys->sys[0] = t.sys[b];
            asm_batch_finish(*one_sys);
            far(*one_sys, std::max(1, std::min((one_sys->far_off[1] + 7) / 8, fps * sm_count())));
        }
    } else {
        far(t, gfar);
    }
    if (near_items) {
        if (prec == 0) k_near<double><<<gnear, block, 0, st>>>(t, ctr);
        else k_near<float><<<gnear, block, 0, st>>>(t, ctr);
    }
    return cudaGetLastError();
}

cudaError_t launch_rhs(const AsmBatch &t, cudaStream_t st) {
    if (t.B <= 0) return cudaSuccess;
    dim3 block(32, 8);
    count_launches(1);
    k_rhs<<<t.rhs_off[t.B], block, 0, st>>>(t);
    return cudaGetLastError();
}

cudaError_t launch_fields(const ProjBatch &t, cudaStream_t st) {
    if (t.B <= 0 || t.fld_off[t.B] == 0) return cudaSuccess;
    count_launches(1);
    k_fields<<<t.fld_off[t.B], 256, 0, st>>>(t);
    return cudaGetLastError();
}

namespace {
// lanes = points (NR right-hand sides at a time), then the slice sums
template <typename T, int NR>
void project_sliced(const ProjBatch &t, cudaStream_t st) {
    k_project_pts<T, NR><<<NR > 1 ? t.lp_off[1] : t.lp_off[t.B], dim3(32, 8), 0, st>>>(t, t.B);
    k_project_sum<T><<<t.ps_off[t.B], 256, 0, st>>>(t);
    count_launches(2);
}
}  // namespace

cudaError_t launch_project_multi(const ProjBatch &t, cudaStream_t st) {
    // the right-hand sides of one solver: same mesh, points and split
    bool shared = t.B >= 2 && t.B <= 8 && t.sys[0].nslice > 0;
    for (int b = 1; b < t.B && shared; ++b)
        shared = t.sys[b].npts == t.sys[0].npts && t.sys[b].pts == t.sys[0].pts &&
                 t.sys[b].nslice == t.sys[0].nslice && t.sys[b].per == t.sys[0].per && t.sys[b].m.n == t.sys[0].m.n;
    if (!shared) return launch_project(t, 1, st);
    if (t.sys[0].npts == 0) return cudaSuccess;
    if (t.B <= 2) project_sliced<float, 2>(t, st);
    else if (t.B <= 4) project_sliced<float, 4>(t, st);
    else project_sliced<float, 8>(t, st);
    return cudaGetLastError();
}

cudaError_t launch_project(const ProjBatch &t, int prec, cudaStream_t st) {
    if (t.B <= 0 || t.pt_off[t.B] == 0) return cudaSuccess;
    bool sliced = true;
    for (int b = 0; b < t.B; ++b)
        if (t.sys[b].npts > 0 && t.sys[b].nslice == 0) sliced = false;   // scratch too short
    if (!sliced) {
        count_launches(1);
        if (prec == 0) k_project<double><<<t.pt_off[t.B], dim3(32, 8), 0, st>>>(t);
        else k_project<float><<<t.pt_off[t.B], dim3(32, 8), 0, st>>>(t);
    } else if (prec == 0) {
        project_sliced<double, 1>(t, st);
    } else {
        project_sliced<float, 1>(t, st);
    }
    return cudaGetLastError();
}

}  // namespace bem
