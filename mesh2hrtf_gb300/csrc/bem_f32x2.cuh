// bem_f32x2.cuh - two floats per register pair.
//
// Packed FP32 arithmetic (PTX fma/mul/add.rn.f32x2): one instruction, two
// IEEE operations.  The FMA pipe does no more of them per cycle, but the
// kernels that are bound by instruction issue need half the slots.  Each half
// rounds exactly as the scalar instruction.
#pragma once

#include <cuda_runtime.h>

namespace bem {

struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 pk2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpk2(F2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// A packed constant kept in registers: as an immediate the compiler forms it
// with two moves at every use.
__device__ __forceinline__ F2 opaque2(float x) {
    F2 r = pk2(x, x);
    asm volatile("" : "+l"(r.v));
    return r;
}
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double opaque2(double x) { return x; }

}  // namespace bem
