// rift_pair.cuh -- FP32 arithmetic on one cell (float) or on two (P2), under the
// same names, so that the reconstruction and the flux (rift_device.cuh) are
// written once and give the same bits either way: every sum, product and fma
// is an instruction of its own (no contraction left to the compiler).
//
// On pairs, sums, products and fmas are the packed instructions (one issue
// slot for two operations; they run on one of the two FMA pipes, two cycles
// each); minima, maxima, reciprocals and square roots stay scalar.
#pragma once
#include <cstdint>

namespace rift {

struct P2 {  // two FP32 values in a register pair
    unsigned long long v;
};

__device__ __forceinline__ P2 pack2(float x, float y) {
    P2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ P2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ float lo(P2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(P2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ P2 vadd(P2 a, P2 b) {
    P2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 vsub(P2 a, P2 b) {
    P2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 vmul(P2 a, P2 b) {
    P2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 vfma(P2 a, P2 b, P2 c) {
    P2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// a + b, a - b where an operand is a product: the assembler contracts a packed
// product and sum into one fma (in some kernels and not in others), scalar ones
// with a rounding mode it leaves alone.
__device__ __forceinline__ float vaddOfMul(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsubOfMul(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ P2 vaddOfMul(P2 a, P2 b) {
    return pack2(__fadd_rn(lo(a), lo(b)), __fadd_rn(hi(a), hi(b)));
}
__device__ __forceinline__ P2 vsubOfMul(P2 a, P2 b) {
    return pack2(__fsub_rn(lo(a), lo(b)), __fsub_rn(hi(a), hi(b)));
}
// c - a b
__device__ __forceinline__ float vfnma(float a, float b, float c) { return __fmaf_rn(-a, b, c); }
__device__ __forceinline__ P2 vfnma(P2 a, P2 b, P2 c) {
    return pack2(vfnma(lo(a), lo(b), lo(c)), vfnma(hi(a), hi(b), hi(c)));
}
// a constant in every lane of V
template <class V>
__device__ __forceinline__ V splat(float x);
template <>
__device__ __forceinline__ float splat<float>(float x) { return x; }
template <>
__device__ __forceinline__ P2 splat<P2>(float x) { return both(x); }

__device__ __forceinline__ float vmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float vmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ P2 vmax(P2 a, P2 b) { return pack2(fmaxf(lo(a), lo(b)), fmaxf(hi(a), hi(b))); }
__device__ __forceinline__ P2 vmin(P2 a, P2 b) { return pack2(fminf(lo(a), lo(b)), fminf(hi(a), hi(b))); }
__device__ __forceinline__ P2 vmax(P2 a, float b) { return pack2(fmaxf(lo(a), b), fmaxf(hi(a), b)); }

// maximum and minimum that are NaN when an argument is (the ones above leave a
// NaN argument out)
__device__ __forceinline__ float vmaxNan(float a, float b) {
    float r;
    asm("max.ftz.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float vminNan(float a, float b) {
    float r;
    asm("min.ftz.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ P2 vmaxNan(P2 a, P2 b) {
    return pack2(vmaxNan(lo(a), lo(b)), vmaxNan(hi(a), hi(b)));
}
__device__ __forceinline__ P2 vminNan(P2 a, P2 b) {
    return pack2(vminNan(lo(a), lo(b)), vminNan(hi(a), hi(b)));
}

// max(a, b, 0): a NaN argument is left out
__device__ __forceinline__ float vmaxz(float a, float b) {
    float r;
    asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(0.f));
    return r;
}
__device__ __forceinline__ P2 vmaxz(P2 a, P2 b) { return pack2(vmaxz(lo(a), lo(b)), vmaxz(hi(a), hi(b))); }

// min(|a|, |b|)
__device__ __forceinline__ float minAbs(float a, float b) { return fminf(fabsf(a), fabsf(b)); }
__device__ __forceinline__ P2 minAbs(P2 a, P2 b) { return pack2(minAbs(lo(a), lo(b)), minAbs(hi(a), hi(b))); }
__device__ __forceinline__ float vrcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ P2 vrcp(P2 a) { return pack2(vrcp(lo(a)), vrcp(hi(a))); }
__device__ __forceinline__ float vsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ P2 vsqrt(P2 a) { return pack2(sqrtf(lo(a)), sqrtf(hi(a))); }

}  // namespace rift
