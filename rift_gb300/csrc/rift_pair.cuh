// rift_pair.cuh -- the reconstruction and the central-upwind flux of
// rift_device.cuh on two cells at a time.
//
// The flux passes are bound by instruction issue, not by a pipe, so pairs of
// cells go through the packed FP32 instructions (fma / mul / add .f32x2: one
// issue slot for two operations); minima, maxima, reciprocals and square
// roots stay scalar.  Three rewrites take instructions out without changing
// what is computed beyond the rounding of a sum:
//   - the wet/dry correction of Construct (grid.cu:91-116).  The two face
//     depths of a cell add up to hBar = 2h - eP - eM, so "if (hP < 0) hP = 0,
//     hM = hBar; if (hM < 0) hM = 0, hP = hBar" is
//     hP' = min(max(hP, 0), hBar), hM' = max(min(hM, hBar), 0);
//   - F(U) is zero where the face depth is not positive: formed from the
//     depth clamped at 0 instead of three selects;
//   - a dry face (a+ = a- = 0) has zero fluxes and zero products, so the
//     division takes 1 / max(d, tiny) instead of a branch.
// The one-sided speed a- enters as its magnitude, which removes the
// negations.
#pragma once
#include "rift_device.cuh"

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
__device__ __forceinline__ float lo(P2 a) {
    return __uint_as_float((unsigned)a.v);
}
__device__ __forceinline__ float hi(P2 a) {
    return __uint_as_float((unsigned)(a.v >> 32));
}
__device__ __forceinline__ P2 add2(P2 a, P2 b) {
    P2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 sub2(P2 a, P2 b) {
    P2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 mul2(P2 a, P2 b) {
    P2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ P2 fma2(P2 a, P2 b, P2 c) {
    P2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ P2 max2(P2 a, float b) { return pack2(fmaxf(lo(a), b), fmaxf(hi(a), b)); }
__device__ __forceinline__ P2 min2(P2 a, P2 b) {
    return pack2(fminf(lo(a), lo(b)), fminf(hi(a), hi(b)));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float minAbs3(float a, float b, float c) {
    float r;
    asm("min.ftz.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float rcpf(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ P2 rcp2(P2 a) { return pack2(rcpf(lo(a)), rcpf(hi(a))); }
__device__ __forceinline__ P2 sqrt2(P2 a) { return pack2(sqrtf(lo(a)), sqrtf(hi(a))); }

// slope() of rift_device.cuh is kSlope times this (kSlope = theta / 2), from
// the two differences: the outer factor goes into the fma that adds the slope.
constexpr float kSlope = 0.5f * kTheta;
constexpr float kMid = 0.5f / kTheta;
__device__ __forceinline__ float limit1(float dp, float dm) { return minAbs3(dp, dm, kMid * (dp + dm)); }
__device__ __forceinline__ P2 limit2(P2 dp, P2 dm) {
    const P2 b = mul2(both(kMid), add2(dp, dm));
    return pack2(minAbs3(lo(dp), lo(dm), lo(b)), minAbs3(hi(dp), hi(dm), hi(b)));
}

struct Face2 {  // depth and momenta on one face of two cells
    P2 h, u, v;
};

// construct() of rift_device.cuh; tw, tu, tv: the limited differences.
__device__ __forceinline__ void construct2(P2 h0, P2 u0, P2 v0, P2 tw, P2 tu, P2 tv, P2 eM, P2 eP,
                                           Face2& P, Face2& M) {
    const P2 k = both(kSlope), nk = both(-kSlope);
    const P2 hP = sub2(fma2(k, tw, h0), eP), hM = sub2(fma2(nk, tw, h0), eM);
    const P2 bar = sub2(add2(h0, h0), add2(eP, eM));
    P.h = min2(max2(hP, 0.f), bar);
    M.h = max2(min2(hM, bar), 0.f);
    P.u = fma2(k, tu, u0);
    M.u = fma2(nk, tu, u0);
    P.v = fma2(k, tv, v0);
    M.v = fma2(nk, tv, v0);
}

// One side of a face: velocities (n: normal, t: tangential), momenta formed
// from them, n + c and c - n, and the flux F(U).
struct Side2 {
    P2 n, qn, qt, sp, sm, f0, fn, ft;
};
__device__ __forceinline__ Side2 side2(P2 h, P2 qn, P2 qt, float kappa) {
    Side2 s;
    // 2h / (h^2 + max(h^2, kappa)), both halves of the fraction halved
    const P2 h2 = mul2(h, h), m = fma2(both(0.5f), h2, both(0.5f * kappa));
    const P2 r = mul2(h, rcp2(pack2(fmaxf(lo(h2), lo(m)), fmaxf(hi(h2), hi(m)))));
    const P2 n = mul2(qn, r), t = mul2(qt, r);
    s.qn = mul2(h, n);
    s.qt = mul2(h, t);
    const P2 c = sqrt2(mul2(both(kG), h));
    s.sp = add2(c, n);
    s.sm = sub2(c, n);
    const P2 hp = max2(h, 0.f);
    s.f0 = mul2(hp, n);
    s.fn = fma2(s.f0, n, mul2(mul2(both(0.5f * kG), hp), hp));
    s.ft = mul2(s.f0, t);
    return s;
}

// faceFlux() of rift_device.cuh; DIR 0: the normal momentum is hu.  f: mass,
// x momentum, y momentum; spd: the local speeds.
template <int DIR>
__device__ __forceinline__ void faceFlux2(const Face2& L, const Face2& R, float kappa, P2 f[3],
                                          P2& spd) {
    const Side2 a = side2(L.h, DIR == 0 ? L.u : L.v, DIR == 0 ? L.v : L.u, kappa);
    const Side2 b = side2(R.h, DIR == 0 ? R.u : R.v, DIR == 0 ? R.v : R.u, kappa);
    const P2 ap = pack2(max3(lo(a.sp), lo(b.sp), 0.f), max3(hi(a.sp), hi(b.sp), 0.f));
    const P2 am = pack2(max3(lo(a.sm), lo(b.sm), 0.f), max3(hi(a.sm), hi(b.sm), 0.f));
    const P2 r = rcp2(max2(add2(ap, am), 1e-30f));
    const P2 k = mul2(mul2(ap, am), r);
    f[0] = fma2(fma2(ap, a.f0, mul2(am, b.f0)), r, mul2(k, sub2(L.h, R.h)));
    const P2 fn = fma2(fma2(ap, a.fn, mul2(am, b.fn)), r, mul2(k, sub2(a.qn, b.qn)));
    const P2 ft = fma2(fma2(ap, a.ft, mul2(am, b.ft)), r, mul2(k, sub2(a.qt, b.qt)));
    f[1] = DIR == 0 ? fn : ft;
    f[2] = DIR == 0 ? ft : fn;
    spd = pack2(fmaxf(lo(ap), lo(am)), fmaxf(hi(ap), hi(am)));
}

}  // namespace rift
