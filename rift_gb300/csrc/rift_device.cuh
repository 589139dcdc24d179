// rift_device.cuh -- per-cell and per-face arithmetic of the GB300 step.
//
// The state is FP32 depth h (not surface elevation w), so the wet threshold
// epsilon (1.19e-7 m, grid.cu:29) is resolved at any bed elevation.  Every
// bed elevation enters through FP32 differences precomputed in FP64:
//   eW, eE : west / east face elevation minus the cell's reference elevation
//   eS, eN : south / north face elevation minus the same
// so w_{i+1} - w_i = (eE_i - eW_{i+1}) + (h_{i+1} - h_i) and the face depth
// w_face - B_face = h +- slope - e_face, with no large absolute elevation ever
// rounded to FP32.
#pragma once
#include <cstdint>

#include "rift_pair.cuh"

namespace rift {

constexpr float kG = 9.80665f;         // grid.cu:28
constexpr float kEps = 1.19209e-07f;   // grid.cu:29
constexpr float kTheta = 1.3f;         // grid.cu:30

// Effective limiter of the reference (grid.cu:62-80).  Its signf reads the
// low word of a double and is never negative, so minmod(a,b,c) evaluates to
// +min(|a|,|b|,|c|) (times a factor within 1.5e-6 of 1) and the slope is
//   0.5 * min(theta|d+|, 0.5|d+ + d-|, theta|d-|)  >= 0
// = 1/4 * min(2 theta min(|d+|, |d-|), |d+ + d-|), the minimum given here: the
// quarter, exact, goes into the fma that adds the slope.  It is zero whenever
// one argument is zero, which min() already gives.
constexpr float kSlope = 0.25f;
template <class V>
__device__ __forceinline__ V limited(V dp, V dm) {
    return minAbs(vmul(splat<V>(2.f * kTheta), minAbs(dp, dm)), vadd(dp, dm));
}

// State at one face of a cell (of two cells: V = P2): depth, hu, hv.
template <class V>
struct Face {
    V h, u, v;
};

// Reconstruction of one cell in one direction (Construct, grid.cu:91-116), in
// depth form, from the limited differences tw, tu, tv of the surface and the
// momenta: P at the face toward +x (+y), M toward -x.  eM/eP: the cell's - and
// + face elevation offsets.
// The wet/dry correction against the face elevations: wBar = 2w, so the face
// depths add up to bar = 2h - eP - eM, and "if (hP < 0) hP = 0, hM = bar; if
// (hM < 0) hM = 0, hP = bar" is min(max(hP, 0), bar) and max(min(hM, bar), 0).
// A NaN depth gives NaN depths at the cell's faces (no comparison holds for it),
// so it shows in the neighbours' momenta after one flux.
template <class V>
__device__ __forceinline__ void construct(V h0, V u0, V v0, V tw, V tu, V tv, V eM, V eP, Face<V>& P,
                                          Face<V>& M) {
    const V k = splat<V>(kSlope), nk = splat<V>(-kSlope), zero = splat<V>(0.f);
    const V hP = vsub(vfma(k, tw, h0), eP), hM = vsub(vfma(nk, tw, h0), eM);
    const V bar = vsub(vadd(h0, h0), vadd(eP, eM));
    P.h = vminNan(vmaxNan(hP, zero), bar);
    M.h = vmaxNan(vminNan(hM, bar), zero);
    P.u = vfma(k, tu, u0);
    M.u = vfma(nk, tu, u0);
    P.v = vfma(k, tv, v0);
    M.v = vfma(nk, tv, v0);
}

// Reconstructed face values of one cell from its neighbours' states.
struct Rec {
    float hP, uP, vP;  // depth, hu, hv at the + face
    float hM, uM, vM;  // at the - face
};

// h0/u0/v0: the cell; hp../hm..: its + and - neighbours in this direction;
// dP, dM: reference elevation steps to the + and - neighbour.
__device__ __forceinline__ Rec construct(float h0, float u0, float v0, float hp, float up, float vp,
                                         float hm, float um, float vm, float eM, float eP,
                                         float dP, float dM) {
    Face<float> P, M;
    construct(h0, u0, v0, limited(vadd(dP, vsub(hp, h0)), vadd(dM, vsub(h0, hm))),
              limited(vsub(up, u0), vsub(u0, um)), limited(vsub(vp, v0), vsub(v0, vm)), eM, eP, P, M);
    return Rec{P.h, P.u, P.v, M.h, M.u, M.v};
}

// Depth-only part of the reconstruction (speed pass): depth and the normal
// momentum at the two faces.
struct RecN {
    float hP, qP, hM, qM;
};

__device__ __forceinline__ RecN constructN(float h0, float q0, float hp, float qp, float hm,
                                           float qm, float eM, float eP, float dP, float dM) {
    Face<float> P, M;
    construct(h0, q0, q0, limited(vadd(dP, vsub(hp, h0)), vadd(dM, vsub(h0, hm))),
              limited(vsub(qp, q0), vsub(q0, qm)), 0.f, eM, eP, P, M);
    return RecN{P.h, P.u, M.h, M.u};
}

// Desingularised velocity factor 2h / (h^2 + max(h^2, kappa)) (grid.cu:82-84),
// both halves of the fraction halved.
template <class V>
__device__ __forceinline__ V velFactor(V h, float kappa) {
    const V h2 = vmul(h, h);
    return vmul(h, vrcp(vmax(h2, vfma(splat<V>(0.5f), h2, splat<V>(0.5f * kappa)))));
}

// One side of a face: velocities (n normal, t tangential), the momenta formed
// from them, the wave speeds n + c and c - n, and the flux F(U), zero where
// the depth is not positive (formed from the depth clamped at 0; a NaN velocity
// there makes it NaN instead).
template <class V>
struct Side {
    V t, qn, qt, sp, sm, f0, fn, ft;
};
template <class V>
__device__ __forceinline__ Side<V> faceSide(V h, V qn, V qt, float kappa) {
    Side<V> s;
    const V r = velFactor(h, kappa);
    const V n = vmul(qn, r), t = vmul(qt, r);
    s.t = t;
    s.qn = vmul(h, n);
    s.qt = vmul(h, t);
    const V c = vsqrt(vmul(splat<V>(kG), h));
    s.sp = vaddOfMul(c, n);
    s.sm = vsubOfMul(c, n);
    const V hp = vmax(h, splat<V>(0.f));
    s.f0 = vmul(hp, n);
    s.fn = vfma(vmul(splat<V>(0.5f * kG), hp), hp, vmul(s.f0, n));
    s.ft = vmul(s.f0, t);
    return s;
}

// Central-upwind numerical flux through one face (getHX for DIR 0, getHY for
// DIR 1; grid.cu:118-214, computeH grid.cu:86-89), from the upstream cell's +
// face (L) and the downstream cell's - face (R).  f[0] mass, f[1] x momentum,
// f[2] y momentum; returns the local speed max(a+, -a-).  a- enters as its
// magnitude; at a dry face (a+ = a- = 0) every product is zero, so 1 / max(a+
// - a-, tiny) takes the place of a branch.
template <int DIR, class V>
__device__ __forceinline__ V faceFlux(const Face<V>& L, const Face<V>& R, float kappa, V f[3]) {
    const Side<V> a = faceSide(L.h, DIR == 0 ? L.u : L.v, DIR == 0 ? L.v : L.u, kappa);
    const Side<V> b = faceSide(R.h, DIR == 0 ? R.u : R.v, DIR == 0 ? R.v : R.u, kappa);
    const V ap = vmaxz(a.sp, b.sp), am = vmaxz(a.sm, b.sm);
    const V r = vrcp(vmax(vadd(ap, am), splat<V>(1e-30f)));
    const V k = vmul(vmul(ap, am), r);
    f[0] = vfma(vfma(ap, a.f0, vmul(am, b.f0)), r, vmul(k, vsub(L.h, R.h)));
    const V fn = vfma(vfma(ap, a.fn, vmul(am, b.fn)), r, vmul(k, vsubOfMul(a.qn, b.qn)));
    const V ft = vfma(vfma(ap, a.ft, vmul(am, b.ft)), r, vmul(k, vfnma(R.h, b.t, a.qt)));
    f[1] = DIR == 0 ? fn : ft;
    f[2] = DIR == 0 ? ft : fn;
    return vmax(ap, am);
}
template <int DIR>
__device__ __forceinline__ float faceFlux(float hL, float huL, float hvL, float hR, float huR,
                                          float hvR, float kappa, float f[3]) {
    return faceFlux<DIR>(Face<float>{hL, huL, hvL}, Face<float>{hR, huR, hvR}, kappa, f);
}

// Local speed at a face (the mx / my of getHX / getHY, grid.cu:118-214) as the
// speed pass takes it, without the fluxes; qn is the momentum normal to the
// face.  Its sums n + c and c - n are fmas, faceFlux's are not: the two may
// differ in the last bit.
__device__ __forceinline__ float faceSpeed(float hL, float qL, float hR, float qR, float kappa) {
    const float rL = velFactor(hL, kappa), rR = velFactor(hR, kappa);
    const float cL = vsqrt(vmul(kG, hL)), cR = vsqrt(vmul(kG, hR));
    return fmaxf(vmaxz(vfma(qL, rL, cL), vfma(qR, rR, cR)), vmaxz(vfnma(qL, rL, cL), vfnma(qR, rR, cR)));
}

// Flux divergence from the differences of the fluxes through a cell's east and
// west (fx) and north and south faces (fy).
template <class V>
__device__ __forceinline__ V divergence(V fx, V fy, float inv_dx, float inv_dy) {
    return vfma(fx, splat<V>(-inv_dx), vmul(fy, splat<V>(-inv_dy)));
}

// d plus the bed-slope source of a momentum equation (grid.cu:701,751-752): eM
// and eP are the cell's face offsets in the direction, inv its inverse width.
template <class V>
__device__ __forceinline__ V addBed(V d, V hC, V eM, V eP, float inv) {
    return vaddOfMul(d, vmul(vmul(splat<V>(-kG), hC), vmul(vsub(eP, eM), splat<V>(inv))));
}

// The sums below state which product goes into an fma: left to the compiler,
// the choice changes with the kernel they are inlined in, and the schedules
// would round apart.

// Green-Ampt infiltration rate (grid.cu:791-805), clamped to [0, h/dt].
// The quadratic root is taken in the cancellation-free form when p1 < 0.
__device__ __forceinline__ float greenAmpt(float K, float F, float psiDtheta, float dt, float hC) {
    float p1 = vfma(K, dt, -2.f * F);
    float p2 = vmul(K, vadd(F, psiDtheta));
    float s = sqrtf(vfma(p1, p1, vmul(8.f * p2, dt)));
    float f = (p1 >= 0.f) ? (p1 + s) / (2.f * dt) : (4.f * p2) / (s - p1);
    float cap = hC / dt;
    f = (f > cap) ? cap : f;
    f = (f > 0.f) ? f : 0.f;
    return f;
}

// Semi-implicit Manning coefficient G (grid.cu:754-760).
__device__ __forceinline__ float manningG(float n, float hu, float hv, float hC, float kappa) {
    float h2 = vmul(hC, hC);
    float den = vadd(h2, fmaxf(h2, kappa));
    return -4.f * kG * n * n * sqrtf(vfma(hu, hu, vmul(hv, hv))) * powf(hC, 5.f / 3.f) / (den * den);
}

// Critical-depth ghost value (ApplyBoundariesX_k / Y_k, grid.cu:1325-1406):
// min((q^2/g)^(1/3), h_interior).
__device__ __forceinline__ float criticalDepth(float q, float h) {
    return fminf(cbrtf(q * q / kG), h);
}

}  // namespace rift
