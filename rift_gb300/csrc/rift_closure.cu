// rift_closure.cu -- learned sub-grid flux closure on a 2x-coarsened grid.
//
// The net (6 -> 32 channels 5x5, 32 -> 32 3x3, 32 -> 4 1x1, ReLU between)
// runs tile by tile: a 22 x 22 block of the six input channels, layer 1 on the
// 18 x 18 cells that layer 2 needs, layers 2 and 3 on the 16 x 16 output cells.
// Every contraction is an implicit GEMM on BF16 operands with FP32
// accumulation: rows are cells, columns output channels, and the reduction
// runs over (tap, input channel).
//
// Inference (k_forward, k_closure) runs on tcgen05.mma with accumulators in
// tensor memory, four blocks in flight per SM.  Training (k_train) recomputes
// the forward pass of its tile and runs the backward pass in the same CTA, on
// mma.sync with fragments by ldmatrix: layer-3 gradients on the CUDA cores
// (4 x 32 weights), the layer-2 and layer-1 weight gradients and the layer-1
// activation gradient as GEMMs.  Weight gradients stay in registers across
// every tile a CTA visits and are added to the global gradient once per CTA.
//
// The flux kernel evaluates the step's central-upwind face flux
// (rift_device.cuh) on a handle's state, for the time-integrated fluxes
// through coarse faces that make the training targets.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/rift_closure.h"
#include "rift_device.cuh"

namespace rc {

constexpr int CIN = 6, C1 = 32, COUT = 4;
constexpr int K1 = 150, K1P = 160, K2 = 288;
constexpr int OT = 16;           // output tile side
constexpr int R1 = OT + 2;       // layer-1 region side (18)
constexpr int RI = OT + 6;       // input region side (22)
constexpr int NR1 = R1 * R1;     // 324
constexpr int NRI = RI * RI;     // 484
constexpr int M1T = (NR1 + 15) / 16;  // 21 MMA row tiles of layer 1
constexpr int SA = 40;           // BF16 row stride of the activation tiles
constexpr int CB = 8;            // BF16 input channels per cell: h, hu, hv, b_hi, b_lo, n, rain, 0
constexpr int NTAP1 = 26;        // layer-1 taps, the 26th a zero-weight pad
constexpr int K1B = NTAP1 * CB;  // 208: layer-1 reduction over the BF16 inputs
constexpr int SW1 = K1B + 8, SW2 = 296, SW3 = 40;  // BF16 row strides of the weights
constexpr int TT = 512;          // threads of a training CTA: 16 warps

constexpr int OFF_W1 = RIFT_CLOSURE_OFF_W1, OFF_B1 = RIFT_CLOSURE_OFF_B1;
constexpr int OFF_W2 = RIFT_CLOSURE_OFF_W2, OFF_B2 = RIFT_CLOSURE_OFF_B2;
constexpr int OFF_W3 = RIFT_CLOSURE_OFF_W3, OFF_B3 = RIFT_CLOSURE_OFF_B3;
static_assert(OFF_B1 == OFF_W1 + C1 * K1P && OFF_W2 == OFF_B1 + C1 && OFF_B2 == OFF_W2 + C1 * K2 &&
                  OFF_W3 == OFF_B2 + C1 && OFF_B3 == OFF_W3 + 8 * C1 &&
                  RIFT_CLOSURE_NPARAM == OFF_B3 + 8,
              "parameter layout");

struct __align__(128) TrainSmem {
    uint16_t xb[NRI * CB];      // input cells: BF16 rows of 8, the bed relative to bref in two halves
    uint16_t a1[NR1 * SA];      // layer-1 activations (BF16); dZ1 in the backward pass
    uint16_t a2[OT * OT * SA];  // layer-2 activations, then dZ2
    uint16_t w1[C1 * SW1];      // W1 over the BF16 inputs: [o][tap*8 + c8]
    uint16_t w2[C1 * SW2];      // W2[o][k]
    uint16_t w3[8 * SW3];       // W3[o][c], rows 4..7 zero
    uint16_t zero[SA];          // a row of zeros, for cells outside
    float dout[OT * OT * 4];
    float w3q[C1][4];           // W3 (FP32), a channel's four weights together
    float xbed[NRI];            // scaled FP32 bed of the input cells
    float b1[C1], b2[C1], b3[8];
    float sbed[C1];             // sum over taps of layer 1's (BF16) bed weights
    int toff[NTAP1];            // cell offset of each layer-1 tap in the input block
    int qcell[M1T * 16];        // input cell of each layer-1 cell (its window's corner)
    float bref;                 // the block's reference bed (scaled)
    double red[TT / 32];
};
static_assert(offsetof(TrainSmem, a1) % 16 == 0 && offsetof(TrainSmem, a2) % 16 == 0 &&
                  offsetof(TrainSmem, w1) % 16 == 0 && offsetof(TrainSmem, w2) % 16 == 0 &&
                  offsetof(TrainSmem, zero) % 16 == 0 && offsetof(TrainSmem, dout) % 16 == 0 &&
                  offsetof(TrainSmem, w3q) % 16 == 0 && SA % 8 == 0 && SW1 % 8 == 0 && SW2 % 8 == 0,
              "fragment loads are 16-byte aligned");

__device__ __forceinline__ uint16_t bf(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float fb(uint16_t x) { return __bfloat162float(__ushort_as_bfloat16(x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    return (uint32_t)bf(lo) | ((uint32_t)bf(hi) << 16);
}
__device__ __forceinline__ uint32_t pack16(uint16_t lo, uint16_t hi) {
    return (uint32_t)lo | ((uint32_t)hi << 16);
}
__device__ __forceinline__ uint32_t ld32(const uint16_t* p) {
    return *reinterpret_cast<const uint32_t*>(p);
}
__device__ __forceinline__ void st32(uint16_t* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }
__device__ __forceinline__ float relu(float x) { return fmaxf(x, 0.f); }

// D += A(16x16, row) * B(16x8, col), BF16 inputs, FP32 accumulators.
// Fragments (g = lane/4, t = lane%4): a[0] rows g, cols 2t..2t+1; a[1] rows
// g+8; a[2] rows g, cols 2t+8..; a[3] rows g+8, cols 2t+8..; b0 rows (k)
// 2t..2t+1 of col g, b1 rows 2t+8..; d[0..1] row g cols 2t..2t+1, d[2..3]
// row g+8.
__device__ __forceinline__ void mma16816(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Four 8x8 BF16 matrices from shared memory; lane l gives the address of
// row l%8 of matrix l/8, and r[i] receives matrix i in the MMA fragment
// layout (thread T: row T/4, columns 2(T%4), 2(T%4)+1).  Row addresses are
// 16-byte aligned.
__device__ __forceinline__ void ldsm4(uint32_t r[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// The same, each matrix transposed: thread T receives rows 2(T%4), 2(T%4)+1 of
// column T/4.
__device__ __forceinline__ void ldsm4t(uint32_t r[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// Weights (BF16), biases and the offset tables, once per CTA.  Layer 1 reads
// the BF16 input rows (h, hu, hv, b_hi, b_lo, n, rain, 0): both bed halves
// take the bed weight.
// Cell offset of a layer-1 tap in the input block (0 for a pad tap).
__device__ __forceinline__ int tapCell(int tap) { return tap < 25 ? (tap / 5) * RI + tap % 5 : 0; }

__device__ void stageNet(TrainSmem& S, const float* __restrict__ P) {
    const int tid = threadIdx.x;
    constexpr int MAP[CB] = {0, 1, 2, 3, 3, 4, 5, -1};
    for (int i = tid; i < C1 * SW1; i += TT) {
        const int o = i / SW1, k = i % SW1, tap = k / CB, c = MAP[k % CB];
        S.w1[i] = bf(k < K1B && tap < 25 && c >= 0 ? P[OFF_W1 + o * K1P + tap * CIN + c] : 0.f);
    }
    for (int i = tid; i < C1 * SW2; i += TT) {
        int o = i / SW2, k = i % SW2;
        S.w2[i] = bf(k < K2 ? P[OFF_W2 + o * K2 + k] : 0.f);
    }
    for (int i = tid; i < 8 * SW3; i += TT) {
        int o = i / SW3, k = i % SW3;
        S.w3[i] = bf(o < COUT && k < C1 ? P[OFF_W3 + o * C1 + k] : 0.f);
    }
    if (tid < 4 * C1) S.w3q[tid % C1][tid / C1] = P[OFF_W3 + tid];
    if (tid < SA) S.zero[tid] = 0;
    if (tid < C1) {
        S.b1[tid] = P[OFF_B1 + tid];
        S.b2[tid] = P[OFF_B2 + tid];
        float sb = 0.f;
        for (int tap = 0; tap < 25; tap++) sb += fb(bf(P[OFF_W1 + tid * K1P + tap * CIN + 3]));
        S.sbed[tid] = sb;
    }
    if (tid < 8) S.b3[tid] = tid < COUT ? P[OFF_B3 + tid] : 0.f;
    if (tid < NTAP1) S.toff[tid] = tapCell(tid);
    if (tid < M1T * 16) {
        const int q = min(tid, NR1 - 1);
        S.qcell[tid] = (q / R1) * RI + q % R1;
    }
}

// This thread's cell of the 22 x 22 input block whose corner is image cell (Y0,
// X0) of sample s, and the block's reference bed (its centre cell's): loaded one
// block ahead.
struct TrainInput {
    float v[CIN];
    float bref;
};
__device__ __forceinline__ void loadInput(TrainInput& R, const rift_closure_src& src, int s, int Y0, int X0) {
    const size_t sbase = (size_t)s * (size_t)src.sample_stride;
    auto at = [&](int ry, int rx) {
        int y = min(max(Y0 + ry, 0), src.H - 1), x = min(max(X0 + rx, 0), src.W - 1);
        return sbase + (size_t)y * (size_t)src.pitch + (size_t)x;
    };
    const int i = min((int)threadIdx.x, NRI - 1);
    const size_t off = at(i / RI, i % RI);
    R.bref = src.plane[3] ? __ldg(src.plane[3] + at(RI / 2, RI / 2)) : src.value[3];
#pragma unroll
    for (int c = 0; c < CIN; c++) R.v[c] = src.plane[c] ? __ldg(src.plane[c] + off) : src.value[c];
}
// ... into shared memory.  The BF16 bed is b - bref, split into a BF16 value and
// its BF16 remainder (16 significant bits together).
__device__ __forceinline__ void storeInput(TrainSmem& S, const TrainInput& R, const rift_closure_src& src) {
    const int i = threadIdx.x;
    const float bref = R.bref * src.scale[3];
    if (i == 0) S.bref = bref;
    if (i >= NRI) return;
    float v[CIN];
#pragma unroll
    for (int c = 0; c < CIN; c++) v[c] = R.v[c] * src.scale[c];
    S.xbed[i] = v[3];
    const float br = v[3] - bref;
    const uint16_t bh = bf(br);
    const uint16_t bl = bf(br - fb(bh));
    uint4 w;
    w.x = pack2(v[0], v[1]);
    w.y = pack16(bf(v[2]), bh);
    w.z = pack16(bl, bf(v[4]));
    w.w = pack16(bf(v[5]), 0);
    *reinterpret_cast<uint4*>(&S.xb[i * CB]) = w;
}

// Passes over the 18 x 18 layer-1 cells: a warp takes one half of the 32
// channels and up to three of the 21 row tiles of 16 cells.
constexpr int WPH = TT / 64, UPW = (M1T + WPH - 1) / WPH;

// Layer 1 on the 18 x 18 region: a1 = relu(W1 x + b1), BF16.  One k step covers
// two taps of the 8-channel BF16 input rows, so each 8 x 8 block of an A
// fragment is 8 cells' rows of one tap and comes with one ldmatrix; the
// bed enters relative to bref and the epilogue subtracts (centre bed -
// bref) x (sum of the bed weights), which makes it relative to the
// window's centre.
__device__ __forceinline__ void conv1(TrainSmem& S, int warp, int lane) {
    const int g = lane >> 2, t = lane & 3;
    // this lane's ldmatrix rows: row (lane & 15) of each of its row tiles,
    // the tap of the k step's second half for lanes 16..31
    const int lrow = lane & 15, lhalf = lane >> 4;
    const int wrow = (lane & 7) + ((lane >> 4) << 3), wk = ((lane >> 3) & 1) * 8;
    const int half = warp & 1, mt0 = warp >> 1;
    int cell[UPW];
#pragma unroll
    for (int j = 0; j < UPW; j++) cell[j] = S.qcell[min(mt0 + WPH * j, M1T - 1) * 16 + lrow];
    const uint16_t* wp = &S.w1[(half * 16 + wrow) * SW1 + wk];
    float acc[UPW][2][4] = {};
#pragma unroll 13
    for (int ks = 0; ks < K1B / 16; ks++) {
        const int toff = S.toff[2 * ks + lhalf];
        uint32_t b[4];
        ldsm4(b, wp + ks * 16);
#pragma unroll
        for (int j = 0; j < UPW; j++) {
            if (mt0 + WPH * j >= M1T) break;
            uint32_t a[4];
            ldsm4(a, &S.xb[(cell[j] + toff) * CB]);
            mma16816(acc[j][0], a, b[0], b[1]);
            mma16816(acc[j][1], a, b[2], b[3]);
        }
    }
    const float bref = S.bref;
#pragma unroll
    for (int j = 0; j < UPW; j++) {
        if (mt0 + WPH * j >= M1T) break;
        const int r0 = (mt0 + WPH * j) * 16 + g, r1 = r0 + 8;
        const float c0 = S.xbed[S.qcell[r0] + 2 * RI + 2] - bref;
        const float c1 = S.xbed[S.qcell[r1] + 2 * RI + 2] - bref;
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
            const int o = half * 16 + nt * 8 + 2 * t;
            const float s0 = S.sbed[o], s1 = S.sbed[o + 1];
            if (r0 < NR1)
                st32(&S.a1[r0 * SA + o], pack2(relu(acc[j][nt][0] + S.b1[o] - c0 * s0),
                                               relu(acc[j][nt][1] + S.b1[o + 1] - c0 * s1)));
            if (r1 < NR1)
                st32(&S.a1[r1 * SA + o], pack2(relu(acc[j][nt][2] + S.b1[o] - c1 * s0),
                                               relu(acc[j][nt][3] + S.b1[o + 1] - c1 * s1)));
        }
    }
}

// Layers 2 and 3 on output row `warp` (A and B fragments by ldmatrix).  z2:
// layer-2 pre-activations (accumulator fragments); out: layer-3 outputs of rows
// g and g+8, channels 2t and 2t+1 (t < 2 valid).
__device__ __forceinline__ void conv23(const TrainSmem& S, int warp, int lane, float z2[4][4], float out[4]) {
    const int g = lane >> 2, t = lane & 3;
    const int lrow = lane & 15, lk = (lane >> 4) * 8;  // A: row, k offset of this lane's address
    const int wrow = (lane & 7) + ((lane >> 4) << 3), wk = ((lane >> 3) & 1) * 8;
    float acc[4][4] = {};
#pragma unroll 3
    for (int tap = 0; tap < 9; tap++) {
        const int dy = tap / 3, dx = tap % 3;
        const uint16_t* p = &S.a1[((warp + dy) * R1 + lrow + dx) * SA + lk];
#pragma unroll
        for (int kb = 0; kb < 2; kb++) {
            const int kk = tap * 32 + kb * 16;
            uint32_t a[4], b0[4], b1[4];
            ldsm4(b0, &S.w2[wrow * SW2 + kk + wk]);
            ldsm4(b1, &S.w2[(16 + wrow) * SW2 + kk + wk]);
            ldsm4(a, p + kb * 16);
            mma16816(acc[0], a, b0[0], b0[1]);
            mma16816(acc[1], a, b0[2], b0[3]);
            mma16816(acc[2], a, b1[0], b1[1]);
            mma16816(acc[3], a, b1[2], b1[3]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
        const int o = nt * 8 + 2 * t;
        z2[nt][0] = acc[nt][0] + S.b2[o];
        z2[nt][1] = acc[nt][1] + S.b2[o + 1];
        z2[nt][2] = acc[nt][2] + S.b2[o];
        z2[nt][3] = acc[nt][3] + S.b2[o + 1];
    }
    float acc3[4] = {};
#pragma unroll
    for (int kb = 0; kb < 2; kb++) {
        uint32_t a[4];
        a[0] = pack2(relu(z2[2 * kb][0]), relu(z2[2 * kb][1]));
        a[1] = pack2(relu(z2[2 * kb][2]), relu(z2[2 * kb][3]));
        a[2] = pack2(relu(z2[2 * kb + 1][0]), relu(z2[2 * kb + 1][1]));
        a[3] = pack2(relu(z2[2 * kb + 1][2]), relu(z2[2 * kb + 1][3]));
        const uint16_t* w = &S.w3[g * SW3 + kb * 16 + 2 * t];
        mma16816(acc3, a, ld32(w), ld32(w + 8));
    }
    const int c = 2 * t;  // b3 holds 8 entries, zero past the fourth
    out[0] = acc3[0] + S.b3[c];
    out[1] = acc3[1] + S.b3[c + 1];
    out[2] = acc3[2] + S.b3[c];
    out[3] = acc3[3] + S.b3[c + 1];
}

struct TileGeom {
    int s, Y, X;  // sample and image coordinates of the tile's first output cell
};
__device__ __forceinline__ TileGeom tileGeom(const rift_closure_src& src, int tile) {
    const int tx = (src.OW + OT - 1) / OT, ty = (src.OH + OT - 1) / OT;
    TileGeom G;
    G.s = tile / (tx * ty);
    int r = tile % (tx * ty);
    G.Y = src.oy0 + (r / tx) * OT;
    G.X = src.ox0 + (r % tx) * OT;
    return G;
}
__host__ __device__ __forceinline__ int tileCount(const rift_closure_src& src) {
    return src.samples * ((src.OW + OT - 1) / OT) * ((src.OH + OT - 1) / OT);
}

// ------------------------------------------------- tcgen05 forward (inference)
// The forward pass of k_forward and k_closure on the 5th-generation tensor
// cores: layers 1 and 2 are tcgen05.mma (kind::f16, BF16 operands from
// shared memory, FP32 accumulators in tensor memory), issued by one thread;
// layer 3 (32 -> 4) runs in FP32 on the CUDA cores in the layer-2 epilogue.
//
// Implicit GEMM without an im2col copy.  The input block and the layer-1
// activations are stored as cells of 8 BF16 channels (16 bytes, one row of
// an 8 x 16-byte core matrix), cell (y, x) of the 22-wide block at linear
// index y*22 + x.  An MMA row is a linear cell index m, so the eight rows of
// a core matrix are eight consecutive cells (16-byte stride) and the row
// groups are 128 bytes apart; the operand of tap (dy, dx) is the same
// layout started dy*22 + dx cells later.  Rows whose column m % 22 is past
// the valid width compute values that no valid output reads.
//  layer 1: M = 512 rows (4 tiles of 128; the 18 x 18 region is rows
//           m < 396 with m % 22 < 18), N = 32, K = 15 steps of 16: taps
//           (dy, dx) and (dy+1, dx) for dy = 0, 2, 4 (dy = 5 carries zero
//           weights), the two 8-channel K chunks 22 cells apart.  (Taps 2s and
//           2s + 1 would need 13 steps, but another order of the sum rounds
//           some activations to another BF16: 2.7e-5 off in the output.);
//  layer 2: M = 384 rows (3 tiles; the 16 x 16 outputs are rows m < 352
//           with m % 22 < 16), N = 32, K = 9 taps x 2 steps of 16 over the
//           four 8-channel planes of the layer-1 activations.
//
// What bounds it: an MMA reads its 4 KB of A from shared memory whatever N is:
// 61 cycles one after another in one CTA, 39 per SM with several CTAs (at N =
// 32, 46 at 64), so a block's 114 take 4,400 cycles of the tensor pipe.  To
// keep that pipe busy, one CTA per SM runs four blocks at a time, each on a
// group of four warps and an issuing warp: the weights are staged once for the
// four (three CTAs of 74 KB fitted before), the groups meet at no barrier, and
// an M tile's epilogue and layer 2's MMAs start as soon as what they read is
// there.  Tensor memory: 128 columns per
// group, all 512; one 32-column accumulator per M tile, layer 2 reuses the
// columns of layer 1 once its epilogue has read them.
// 256 patches of 64 x 64 (4,096 blocks): 125 us with three CTAs per SM, tensor
// pipe 59% busy; 89 with four groups and issuing warps, 77% busy; 78 with the
// parameters read in their own order.
constexpr int XBC = 640;             // BF16 input cells staged (reads reach m + 5*22 + 4 < 640)
constexpr int A1C = 432;             // layer-1 cells kept per plane (layer 2 reads < 384 + 46)
constexpr int M1TC = 4, M2TC = 3;    // M tiles of 128 rows
constexpr int KS1 = 15, KS2 = 18;    // K steps of 16
constexpr int TCG = 4;               // groups (blocks in flight) per CTA
constexpr int GT = 128;              // threads per group
constexpr int TCT = TCG * (GT + 32); // threads per CTA: the groups', then an issuing warp for each
constexpr int NTAPT = 26;            // layer-1 weight blocks: the 25 taps, then one of zeros
constexpr uint32_t TMEM_COLS = 128;
constexpr uint32_t A1PLANE = A1C * 16;  // bytes per 8-channel plane
// instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and B
// BF16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at
// bits 24-28
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

struct __align__(128) TcGroup {  // one block in flight
    uint16_t xb[XBC * 8];        // input cells (BF16 x 8), zero past the 22 x 22 block
    uint16_t a1[4][A1C * 8];     // layer-1 activations, channels 8p..8p+7 in plane p
    float xh[NRI];               // scaled FP32 depth of the input cells
    float xbed[NRI];             // scaled FP32 bed of the input cells
    float bref;
    int red;
    int stop;                    // to the issuing warp: no more blocks
    int next;                    // the group's next block
    uint64_t bar[M1TC + M2TC];   // completion of each M tile's MMAs: layer 1, then layer 2
    uint64_t in;                 // a block is staged, or `stop` set (1 arrival)
    uint64_t act[M1TC];          // the tile's layer-1 epilogue is done (4 arrivals)
};
struct __align__(128) TcSmem {
    TcGroup g[TCG];
    uint16_t w1t[NTAPT * 32 * 8];  // [dy*5 + dx][o][c8]; block 25 all zero
    uint16_t w2t[36 * 32 * 8];   // [tap*4 + c/8][o][c%8]
    float w3[C1][COUT];
    float b1[C1], b2[C1], b3[COUT], sbed[C1];
    uint32_t tmem;
};
static_assert(sizeof(TcGroup) % 128 == 0 && offsetof(TcGroup, a1) % 16 == 0 &&
                  offsetof(TcGroup, bar) % 8 == 0 && offsetof(TcSmem, w1t) % 16 == 0 &&
                  offsetof(TcSmem, w2t) % 16 == 0 && offsetof(TcSmem, w3) % 16 == 0 &&
                  offsetof(TcSmem, b1) % 16 == 0 && offsetof(TcSmem, sbed) % 16 == 0,
              "operand alignment");
static_assert(sizeof(TcSmem) <= 227 * 1024, "shared memory of one CTA");

// Group of this thread (of the group itself, or of its issuing warp).
__device__ __forceinline__ int tcGroupOf() {
    const int t = threadIdx.x;
    return t < TCG * GT ? t / GT : (t - TCG * GT) / 32;
}
// Barrier of one group's threads (barrier 0 is the CTA's).
__device__ __forceinline__ void groupSync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(GT) : "memory");
}
__device__ __forceinline__ bool groupAnd(int g, bool p) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, %2, %3, p;\n"
        " selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(g + 1), "n"(GT)
        : "memory");
    return r != 0;
}

__device__ int g_tc_error;  // 1: a tensor-core completion wait gave up

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (tcgen05): start address, leading (K)
// and stride (M/N) byte offsets, each >> 4; version 1 at bit 46; no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
           ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, bool acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(IDESC), "r"((uint32_t)acc)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count = 1) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
// Bounded wait on an mbarrier phase: false after the spin limit.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// 32 consecutive FP32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
        "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; k++) v[k] = __uint_as_float(r[k]);
}

// Weights in the operand layouts, biases, the bed-weight sums; the zero pad
// of the input cells.  Tensor memory (warp 0) and the completion barriers.
// The parameters are read in their own order, a run of independent coalesced
// loads per thread, and scattered in shared memory: read in the order of the
// operands, the setup was most of a one-block launch (19.8 us).
__device__ void tcSetup(TcSmem& S, const float* __restrict__ P) {
    const int tid = threadIdx.x;
    constexpr int NP = RIFT_CLOSURE_NPARAM;
    constexpr int PT = (NP + TCT - 1) / TCT;
    float v[PT];
#pragma unroll
    for (int q = 0; q < PT; q++) v[q] = tid + q * TCT < NP ? __ldg(P + tid + q * TCT) : 0.f;
    // channel 7 of every layer-1 cell and the last weight block are zero
    for (int i = tid; i < NTAPT * 32; i += TCT) {
        S.w1t[i * 8 + 7] = 0;
        if (i >= 25 * 32) *reinterpret_cast<uint4*>(&S.w1t[i * 8]) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int i = tid; i < TCG * (XBC - NRI) * 8; i += TCT)
        S.g[i / ((XBC - NRI) * 8)].xb[NRI * 8 + i % ((XBC - NRI) * 8)] = 0;
#pragma unroll
    for (int q = 0; q < PT; q++) {
        const int i = tid + q * TCT;
        if (i < OFF_B1) {
            const int o = i / K1P, k = i % K1P, tap = k / CIN, c = k % CIN;
            if (k < K1) {  // both halves of the bed (channels 3, 4) take its weight
                uint16_t* w = &S.w1t[(tap * 32 + o) * 8];
                w[c < 4 ? c : c + 1] = bf(v[q]);
                if (c == 3) w[4] = bf(v[q]);
            }
        } else if (i < OFF_W2) {
            S.b1[i - OFF_B1] = v[q];
        } else if (i < OFF_B2) {
            const int o = (i - OFF_W2) / K2, k = (i - OFF_W2) % K2, tap = k / C1, c = k % C1;
            S.w2t[((tap * 4 + c / 8) * 32 + o) * 8 + c % 8] = bf(v[q]);
        } else if (i < OFF_W3) {
            S.b2[i - OFF_B2] = v[q];
        } else if (i < OFF_W3 + COUT * C1) {
            S.w3[(i - OFF_W3) % C1][(i - OFF_W3) / C1] = v[q];
        } else if (i >= OFF_B3 && i < OFF_B3 + COUT) {
            S.b3[i - OFF_B3] = v[q];
        }
    }
    if (tid < TCG) {
        TcGroup& G = S.g[tid];
        for (int k = 0; k < M1TC + M2TC; k++) bar_init(&G.bar[k]);
        for (int k = 0; k < M1TC; k++) bar_init(&G.act[k], GT / 32);
        bar_init(&G.in);
        G.stop = 0;
    }
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         saddr(&S.tmem)),
                     "r"(TCG * TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    proxy_fence();  // the weights are read by the tensor cores
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (tid >= TCG * GT && tid < TCG * GT + C1) {
        const int o = tid - TCG * GT;
        float sb = 0.f;
        for (int tap = 0; tap < 25; tap++) sb += fb(S.w1t[(tap * 32 + o) * 8 + 3]);
        S.sbed[o] = sb;
    }
    __syncthreads();
}

__device__ void tcTeardown(TcSmem& S) {
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem),
                     "r"(TCG * TMEM_COLS)
                     : "memory");
}

// A block's raw inputs in registers: this thread's cells of the 22 x 22 block
// (484 < 4 GT), and the block's reference bed.  Loaded one block ahead, while
// the tensor cores work on the current one.
constexpr int TCC = (NRI + GT - 1) / GT;
struct TcInput {
    float v[TCC][CIN];
    float bref;
};
__device__ __forceinline__ void tcLoadInput(TcInput& R, const rift_closure_src& src, int s, int Y0,
                                            int X0) {
    const size_t sbase = (size_t)s * (size_t)src.sample_stride;
    auto at = [&](int ry, int rx) {
        int y = min(max(Y0 + ry, 0), src.H - 1), x = min(max(X0 + rx, 0), src.W - 1);
        return sbase + (size_t)y * (size_t)src.pitch + (size_t)x;
    };
    R.bref = src.plane[3] ? __ldg(src.plane[3] + at(RI / 2, RI / 2)) : src.value[3];
#pragma unroll
    for (int k = 0; k < TCC; k++) {
        const int i = threadIdx.x % GT + k * GT;
        if (i >= NRI) break;
        const size_t off = at(i / RI, i % RI);
#pragma unroll
        for (int c = 0; c < CIN; c++) R.v[k][c] = src.plane[c] ? __ldg(src.plane[c] + off) : src.value[c];
    }
}

// The loaded block into shared memory: scaled FP32 depth and bed and the
// BF16 cells of the layer-1 operand (the bed relative to bref in two
// halves); each writer fences its shared stores for the async proxy.
__device__ __forceinline__ void tcStoreInput(TcGroup& S, const TcInput& R, const rift_closure_src& src) {
    const float bref = R.bref * src.scale[3];
    if (threadIdx.x % GT == 0) S.bref = bref;
#pragma unroll
    for (int k = 0; k < TCC; k++) {
        const int i = threadIdx.x % GT + k * GT;
        if (i >= NRI) break;
        float v[CIN];
#pragma unroll
        for (int c = 0; c < CIN; c++) v[c] = R.v[k][c] * src.scale[c];
        S.xh[i] = v[0];
        S.xbed[i] = v[3];
        const float br = v[3] - bref;
        const uint16_t bh = bf(br);
        const uint16_t bl = bf(br - fb(bh));
        uint4 w;
        w.x = pack2(v[0], v[1]);
        w.y = pack16(bf(v[2]), bh);
        w.z = pack16(bl, bf(v[4]));
        w.w = pack16(bf(v[5]), 0);
        *reinterpret_cast<uint4*>(&S.xb[i * CB]) = w;
    }
    proxy_fence();
}

// One thread: the MMAs of layer 1 / of M tile mt of layer 2, each
// M tile's completion on a barrier of its own.  The loops unroll completely:
// every operand offset is a compile-time constant added to a base descriptor
// (its address field counts 16-byte units, and no shared address reaches 256
// KB, so the sum never carries out of the field), so the issuing thread spends
// a few instructions per MMA.
__device__ __forceinline__ void tcIssue1(const TcSmem& S, TcGroup& G, uint32_t tmem) {
    tc_after_sync();
    // B: the K chunks of step s are taps (dy, dx) and (dy + 1, dx), dy = 2(s/5), five weight
    // blocks apart; for dy = 4 the second chunk is the zero block
    const uint64_t a0 = sdesc(saddr(G.xb), RI * 16, 128), b0 = sdesc(saddr(S.w1t), 0, 128);
#pragma unroll
    for (int mt = 0; mt < M1TC; mt++) {
#pragma unroll
        for (int s = 0; s < KS1; s++) {
            const uint32_t cell = mt * 128 + (s / 5) * 2 * RI + s % 5;  // 16-byte cells
            const uint32_t T0 = (s / 5) * 10 + s % 5, T1 = s < 10 ? T0 + 5 : 25;
            const uint64_t lbo = (uint64_t)((T1 - T0) * 512 / 16) << 16;
            tc_mma(tmem + mt * 32, a0 + cell, b0 + T0 * (512 / 16) + lbo, s > 0);
        }
        tc_commit(&G.bar[mt]);
    }
}
__device__ __forceinline__ void tcIssue2(const TcSmem& S, TcGroup& G, uint32_t tmem, int mt) {
    tc_after_sync();
    const uint64_t a0 = sdesc(saddr(G.a1), A1PLANE, 128) + mt * 128, b0 = sdesc(saddr(S.w2t), 512, 128);
#pragma unroll
    for (int s = 0; s < KS2; s++) {
        const int tap = s >> 1, kb = s & 1;
        const uint32_t cell = kb * 2 * A1C + (tap / 3) * RI + tap % 3;
        tc_mma(tmem + mt * 32, a0 + cell, b0 + (tap * 4 + 2 * kb) * (512 / 16), s > 0);
    }
    tc_commit(&G.bar[M1TC + mt]);
}

// The issuing warp of a group (one lane): each staged block's MMAs as their
// operands come, until the group says stop.  A warp of its own, because
// issuing an MMA waits while the tensor pipe's queue is full: issued from a
// warp of the group, that warp's epilogue (and so the group's) started when
// nearly all MMAs were done, and four groups were no faster than three CTAs.
__device__ void tcIssuer(const TcSmem& S, TcGroup& G, uint32_t tmem) {
    uint32_t phase = 0;
    bool ok = true;
    while (ok) {
        ok = bar_wait(&G.in, phase);
        if (!ok || *(volatile int*)&G.stop) break;
        tcIssue1(S, G, tmem);
        // layer 2 of tile mt reads rows up to 46 past the tile's: it follows
        // the epilogues of tiles mt and mt + 1
        ok = bar_wait(&G.act[0], phase);
        for (int mt = 0; mt < M2TC && ok; mt++) {
            ok = bar_wait(&G.act[mt + 1], phase);
            if (ok) tcIssue2(S, G, tmem, mt);
        }
        phase ^= 1u;
    }
    if (!ok) atomicOr(&g_tc_error, 1);
}

// A completion wait of the group gave up: the device error flag, a bounded
// wait for the MMAs in flight (before the CTA's memory goes).
__device__ void tcFail(TcGroup& G, uint32_t phase) {
    for (int k = 0; k < M1TC + M2TC; k++) bar_wait(&G.bar[k], phase);
    if (threadIdx.x % GT == 0) atomicOr(&g_tc_error, 1);
}
// End of a group's blocks (every thread of the group).
__device__ __forceinline__ void tcEnd(TcGroup& G, int g, uint32_t phase, bool ok) {
    if (!groupAnd(g, ok)) tcFail(G, phase ^ 1u);
    if (threadIdx.x % GT == 0) {
        G.stop = 1;
        bar_arrive(&G.in);
    }
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Layer-1 epilogue: this warp's quarter of the rows of M tile mt ->
// relu(acc + b1 - (centre bed - bref) sbed) as BF16 into the activation planes.
__device__ __forceinline__ void tcEpilogue1(const TcSmem& S, TcGroup& G, uint32_t tmem, int mt) {
    const int lg = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
    if (mt * 128 + 32 * lg >= A1C) return;  // (warp-uniform) rows that no output reads
    const int m = mt * 128 + 32 * lg + lane;
    const float cb = G.xbed[min(m, A1C - 1) + 2 * RI + 2] - G.bref;
    float v[32];
    tc_ld32(tmem + ((uint32_t)(32 * lg) << 16) + mt * 32, v);
    if (m < A1C) {
#pragma unroll
        for (int p = 0; p < 4; p++) {  // 8 channels: one plane
            uint32_t q[4];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int o = 8 * p + 4 * e;
                const float4 b = ld4(&S.b1[o]), w = ld4(&S.sbed[o]);
                q[2 * e] = pack2(relu(v[o] + b.x - cb * w.x), relu(v[o + 1] + b.y - cb * w.y));
                q[2 * e + 1] = pack2(relu(v[o + 2] + b.z - cb * w.z), relu(v[o + 3] + b.w - cb * w.w));
            }
            *reinterpret_cast<uint4*>(&G.a1[p][m * 8]) = make_uint4(q[0], q[1], q[2], q[3]);
        }
    }
    proxy_fence();
    tc_before_sync();
}

// The staged block's layer 1 by its group (threads of the group, after their
// barrier): an M tile's epilogue starts as soon as its own MMAs are done.
// False when a wait of this thread's warp gave up.
__device__ __forceinline__ bool tcLayer1(const TcSmem& S, TcGroup& G, uint32_t tmem, uint32_t phase) {
    bool ok = true;
#pragma unroll 1
    for (int mt = 0; mt < M1TC; mt++) {
        ok = __all_sync(0xffffffffu, bar_wait(&G.bar[mt], phase)) && ok;
        tc_after_sync();
        tcEpilogue1(S, G, tmem, mt);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) bar_arrive(&G.act[mt]);
    }
    return ok;
}
// Wait for M tile mt of layer 2.
__device__ __forceinline__ bool tcWait2(TcGroup& G, int mt, uint32_t phase) {
    const bool ok = bar_wait(&G.bar[M1TC + mt], phase);
    tc_after_sync();
    return ok;
}

// Layer-2 epilogue and layer 3 for the row of M tile mt at this thread's
// lane: out = W3 relu(acc + b2) + b3.  Returns the output cell's index in
// the 16 x 16 tile (oy*16 + ox), or -1 for a row that is not an output.
__device__ __forceinline__ int tcOutputs(const TcSmem& S, uint32_t tmem, int mt, float out[COUT]) {
    const int lg = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
    const int m = mt * 128 + 32 * lg + lane, oy = m / RI, ox = m % RI;
#pragma unroll
    for (int c = 0; c < COUT; c++) out[c] = S.b3[c];
    float v[32];
    tc_ld32(tmem + ((uint32_t)(32 * lg) << 16) + mt * 32, v);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float4 b = ld4(&S.b2[4 * q]);
        const float bq[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float a = relu(v[4 * q + k] + bq[k]);
            const float4 w = ld4(S.w3[4 * q + k]);
            out[0] = fmaf(w.x, a, out[0]);
            out[1] = fmaf(w.y, a, out[1]);
            out[2] = fmaf(w.z, a, out[2]);
            out[3] = fmaf(w.w, a, out[3]);
        }
    }
    return (oy >= OT || ox >= OT) ? -1 : oy * OT + ox;
}

// One tcgen05.mma (M 128, N 32, K 16) on fixed BF16 values, with the
// operand layout of the forward pass (K-major, no swizzle, 8-row groups
// 128 bytes apart, the two K chunks LBO bytes apart: 2048 for A, 512 for B),
// and the accumulator read back through tcgen05.ld: out[row * 32 + col] = D.
// A[r][k] = (r % 7) - 3 + (k % 5) / 4, B[n][k] = (n % 5) - 2 + (k % 3) / 2,
// so every product and sum is exact in FP32.  The buffers are larger than
// the operands so that any reading of the two offsets stays inside them.
__global__ void __launch_bounds__(128) k_tc_selftest(float* __restrict__ out) {
    __shared__ __align__(128) uint16_t a[16384];
    __shared__ __align__(128) uint16_t b[1024];
    __shared__ uint64_t bar;
    __shared__ uint32_t tm;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 16384; i += 128) a[i] = 0;
    for (int i = tid; i < 1024; i += 128) b[i] = 0;
    __syncthreads();
    for (int i = tid; i < 128 * 16; i += 128) {
        const int r = i / 16, k = i % 16;
        a[((r / 8) * 128 + (k / 8) * 2048 + (r % 8) * 16) / 2 + k % 8] = bf((r % 7) - 3 + 0.25f * (k % 5));
    }
    for (int i = tid; i < 32 * 16; i += 128) {
        const int n = i / 16, k = i % 16;
        b[((n / 8) * 128 + (k / 8) * 512 + (n % 8) * 16) / 2 + k % 8] = bf((n % 5) - 2 + 0.5f * (k % 3));
    }
    proxy_fence();
    if (tid == 0) bar_init(&bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tm)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = tm;
    if (tid == 0) {
        tc_mma(tmem, sdesc(saddr(a), 2048, 128), sdesc(saddr(b), 512, 128), false);
        tc_commit(&bar);
    }
    const bool ok = __syncthreads_and(bar_wait(&bar, 0));
    if (!ok) {
        bar_wait(&bar, 0);
        if (tid == 0) atomicOr(&g_tc_error, 1);
    }
    tc_after_sync();
    if (ok) {
        float v[32];
        tc_ld32(tmem + ((uint32_t)(32 * warp) << 16), v);
#pragma unroll
        for (int c = 0; c < 32; c++) out[(32 * warp + lane) * 32 + c] = v[c];
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
}

// ------------------------------------------------------------------ forward
// Raw net outputs of every output cell of src.
__global__ void __launch_bounds__(TCT, 1) k_forward(rift_closure_src src, const float* __restrict__ P,
                                                    float* __restrict__ out) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(smem_raw);
    const int g = tcGroupOf(), lane = threadIdx.x & 31;
    TcGroup& T = S.g[g];
    const int ntile = tileCount(src), stride = TCG * (int)gridDim.x;
    int tile = g * (int)gridDim.x + (int)blockIdx.x;
    TcInput R;
    if (threadIdx.x < TCG * GT && tile < ntile) {
        const TileGeom G0 = tileGeom(src, tile);
        tcLoadInput(R, src, G0.s, G0.Y - 3, G0.X - 3);
    }
    tcSetup(S, P);
    const uint32_t tmem = S.tmem + g * TMEM_COLS;
    if (threadIdx.x >= TCG * GT) {
        if (lane == 0) tcIssuer(S, T, tmem);
        __syncwarp();
        tcTeardown(S);
        return;
    }
    uint32_t phase = 0;
    bool ok = true;
    for (; tile < ntile; tile += stride, phase ^= 1u) {
        const TileGeom G = tileGeom(src, tile);
        tcStoreInput(T, R, src);
        if (!groupAnd(g, ok)) break;
        if (threadIdx.x % GT == 0) bar_arrive(&T.in);
        if (tile + stride < ntile) {  // the next block's inputs, during the MMAs
            const TileGeom Gn = tileGeom(src, tile + stride);
            tcLoadInput(R, src, Gn.s, Gn.Y - 3, Gn.X - 3);
        }
        ok = tcLayer1(S, T, tmem, phase);
#pragma unroll 1
        for (int mt = 0; mt < M2TC; mt++) {
            ok = __all_sync(0xffffffffu, tcWait2(T, mt, phase)) && ok;
            float o[COUT];
            const int q = tcOutputs(S, tmem, mt, o);
            if (q < 0 || !ok) continue;
            const int y = G.Y + q / OT - src.oy0, x = G.X + q % OT - src.ox0;
            if (y >= src.OH || x >= src.OW) continue;
#pragma unroll
            for (int c = 0; c < COUT; c++)
                out[(((size_t)G.s * COUT + c) * src.OH + y) * src.OW + x] = o[c];
        }
        tc_before_sync();
    }
    tcEnd(T, g, phase, ok);
    tcTeardown(S);
}

// ----------------------------------------------------------------- training
struct TrainArgs {
    rift_closure_src src;
    const float* P;
    const float* target;
    const float* weight;
    float lossScale;
    float* grad;
    double* loss;
};

// One CTA of 16 warps per SM.  Every contraction is a GEMM on mma.sync whose
// fragments all come by ldmatrix: where an operand lies transposed (the weight
// gradients reduce over cells, the activation gradient over output channels),
// by its .trans form, so nothing is staged twice.  The layer-1 weight gradient
// takes its inputs from the BF16 cells of the forward pass; only the bed, which
// enters relative to each window's centre, is formed again from FP32.
// What bounds it: 256 patches of 70 x 70, 0.56 ms, one CTA per SM: the shared-memory
// pipe is 64% busy with fragments, the tensor pipe 32%, issue 34%; a warp waits
// for shared memory (short scoreboard 3.6 of 11.7 cycles an instruction), fixed
// latencies (2.8) and the barriers between the phases (1.5).
__global__ void __launch_bounds__(TT, 1) k_train(TrainArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
    const rift_closure_src& src = A.src;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // lane addresses of the fragment loads: rows of an A operand, of a
    // transposed A operand, of a transposed B operand
    const int lrow = lane & 15, lk = (lane >> 4) * 8;
    const int tr = (lane & 7) + (lane >> 4) * 8, tc = ((lane >> 3) & 1) * 8;  // A^T: k row, m column
    const int br = (lane & 7) + ((lane >> 3) & 1) * 8, bc = (lane >> 4) * 8;   // B^T: k row, n column
    TrainInput R;
    const int ntile = tileCount(src);
    if ((int)blockIdx.x < ntile) {
        const TileGeom G0 = tileGeom(src, blockIdx.x);
        loadInput(R, src, G0.s, G0.Y - 3, G0.X - 3);
    }
    stageNet(S, A.P);

    // gradient accumulators held across tiles.  Layer 2: row tile `warp` of 18
    // (16 k each) with every column tile, and of tiles 16 and 17 one column
    // tile each on warps 0..7.  Layer 1: over half of the cells, taps 4 p ..
    // 4 p + 3 of the BF16 channels on warp pair p = 0..6, the bed's 25 taps on
    // the last pair; the two row tiles of a warp share their B fragments.
    float gW2[5][4] = {}, gW1[2][4][4] = {};
    const bool bed = warp >= 14;
    const int toff0 = CB * tapCell((warp >> 1) * 4 + (tc >> 3));
    const int toff1 = CB * tapCell((warp >> 1) * 4 + 2 + (tc >> 3));
    float gW3 = 0.f, gB3[COUT] = {}, gB2 = 0.f, gB1 = 0.f;
    double lossAcc = 0.0;
    const int mtX = 16 + ((warp >> 2) & 1), ntX = warp & 3;  // the extra layer-2 tile

    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const TileGeom G = tileGeom(src, tile);
        __syncthreads();
        storeInput(S, R, src);
        if (tile + (int)gridDim.x < ntile) {
            const TileGeom Gn = tileGeom(src, tile + gridDim.x);
            loadInput(R, src, Gn.s, Gn.Y - 3, Gn.X - 3);
        }
        __syncthreads();
        conv1(S, warp, lane);
        __syncthreads();
        {
            float z2[4][4], o[4];
            conv23(S, warp, lane, z2, o);
            // loss and d loss / d out; layer-2 activations to shared memory
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int ox = g + 8 * r, p = warp * OT + ox;
                if (t < 2) {
                    const int y = G.Y + warp - src.oy0, x = G.X + ox - src.ox0;
                    const bool in = y < src.OH && x < src.OW;
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int ch = 2 * t + e;
                        float d = 0.f;
                        if (in) {
                            size_t at = (((size_t)G.s * COUT + ch) * src.OH + y) * src.OW + x;
                            float w = __ldg(A.weight + at);
                            float diff = o[2 * r + e] - __ldg(A.target + at);
                            lossAcc += (double)(w * diff * diff);
                            d = 2.f * w * diff * A.lossScale;
                        }
                        S.dout[p * 4 + ch] = d;
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 4; nt++)
                    st32(&S.a2[p * SA + nt * 8 + 2 * t], pack2(relu(z2[nt][2 * r]), relu(z2[nt][2 * r + 1])));
            }
        }
        __syncthreads();
        // layer 3: dW3, db3 (CUDA cores)
        {
            const int oc = (tid >> 5) & 3, c = lane, part = tid >> 7;
            float acc = 0.f;
#pragma unroll 8
            for (int p = part * 64; p < part * 64 + 64; p++) acc += S.dout[p * 4 + oc] * fb(S.a2[p * SA + c]);
            gW3 += acc;
            if (tid < OT * OT) {
                const float4 d = *reinterpret_cast<const float4*>(&S.dout[tid * 4]);
                float v[COUT] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int k = 0; k < COUT; k++) {
                    for (int s = 16; s > 0; s >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], s);
                    gB3[k] += v[k];
                }
            }
        }
        __syncthreads();
        // dZ2 = (W3^T dout) * relu'(z2), in place of a2: 16 channels per thread
        {
            const int p = tid >> 1, c0 = (tid & 1) * 16;
            const float4 d = *reinterpret_cast<const float4*>(&S.dout[p * 4]);
            uint4* z = reinterpret_cast<uint4*>(&S.a2[p * SA + c0]);
            uint32_t q[8];
            *reinterpret_cast<uint4*>(&q[0]) = z[0];
            *reinterpret_cast<uint4*>(&q[4]) = z[1];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                float v[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float4 w = *reinterpret_cast<const float4*>(S.w3q[c0 + 2 * k + e]);
                    const float a = fb((uint16_t)(q[k] >> (16 * e)));
                    const float x = d.x * w.x + d.y * w.y + d.z * w.z + d.w * w.w;
                    v[e] = a > 0.f ? x : 0.f;
                }
                q[k] = pack2(v[0], v[1]);
            }
            z[0] = *reinterpret_cast<uint4*>(&q[0]);
            z[1] = *reinterpret_cast<uint4*>(&q[4]);
        }
        __syncthreads();
        {
            float b = 0.f;
#pragma unroll 8
            for (int p = warp; p < OT * OT; p += TT / 32) b += fb(S.a2[p * SA + lane]);
            gB2 += b;
        }
        // dW2[k][o] += sum_p a1[p + tap(k)][ch(k)] dZ2[p][o]
        {
            const int tap = warp >> 1, tapX = mtX >> 1;
            const uint16_t* pa = &S.a1[((tap / 3) * R1 + tap % 3 + tr) * SA + (warp & 1) * 16 + tc];
            const uint16_t* px = &S.a1[((tapX / 3) * R1 + tapX % 3 + tr) * SA + (mtX & 1) * 16 + tc];
            const uint16_t* pb = &S.a2[br * SA + bc];
#pragma unroll 4
            for (int oyp = 0; oyp < OT; oyp++) {
                uint32_t a[4], b0[4], b1[4];
                ldsm4t(b0, pb + oyp * OT * SA);
                ldsm4t(b1, pb + oyp * OT * SA + 16);
                ldsm4t(a, pa + oyp * R1 * SA);
                mma16816(gW2[0], a, b0[0], b0[1]);
                mma16816(gW2[1], a, b0[2], b0[3]);
                mma16816(gW2[2], a, b1[0], b1[1]);
                mma16816(gW2[3], a, b1[2], b1[3]);
                if (warp < 8) {
                    ldsm4t(a, px + oyp * R1 * SA);
                    const uint32_t x0 = ntX & 2 ? (ntX & 1 ? b1[2] : b1[0]) : (ntX & 1 ? b0[2] : b0[0]);
                    const uint32_t x1 = ntX & 2 ? (ntX & 1 ? b1[3] : b1[1]) : (ntX & 1 ? b0[3] : b0[1]);
                    mma16816(gW2[4], a, x0, x1);
                }
            }
        }
        __syncthreads();
        // dA1[q][c] = sum_{tap,o} dZ2[q - tap][o] W2[o][tap*32 + c]; dZ1 = dA1 * relu'(z1),
        // written over a1 (each element read and written by the same thread)
        {
            const int half = warp & 1, mt0 = warp >> 1;
            int qy[UPW], qx[UPW];
#pragma unroll
            for (int j = 0; j < UPW; j++) {
                const int q = (mt0 + WPH * j) * 16 + lrow;
                qy[j] = q < NR1 ? q / R1 : -OT;  // (a row past the region: outside for every tap)
                qx[j] = q % R1;
            }
            const uint16_t* wp = &S.w2[br * SW2 + half * 16 + bc];
            float acc[UPW][2][4] = {};
#pragma unroll 3
            for (int tap = 0; tap < 9; tap++) {
                const int dy = tap / 3, dx = tap % 3;
                uint32_t b[2][4];
                ldsm4t(b[0], wp + tap * 32);
                ldsm4t(b[1], wp + 16 * SW2 + tap * 32);
#pragma unroll
                for (int j = 0; j < UPW; j++) {
                    if (mt0 + WPH * j >= M1T) break;
                    const int py = qy[j] - dy, px = qx[j] - dx;
                    const bool in = (unsigned)py < (unsigned)OT && (unsigned)px < (unsigned)OT;
                    const uint16_t* d = (in ? &S.a2[(py * OT + px) * SA] : S.zero) + lk;
#pragma unroll
                    for (int ob = 0; ob < 2; ob++) {
                        uint32_t a[4];
                        ldsm4(a, d + ob * 16);
                        mma16816(acc[j][0], a, b[ob][0], b[ob][1]);
                        mma16816(acc[j][1], a, b[ob][2], b[ob][3]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < UPW; j++) {
                if (mt0 + WPH * j >= M1T) break;
                const int q0 = (mt0 + WPH * j) * 16 + g, q1 = q0 + 8;
#pragma unroll
                for (int nt = 0; nt < 2; nt++) {
                    const int c = half * 16 + nt * 8 + 2 * t;
                    if (q0 < NR1) {
                        uint16_t* z = &S.a1[q0 * SA + c];
                        st32(z, pack2(fb(z[0]) > 0.f ? acc[j][nt][0] : 0.f, fb(z[1]) > 0.f ? acc[j][nt][1] : 0.f));
                    }
                    if (q1 < NR1) {
                        uint16_t* z = &S.a1[q1 * SA + c];
                        st32(z, pack2(fb(z[0]) > 0.f ? acc[j][nt][2] : 0.f, fb(z[1]) > 0.f ? acc[j][nt][3] : 0.f));
                    }
                }
            }
        }
        __syncthreads();
        {
            float b = 0.f;
#pragma unroll 4
            for (int q = warp; q < NR1; q += TT / 32) b += fb(S.a1[q * SA + lane]);
            gB1 += b;
        }
        // dW1[k][o] += sum_q x(q, k) dZ1[q][o]
#pragma unroll 2
        for (int ks = warp & 1; ks < M1T; ks += 2) {
            uint32_t a[2][4], b0[4], b1[4];
            const int qb = ks * 16 + br;
            const uint16_t* pb = (qb < NR1 ? &S.a1[qb * SA] : S.zero) + bc;
            ldsm4t(b0, pb);
            ldsm4t(b1, pb + 16);
            if (!bed) {
                const uint16_t* px = &S.xb[S.qcell[ks * 16 + tr] * CB];
                ldsm4t(a[0], px + toff0);
                ldsm4t(a[1], px + toff1);
            } else {
                float x[4][4];  // this thread's taps g, g + 8, g + 16 and g + 24
#pragma unroll
                for (int u = 0; u < 4; u++) {  // cells 2t, 2t + 1, 2t + 8, 2t + 9
                    const int cell = S.qcell[ks * 16 + 2 * t + (u & 1) + 8 * (u >> 1)];
                    const float mid = S.xbed[cell + 2 * RI + 2];
#pragma unroll
                    for (int r = 0; r < 3; r++) x[r][u] = S.xbed[cell + S.toff[g + 8 * r]] - mid;
                    x[3][u] = g == 0 ? S.xbed[cell + 4 * RI + 4] - mid : 0.f;
                }
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    a[m][0] = pack2(x[2 * m][0], x[2 * m][1]);
                    a[m][1] = pack2(x[2 * m + 1][0], x[2 * m + 1][1]);
                    a[m][2] = pack2(x[2 * m][2], x[2 * m][3]);
                    a[m][3] = pack2(x[2 * m + 1][2], x[2 * m + 1][3]);
                }
            }
#pragma unroll
            for (int m = 0; m < 2; m++) {
                mma16816(gW1[m][0], a[m], b0[0], b0[1]);
                mma16816(gW1[m][1], a[m], b0[2], b0[3]);
                mma16816(gW1[m][2], a[m], b1[0], b1[1]);
                mma16816(gW1[m][3], a[m], b1[2], b1[3]);
            }
        }
    }

    // one addition per CTA of every gradient it holds
#pragma unroll
    for (int j = 0; j < 5; j++) {
        if (j == 4 && warp >= 8) break;
        const int mt = j < 4 ? warp : mtX, nt = j < 4 ? j : ntX;
        const int k0 = mt * 16 + g, o0 = nt * 8 + 2 * t;
        atomicAdd(&A.grad[OFF_W2 + o0 * K2 + k0], gW2[j][0]);
        atomicAdd(&A.grad[OFF_W2 + (o0 + 1) * K2 + k0], gW2[j][1]);
        atomicAdd(&A.grad[OFF_W2 + o0 * K2 + k0 + 8], gW2[j][2]);
        atomicAdd(&A.grad[OFF_W2 + (o0 + 1) * K2 + k0 + 8], gW2[j][3]);
    }
    {
        // the two rows of a fragment: channel g of two taps (h, hu, hv, -, -, n,
        // rain, -), or the bed of two taps
        const int c = bed ? 3 : g < 3 ? g : g == 5 ? 4 : g == 6 ? 5 : -1;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int tap = bed ? g + 8 * r : (warp >> 1) * 4 + r;
            if (c < 0 || tap >= 25) continue;
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
                const int o0 = nt * 8 + 2 * t, k = tap * CIN + c;
                atomicAdd(&A.grad[OFF_W1 + o0 * K1P + k], gW1[r >> 1][nt][2 * (r & 1)]);
                atomicAdd(&A.grad[OFF_W1 + (o0 + 1) * K1P + k], gW1[r >> 1][nt][2 * (r & 1) + 1]);
            }
        }
    }
    atomicAdd(&A.grad[OFF_W3 + (tid & 127)], gW3);
    if (tid < OT * OT && lane == 0)
        for (int k = 0; k < COUT; k++) atomicAdd(&A.grad[OFF_B3 + k], gB3[k]);
    atomicAdd(&A.grad[OFF_B2 + lane], gB2);
    atomicAdd(&A.grad[OFF_B1 + lane], gB1);
    // loss: warp sums, then one atomic per CTA
    for (int s = 16; s > 0; s >>= 1) lossAcc += __shfl_xor_sync(0xffffffffu, lossAcc, s);
    if (lane == 0) S.red[warp] = lossAcc;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < TT / 32; w++) s += S.red[w];
        atomicAdd(A.loss, s * (double)A.lossScale);
    }
}

// --------------------------------------------------------------------- Adam
__global__ void k_adam(float* __restrict__ p, float* __restrict__ gr, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps,
                       float bias1, float bias2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float gi = gr[i];
        float mi = b1 * m[i] + (1.f - b1) * gi;
        float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / bias1) / (sqrtf(vi / bias2) + eps);
        gr[i] = 0.f;
    }
}

// ------------------------------------------------------------ face fluxes
// Central-upwind flux through the east (DIR 0) or north (DIR 1) face of
// cell (j, i) of a handle's U^n, built as the step builds it: the
// reconstruction of both cells (construct) and the face flux (faceFlux).
template <int DIR>
__device__ __forceinline__ void faceFluxAt(const rift_device_view& V, int j, int i, float f[3]) {
    const size_t pitch = (size_t)V.pitch, pl = (size_t)V.rows * pitch;
    const int sj = DIR ? 1 : 0, si = DIR ? 0 : 1;
    auto at = [&](const float* P, int jj, int ii) { return __ldg(P + (size_t)jj * pitch + ii); };
    const float* eM = V.e + (DIR ? 2 : 0) * pl;  // eW / eS
    const float* eP = V.e + (DIR ? 3 : 1) * pl;  // eE / eN
    float hh[4], uu[4], vv[4], em[4], ep[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {  // cells -1 .. +2 along DIR
        const int jj = j + (k - 1) * sj, ii = i + (k - 1) * si;
        hh[k] = at(V.h, jj, ii);
        uu[k] = at(V.hu, jj, ii);
        vv[k] = at(V.hv, jj, ii);
        em[k] = at(eM, jj, ii);
        ep[k] = at(eP, jj, ii);
    }
    const float kappa = (float)V.kappa;
    rift::Rec L = rift::construct(hh[1], uu[1], vv[1], hh[2], uu[2], vv[2], hh[0], uu[0], vv[0], em[1],
                                  ep[1], ep[1] - em[2], ep[0] - em[1]);
    rift::Rec R = rift::construct(hh[2], uu[2], vv[2], hh[3], uu[3], vv[3], hh[1], uu[1], vv[1], em[2],
                                  ep[2], ep[2] - em[3], ep[1] - em[2]);
    rift::faceFlux<DIR>(L.hP, L.uP, L.vP, R.hM, R.uM, R.vM, kappa, f);
}

__global__ void k_faceflux(rift_device_view V, int ratio, float w, float* __restrict__ acc,
                           int apitch, int arows, int anx, int any) {
    const int I = 2 + blockIdx.x * blockDim.x + threadIdx.x;
    const int J = 2 + blockIdx.y * blockDim.y + threadIdx.y;
    if (I > anx - 3 || J > any - 3) return;
    const size_t pl = (size_t)arows * apitch, c = (size_t)J * apitch + I;
    float fe[3], fn[3];
    float e0, e1, n0, n2;
    if (ratio == 1) {
        faceFluxAt<0>(V, J, I, fe);
        faceFluxAt<1>(V, J, I, fn);
        e0 = fe[0], e1 = fe[1], n0 = fn[0], n2 = fn[2];
    } else {
        const int jf = 2 * (J - 2) + 2, jf2 = jf + 1, i0 = 2 * (I - 2) + 2;
        float fa[3], fb2[3];
        faceFluxAt<0>(V, jf, i0 + 1, fa);
        faceFluxAt<0>(V, jf2, i0 + 1, fb2);
        e0 = 0.5f * (fa[0] + fb2[0]);
        e1 = 0.5f * (fa[1] + fb2[1]);
        faceFluxAt<1>(V, jf2, i0, fa);
        faceFluxAt<1>(V, jf2, i0 + 1, fb2);
        n0 = 0.5f * (fa[0] + fb2[0]);
        n2 = 0.5f * (fa[2] + fb2[2]);
    }
    acc[c] += w * e0;
    acc[pl + c] += w * e1;
    acc[2 * pl + c] += w * n0;
    acc[3 * pl + c] += w * n2;
}

// ----------------------------------------------------------- closure step
struct ApplyArgs {
    rift_closure_src src;
    const float* P;
    float osc[4];
    float* corr;
    size_t plane;
    int pitch, nx, ny;
    float dtw, inv_dx, inv_dy, hmin, lim, tau;
    int* ticket;    // blocks drawn so far (zero at the launch)
    uint8_t* fell;  // per 16 x 16 block: 1 when it fell back to the plain solve
    int* counters;
};

// Net outputs -> gated, limited face corrections of every 16 x 16 block of
// interior cells (zeros for dry blocks and blocks that fall back).
// The groups draw their blocks from a ticket (dry blocks cost next to nothing,
// and water lies in patches: with fixed shares an SM held up to 1.4 times the
// mean of the wet ones).  A leader draws two blocks ahead, so no one waits for
// the ticket.
__global__ void __launch_bounds__(TCT, 1) k_closure(ApplyArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(smem_raw);
    const rift_closure_src& src = A.src;
    const int g = tcGroupOf(), tid = threadIdx.x % GT, lane = tid & 31;
    TcGroup& T = S.g[g];
    const float hminS = A.hmin * src.scale[0], invS0 = 1.f / src.scale[0];
    const int ntile = tileCount(src), first = TCG * (int)gridDim.x;
    int tile = g * (int)gridDim.x + (int)blockIdx.x, next = 0;
    int drawn = 0;  // leader: the ticket after the next
    if (threadIdx.x < TCG * GT && tid == 0) drawn = first + atomicAdd(A.ticket, 1);
    TcInput R;
    if (threadIdx.x < TCG * GT && tile < ntile) {
        const TileGeom G0 = tileGeom(src, tile);
        tcLoadInput(R, src, 0, G0.Y - 3, G0.X - 3);
    }
    tcSetup(S, A.P);
    const uint32_t tmem = S.tmem + g * TMEM_COLS;
    if (threadIdx.x >= TCG * GT) {
        if (lane == 0) tcIssuer(S, T, tmem);
        __syncwarp();
        tcTeardown(S);
        return;
    }
    uint32_t phase = 0;
    bool ok = true;
    for (; tile < ntile; tile = next) {
        const TileGeom G = tileGeom(src, tile);
        if (tid == 0) {
            T.red = 0;
            T.next = drawn;
            drawn = first + atomicAdd(A.ticket, 1);
        }
        tcStoreInput(T, R, src);
        if (!groupAnd(g, ok)) break;
        // T.next is read between the block's first two barriers: after the first
        // it is written, and after the second the leader may write it again (a
        // dry block has no barrier after that one)
        next = T.next;
        bool dry = true;
        for (int i = tid; i < (OT + 1) * (OT + 1); i += GT) {
            int ry = 3 + i / (OT + 1), rx = 3 + i % (OT + 1);
            dry &= !(T.xh[ry * RI + rx] > hminS);
        }
        dry = groupAnd(g, dry);
        if (tid == 0 && !dry) bar_arrive(&T.in);
        if (next < ntile) {  // the next block's inputs, in flight meanwhile
            const TileGeom Gn = tileGeom(src, next);
            tcLoadInput(R, src, 0, Gn.Y - 3, Gn.X - 3);
        }
        if (dry) {
            if (tid == 0) A.fell[tile] = 0;
            for (int i = tid; i < OT * OT; i += GT) {
                int y = G.Y + i / OT, x = G.X + i % OT;
                if (y - src.oy0 >= src.OH || x - src.ox0 >= src.OW) continue;
                size_t c = (size_t)y * A.pitch + x;
#pragma unroll
                for (int ch = 0; ch < 4; ch++) A.corr[ch * A.plane + c] = 0.f;
            }
            continue;
        }
        ok = tcLayer1(S, T, tmem, phase);
        // this thread's output cells (up to three) and their four corrections:
        // east-face mass and momentum, north-face mass and momentum
        int cell[M2TC] = {-1, -1, -1};
        float cv[M2TC][4] = {};
        float ind = 0.f;
#pragma unroll
        for (int k = 0; k < M2TC; k++) {
            ok = __all_sync(0xffffffffu, tcWait2(T, k, phase)) && ok;
            float o[COUT];
            const int q = tcOutputs(S, tmem, k, o);
            if (q < 0 || !ok) continue;
            const int oy = q / OT, ox = q % OT, y = G.Y + oy, x = G.X + ox;
            if (y - src.oy0 >= src.OH || x - src.ox0 >= src.OW) continue;
            cell[k] = q;
            const float hc = T.xh[(oy + 3) * RI + ox + 3] * invS0;
#pragma unroll
            for (int f = 0; f < 2; f++) {
                const bool east = f == 0;
                const float inv = east ? A.inv_dx : A.inv_dy;
                const int yn = east ? y : y + 1, xn = east ? x + 1 : x;
                const float hn = T.xh[(oy + 3 + (east ? 0 : 1)) * RI + ox + 3 + (east ? 1 : 0)] * invS0;
                const bool ok = x >= 3 && y >= 3 && xn <= A.nx - 4 && yn <= A.ny - 4 && hc > A.hmin &&
                                hn > A.hmin;
                float vm = ok ? o[2 * f] * A.osc[2 * f] : 0.f;
                const float vq = ok ? o[2 * f + 1] * A.osc[2 * f + 1] : 0.f;
                const float hd = vm > 0.f ? hc : hn;
                if (ok) {
                    ind = fmaxf(ind, fabsf(vm) * A.dtw * inv / hd);
                    const float cap = A.lim * hd / (A.dtw * inv);
                    vm = fminf(fmaxf(vm, -cap), cap);
                }
                cv[k][2 * f] = vm;
                cv[k][2 * f + 1] = vq;
            }
        }
        tc_before_sync();
        for (int s = 16; s > 0; s >>= 1) ind = fmaxf(ind, __shfl_xor_sync(0xffffffffu, ind, s));
        if (lane == 0) atomicMax(&T.red, __float_as_int(ind));
        groupSync(g);
        const bool fallback = __int_as_float(T.red) > A.tau;
#pragma unroll
        for (int k = 0; k < M2TC; k++) {
            if (cell[k] < 0) continue;
            const size_t c = (size_t)(G.Y + cell[k] / OT) * A.pitch + G.X + cell[k] % OT;
#pragma unroll
            for (int ch = 0; ch < 4; ch++) A.corr[ch * A.plane + c] = fallback ? 0.f : cv[k][ch];
        }
        if (tid == 0) {
            A.fell[tile] = fallback ? 1 : 0;
            atomicAdd(&A.counters[0], 1);
            if (fallback) atomicAdd(&A.counters[1], 1);
        }
        groupSync(g);  // red is read before the next block clears it
        phase ^= 1u;
    }
    tcEnd(T, g, phase, ok);
    tcTeardown(S);
}

// U^n -= dtw x divergence of the face corrections (cells one inside the
// ghost ring and beyond).  A face is corrected only when neither of the
// 16 x 16 blocks of its two cells fell back: both cells then see the same
// correction (mass stays conserved) and every cell of a fallen-back block
// keeps the plain solve exactly.
// (Loads first, tests after: behind the tests each load waited for the last,
// 17 us on 1024^2 cells.)
__global__ void k_apply(float* __restrict__ h, float* __restrict__ hu, float* __restrict__ hv,
                        float* __restrict__ corr, const uint8_t* __restrict__ fell, size_t plane,
                        int pitch, int nx, int ny, float sx, float sy) {
    const int i = 3 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 3 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i == 3 && j == 3) corr[0] = 0.f;  // k_closure's ticket (a corner of the ghost ring)
    if (i > nx - 4 || j > ny - 4) return;
    const size_t c = (size_t)j * pitch + i;
    const float cE = corr[c], cW = corr[c - 1], dE = corr[plane + c], dW = corr[plane + c - 1];
    const float cN = corr[2 * plane + c], cS = corr[2 * plane + c - pitch];
    const float dN = corr[3 * plane + c], dS = corr[3 * plane + c - pitch];
    const float h0 = h[c], u0 = hu[c], v0 = hv[c];
    const int tx = (nx - 4 + OT - 1) / OT;
    const int bx = (i - 2) / OT, by = (j - 2) / OT, b = by * tx + bx;
    const bool w = (i - 2) % OT == 0, e = (i - 1) % OT == 0 && i + 1 <= nx - 3;
    const bool s = (j - 2) % OT == 0, n = (j - 1) % OT == 0 && j + 1 <= ny - 3;
    // (i, j >= 3: a cell on its block's west or south side has a block there)
    const bool own = fell[b] != 0, fW = fell[w ? b - 1 : b], fE = fell[e ? b + 1 : b];
    const bool fS = fell[s ? b - tx : b], fN = fell[n ? b + tx : b];
    // a tensor-core wait of k_closure gave up: some blocks' corrections were
    // not written, so the whole step keeps the plain solve
    const bool failed = *(volatile int*)&g_tc_error != 0;
    if (own || failed) return;  // own: every face of this cell touches its own block
    const float mE = fE ? 0.f : cE, mW = fW ? 0.f : cW, mN = fN ? 0.f : cN, mS = fS ? 0.f : cS;
    const float uE = fE ? 0.f : dE, uW = fW ? 0.f : dW, vN = fN ? 0.f : dN, vS = fS ? 0.f : dS;
    if (mE == 0.f && mW == 0.f && mN == 0.f && mS == 0.f && uE == 0.f && uW == 0.f && vN == 0.f &&
        vS == 0.f)
        return;
    h[c] = h0 - (sx * (mE - mW) + sy * (mN - mS));
    hu[c] = u0 - sx * (uE - uW);
    hv[c] = v0 - sy * (vN - vS);
}

}  // namespace rc

// ------------------------------------------------------------------- C ABI
namespace {
thread_local std::string g_err;

int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

int launched(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(RIFT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    return RIFT_OK;
}

bool srcOk(const rift_closure_src* s) {
    return s && s->samples >= 1 && s->H >= 1 && s->W >= 1 && s->pitch >= s->W && s->OH >= 1 &&
           s->OW >= 1 && s->oy0 >= 0 && s->ox0 >= 0 && s->sample_stride >= 0 &&
           (s->samples == 1 || s->sample_stride >= (int64_t)s->pitch * s->H);
}

// CTAs of kernel k with `smem` bytes: one per SM, capped by the tile count.
int onePerSM(const void* k, size_t smem, int tiles, int* out) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return fail(RIFT_ERR_CUDA, "no device");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(RIFT_ERR_CUDA, cudaGetErrorString(e));
    *out = tiles < sms ? tiles : sms;
    return RIFT_OK;
}
}  // namespace

extern "C" {

int rift_closure_forward(const rift_closure_src* src, const float* params, float* out, void* stream) {
    if (!srcOk(src) || !params || !out) return fail(RIFT_ERR_ARG, "rift_closure_forward: bad argument");
    const size_t smem = sizeof(rc::TcSmem);
    const int tiles = rc::tileCount(*src);
    int grid = 0, rc_;
    if ((rc_ = onePerSM((const void*)rc::k_forward, smem, tiles, &grid))) return rc_;
    rc::k_forward<<<grid, rc::TCT, smem, (cudaStream_t)stream>>>(*src, params, out);
    return launched("k_forward");
}

int rift_closure_train(const rift_closure_src* src, const float* params, const float* target,
                       const float* weight, float loss_scale, float* grad, double* loss, void* stream) {
    if (!srcOk(src) || !params || !target || !weight || !grad || !loss)
        return fail(RIFT_ERR_ARG, "rift_closure_train: bad argument");
    const size_t smem = sizeof(rc::TrainSmem);
    const int tiles = rc::tileCount(*src);
    int grid = 0, rc_;
    if ((rc_ = onePerSM((const void*)rc::k_train, smem, tiles, &grid))) return rc_;
    rc::TrainArgs A{*src, params, target, weight, loss_scale, grad, loss};
    rc::k_train<<<grid, rc::TT, smem, (cudaStream_t)stream>>>(A);
    return launched("k_train");
}

int rift_closure_adam(float* params, float* grad, float* m, float* v, int32_t n, float lr, float beta1,
                      float beta2, float eps, float bias1, float bias2, void* stream) {
    if (!params || !grad || !m || !v || n < 1 || !(bias1 > 0.f) || !(bias2 > 0.f))
        return fail(RIFT_ERR_ARG, "rift_closure_adam: bad argument");
    const int blocks = (n + 255) / 256;
    rc::k_adam<<<blocks, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, n, lr, beta1, beta2, eps,
                                                         bias1, bias2);
    return launched("k_adam");
}

int rift_closure_face_flux(const rift_device_view* view, int32_t ratio, float weight, float* acc,
                           int32_t acc_pitch, int32_t acc_rows, int32_t acc_nx, int32_t acc_ny) {
    if (!view || !acc || (ratio != 1 && ratio != 2) || acc_nx < 5 || acc_ny < 5 || acc_pitch < acc_nx ||
        acc_rows < acc_ny)
        return fail(RIFT_ERR_ARG, "rift_closure_face_flux: bad argument");
    if (view->h_nx - 4 != ratio * (acc_nx - 4) || view->h_ny - 4 != ratio * (acc_ny - 4))
        return fail(RIFT_ERR_ARG, "rift_closure_face_flux: grids do not match the ratio");
    dim3 blk(32, 8), grd((acc_nx - 4 + 31) / 32, (acc_ny - 4 + 7) / 8);
    rc::k_faceflux<<<grd, blk, 0, (cudaStream_t)view->stream>>>(*view, ratio, weight, acc, acc_pitch,
                                                                 acc_rows, acc_nx, acc_ny);
    return launched("k_faceflux");
}

int rift_closure_apply(const rift_device_view* view, const rift_closure_src* src, const float* params,
                       const float* oscale_host, float dtw, float hmin, float lim, float tau, float* corr,
                       uint8_t* block_fell, int32_t* counters) {
    if (!view || !srcOk(src) || !params || !oscale_host || !corr || !block_fell || !counters ||
        !(hmin > 0.f) || !(lim > 0.f) || !(src->scale[0] > 0.f) || src->samples != 1)
        return fail(RIFT_ERR_ARG, "rift_closure_apply: bad argument");
    // Each of a cell's four faces may carry up to lim x its depth out of it:
    // a cell deeper than hmin keeps at least hmin (1 - 4 lim), which must stay
    // above the wet threshold so that no wet cell is dried.
    if (!(lim < 0.25f) || !(hmin * (1.f - 4.f * lim) > 1.19209e-07f))
        return fail(RIFT_ERR_ARG, "rift_closure_apply: lim must be < 0.25 and hmin (1 - 4 lim) > 1.19e-7 m");
    if (src->H != view->h_ny || src->W != view->h_nx || src->pitch != view->pitch || src->oy0 != 2 ||
        src->ox0 != 2 || src->OH != view->h_ny - 4 || src->OW != view->h_nx - 4)
        return fail(RIFT_ERR_ARG, "rift_closure_apply: src is not the view's interior");
    if (!(dtw > 0.f)) return RIFT_OK;
    cudaStream_t st = (cudaStream_t)view->stream;
    rc::ApplyArgs A{};
    A.src = *src;
    A.P = params;
    for (int c = 0; c < 4; c++) A.osc[c] = oscale_host[c];
    A.corr = corr;
    A.plane = (size_t)view->rows * view->pitch;
    A.pitch = view->pitch;
    A.nx = view->h_nx;
    A.ny = view->h_ny;
    A.dtw = dtw;
    A.inv_dx = (float)(1.0 / view->dx);
    A.inv_dy = (float)(1.0 / view->dy);
    A.hmin = hmin;
    A.lim = lim;
    A.tau = tau;
    A.fell = block_fell;
    A.counters = counters;
    const size_t smem = sizeof(rc::TcSmem);
    const int tiles = rc::tileCount(*src);
    int grid = 0, rc_;
    if ((rc_ = onePerSM((const void*)rc::k_closure, smem, tiles, &grid))) return rc_;
    // the blocks' ticket: a corner of the ghost ring of corr, which holds no correction
    A.ticket = reinterpret_cast<int*>(corr);
    if (cudaMemsetAsync(A.ticket, 0, sizeof(int), st) != cudaSuccess) return launched("ticket");
    rc::k_closure<<<grid, rc::TCT, smem, st>>>(A);
    if ((rc_ = launched("k_closure"))) return rc_;
    dim3 blk(32, 8), grd((view->h_nx - 6 + 31) / 32, (view->h_ny - 6 + 7) / 8);
    rc::k_apply<<<grd, blk, 0, st>>>(view->h, view->hu, view->hv, corr, block_fell, A.plane, view->pitch,
                                     view->h_nx, view->h_ny, (float)(dtw / view->dx), (float)(dtw / view->dy));
    return launched("k_apply");
}

int rift_closure_selftest(float* out, void* stream) {
    if (!out) return fail(RIFT_ERR_ARG, "rift_closure_selftest: bad argument");
    rc::k_tc_selftest<<<1, 128, 0, (cudaStream_t)stream>>>(out);
    return launched("k_tc_selftest");
}

int rift_closure_check(void* stream) {
    // one copy on the stream and one wait; the flag is written back only when it was set
    const cudaStream_t st = (cudaStream_t)stream;
    int flag = 0;
    const int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&flag, rc::g_tc_error, sizeof(int), 0, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(RIFT_ERR_CUDA, std::string("rift_closure_check: ") + cudaGetErrorString(e));
    if (flag && cudaMemcpyToSymbol(rc::g_tc_error, &zero, sizeof(int)) != cudaSuccess)
        return fail(RIFT_ERR_CUDA, "rift_closure_check: status reset failed");
    if (flag) return fail(RIFT_ERR_CUDA, "rift_closure_check: a tensor-core completion wait gave up");
    return RIFT_OK;
}

const char* rift_closure_last_error(void) { return g_err.c_str(); }

}  // extern "C"
