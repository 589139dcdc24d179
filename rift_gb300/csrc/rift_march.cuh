// rift_march.cuh -- the two flux passes of a step as a column march by warps.
//
// Work item: 60 columns x `itemRows` rows of the grid, walked row by row by
// one warp with no CTA barrier.  Lane l holds the two
// columns 60 s + 2l and 60 s + 2l + 1 of segment s as a pair, so the
// arithmetic runs on the packed FP32 instructions (rift_pair.cuh); lanes 1..30
// own their columns, lanes 0 and 31 supply the x halo (4 of 64 columns).
// Per row:
//   - the y reconstruction of the row above and the flux through the row's
//     north face come from registers rolled down the columns;
//   - the differences to the east are formed once per face: the west ones are
//     the neighbour's, one shuffle each, and the west-face flux is the
//     neighbour's east-face flux (13 shuffles for two cells);
//   - the cell update is the same arithmetic as grid.cu's Integrate kernels.
// Rows arrive through TMA in chunks of two rows of 64 columns, a ring of
// three chunks per warp: two hold the three rows a step of the march reads,
// the third is in flight during two rows.  The cell's own values (stage 2:
// U^n, maps, infiltration) are loaded at the start of its row; on grids
// larger than L2 one prefetch instruction per row asks for them MPF rows
// ahead (lane q takes one 128-byte line).
// A cell is updated only when its reference tile is active, so results and
// tile flags are those of the per-tile schedule of the reference.
//
// Stage 1 needs dt, and dt needs the speeds of stage 1's own fluxes (the
// first ComputeFluxes of the step).  So the stage-1 march computes the
// fluxes, the speed maxima and dt (last CTA), and stores each cell's flux
// divergence with the bed-slope source folded in (3 words); k_update1
// (rift_update1.cuh) then applies the rest of Integrate_1_k.  The step does
// one flux pass per stage and no separate speed pass.
//
// What bounds it: on 4096^2 cells of urban rain the passes issue 201 and 292
// lane instructions per cell (397 and 505 with one column per lane, a CTA of
// four warps in step and scalar arithmetic) and take 154 and 226 us (219 and
// 294); they issue on 60% of cycles, the packed instructions' FMA pipe is 60%
// busy, DRAM moves at 4.6 and 5.0 TB/s.  A lone warp needs 0.56 us per row.
#pragma once
#include "rift_grow.cuh"

namespace rift {

constexpr int MW = 4;                  // warps per CTA
constexpr int MT = MW * 32;            // threads per CTA
constexpr int MCOLS = STRIP_TX * TW;   // columns of the grow's strips (112)
constexpr int MSEG = SEG;              // columns a warp owns
constexpr int MBOX = 64;               // columns a warp stages
constexpr int MCR = 2;                 // rows per staged chunk
constexpr int MNS = 3;                 // chunks in a warp's ring
constexpr int MPF = 5;                 // rows ahead of the L2 prefetch of the centre values
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ P2 ld2(const float* p) {
    return P2{*reinterpret_cast<const unsigned long long*>(p)};
}
__device__ __forceinline__ void st2(float* p, P2 a) {
    *reinterpret_cast<unsigned long long*>(p) = a.v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// A warp's ring of staged rows: chunks of two rows of 64 columns of h, hu, hv
// (one TMA copy) and of the four face offsets (another).
struct __align__(128) MarchSlot {
    float s[3][MCR][MBOX];
    float e[4][MCR][MBOX];
};
static_assert(sizeof(MarchSlot) % 128 == 0 && offsetof(MarchSlot, e) % 128 == 0,
              "TMA destination alignment");
struct __align__(128) MarchRing {
    MarchSlot slot[MNS];
    uint64_t bar[MNS];
};
// Plane p (0..2 h, hu, hv, 3..6 eW, eE, eS, eN) of a staged row at this
// lane's columns; r points at plane 0 of the row.
__device__ __forceinline__ P2 row2(const float* r, int p) { return ld2(r + p * MCR * MBOX); }

// Maximum of a warp's speeds in every lane.
__device__ __forceinline__ float warpMax(float v) {
    return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(v)));
}

struct Cell2 {  // state of this lane's two columns in one row
    P2 h, u, v;
};
__device__ __forceinline__ Cell2 loadCell2(const float* r) {
    return Cell2{row2(r, 0), row2(r, 1), row2(r, 2)};
}

struct Diff2 {  // differences of surface and momenta across the faces of two columns
    P2 w, u, v;
};
// from row a to the row b above it (their staged rows ra, rb)
__device__ __forceinline__ Diff2 diffY(const Cell2& a, const float* ra, const Cell2& b, const float* rb) {
    return Diff2{vadd(vsub(row2(ra, 6), row2(rb, 5)), vsub(b.h, a.h)), vsub(b.u, a.u), vsub(b.v, a.v)};
}
__device__ __forceinline__ void constructY2(const Cell2& c, const float* r, const Diff2& dP,
                                            const Diff2& dM, Face<P2>& P, Face<P2>& M) {
    construct(c.h, c.u, c.v, limited(dP.w, dM.w), limited(dP.u, dM.u), limited(dP.v, dM.v), row2(r, 5),
              row2(r, 6), P, M);
}
// x reconstruction of a row: the states L, R on both sides of the east faces of
// both columns.  The differences mix neighbours of a pair, so they stay scalar
// (packing them would cost a move each).
__device__ __forceinline__ void rowFacesX(const Cell2& c, P2 eW, P2 eE, Face<P2>& L, Face<P2>& R) {
    auto down = [](float a) { return __shfl_down_sync(FULL, a, 1); };
    auto up = [](float a) { return __shfl_up_sync(FULL, a, 1); };
    // limited differences of both columns from d0 (across the face between
    // them) and d1 (across the east face of the second)
    auto limit = [&](float d0, float d1) { return pack2(limited(d0, up(d1)), limited(d1, d0)); };
    const P2 tw = limit(vadd(vsub(lo(eE), hi(eW)), vsub(hi(c.h), lo(c.h))),
                        vadd(vsub(hi(eE), down(lo(eW))), vsub(down(lo(c.h)), hi(c.h))));
    const P2 tu = limit(vsub(hi(c.u), lo(c.u)), vsub(down(lo(c.u)), hi(c.u)));
    const P2 tv = limit(vsub(hi(c.v), lo(c.v)), vsub(down(lo(c.v)), hi(c.v)));
    Face<P2> M;
    construct(c.h, c.u, c.v, tw, tu, tv, eW, eE, L, M);
    auto east = [&](P2 a) { return pack2(hi(a), down(lo(a))); };
    R = Face<P2>{east(M.h), east(M.u), east(M.v)};
}
// The fluxes through the faces between L and R; fx: the difference of each
// column's east and west fluxes, fW0, fE0 the mass fluxes through both.
__device__ __forceinline__ void rowFluxX(const Face<P2>& L, const Face<P2>& R, float kappa, P2 fx[3],
                                         P2& fW0, P2& fE0, P2& spd) {
    P2 f[3];
    spd = faceFlux<0>(L, R, kappa, f);
    float w[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        w[q] = __shfl_up_sync(FULL, hi(f[q]), 1);
        fx[q] = pack2(vsub(lo(f[q]), w[q]), vsub(hi(f[q]), lo(f[q])));
    }
    fW0 = pack2(w[0], lo(f[0]));
    fE0 = f[0];
}

// Rows per item: every warp gets the same number of items, as few rows as
// that allows (an item also loads 4 halo rows and reconstructs about 3 rows'
// worth before its first).  4096^2 cells on 2432 warps: 59 rows in two rounds.
inline int marchItemRows(int nx, int ny, int warps) {
    const long long segs = segCount(nx);
    int best = 2;
    double cost = 1e300;
    for (int r = 2; r <= 64; r++) {
        const long long items = segs * ((ny - 4 + r - 1) / r);
        const double c = (double)((items + warps - 1) / warps) * (r + 3.0);
        if (c < cost) {
            cost = c;
            best = r;
        }
    }
    return best;
}

// Ghost columns of U beside rows [j0, j1) of segment seg, a row per lane (the
// cube root is long: once per 32 rows instead of once per row).
template <class On>
__device__ __forceinline__ void ghostColumns(const Params& P, float* U, int seg, int j0, int j1, On on) {
    const size_t pl = (size_t)P.planeSize;
    __syncwarp();
    for (int side = 0; side < 2; side++) {
        const int gi = side ? P.nx - 3 : 2;
        if (gi < MSEG * seg + 2 || gi >= MSEG * (seg + 1) + 2) continue;
        for (int j = j0 + (int)(threadIdx.x & 31); j < j1; j += 32) {
            if (!on((j - 2) / TH, (gi - 2) / TW)) continue;
            const unsigned c = (unsigned)j * (unsigned)P.pitch + (unsigned)gi;
            writeGhostCols(P, U, j, gi, U[c], U[pl + c], U[2 * pl + c]);
        }
    }
}

// Stage 2 (RK2) folds an active tile's wet flag and speeds into cleared
// entries: cleared between the grow and stage 2, by every item that holds
// rows of the tile.  (Euler: the speeds are stage 1's, into entries the grow
// cleared.)
__device__ __forceinline__ void clearTile(const Params& P, int tile, bool euler) {
    P.wet[tile] = 0;
    if (euler) return;
    P.mx[tile] = 0.f;
    P.my[tile] = 0.f;
}

// Rows [j0, j1) of segment seg by one warp.  on(by, bx): is the tile active?
// (called by all lanes; false for lanes that own no interior column).
// CLEAR (stage 1): see clearTile.  DTS (stage 1): tmx, tmy are the warp's, of
// faceSpeed, instead of this lane's, of faceFlux; maxima below seedX, seedY may
// be missed.
// STAGE 1: reads U^n (A) -> flux divergence + bed source (D), the speed
//          maxima of active cells (tmx, tmy); Euler mode: tile speeds.
// STAGE 2: reads U* (B) and U^n (A) at the cell -> writes U^{n+1} (A),
//          F^{n+1} (FA), outputs, tile wet flags and tile speeds.
template <int STAGE, uint32_t FIX, bool CLEAR, bool DTS, class On>
__device__ __forceinline__ bool marchRows(const Params& P, const StageConsts& C, const CUtensorMap* tmIn,
                                          const CUtensorMap* tmE, MarchRing& S, uint32_t& par, int seg,
                                          int j0, int j1, On on, bool led, Led& L, float& tmx,
                                          float& tmy, bool pf, float seedX = 0.f, float seedY = 0.f) {
    constexpr bool RAINPRE = STAGE == 2 && (FIX & F_RAIN_G) != 0;
    constexpr bool INFPRE = STAGE == 2 && (FIX & F_INFIL) != 0;
    const int lane = threadIdx.x & 31;
    const int i = MSEG * seg + 2 * lane;            // this lane's columns i, i + 1
    const unsigned ic = (unsigned)min(i, P.pitch - 2);
    const bool own = lane >= 1 && lane <= 30;
    const bool inX = own && i <= P.nx - 3, inY = own && i + 1 <= P.nx - 3;
    const int bx = inX ? (i - 2) / TW : -1;         // both columns lie in one tile
    const unsigned group = __match_any_sync(FULL, bx);
    const bool leader = inX && lane == __ffs(group) - 1;
    const bool edge = seg == 0 || MSEG * (seg + 1) + 1 >= P.nx - 3 || j0 == 2 || j1 - 1 >= P.ny - 3;
    const float kappa = C.kappa;
    const unsigned pitch = (unsigned)P.pitch;
    const size_t pl = (size_t)P.planeSize;
    const uint32_t fl = cellFlags<FIX>(C.fl);
    const bool euler = FIX ? (FIX & F_EULER) != 0 : C.euler;

    // the line of plane lane / 4 this lane prefetches (3 lines hold the 64 columns)
    const float* pfB = nullptr;
    if (STAGE == 2 && pf && (lane & 3) < 3) {
        const int p = lane >> 2;
        const unsigned pc = (unsigned)min(MSEG * seg + 32 * (lane & 3), P.pitch - 1);
        if (p < 3) pfB = P.A + p * pl + pc;
        if (RAINPRE && p >= 3 && p < 5 && P.mapMode[0] >= p - 2)
            pfB = (p == 3 ? P.map0[0] : P.map1[0]) + pc;
    }
    // staged row r is grid row j0 - 2 + r; chunk c holds rows 2c and 2c + 1
    const int nch = (j1 - j0 + 4 + MCR - 1) / MCR;
    auto issue = [&](int c, int sl) {
        fence_proxy_async();
        mbar_expect_tx(&S.bar[sl], (uint32_t)sizeof(MarchSlot));
        tma_load_3d(&S.slot[sl].s[0][0][0], tmIn, &S.bar[sl], MSEG * seg, j0 - 2 + MCR * c, 0);
        tma_load_3d(&S.slot[sl].e[0][0][0], tmE, &S.bar[sl], MSEG * seg, j0 - 2 + MCR * c, 0);
    };
    // wait for the chunk in slot sl; false after the spin limit, once the
    // copies in flight have landed or given up too
    auto acquire = [&](int sl) {
        const bool ok = __all_sync(FULL, mbar_wait_bounded(&S.bar[sl], (par >> sl) & 1u));
        if (!ok)
            for (int q = 0; q < MNS; q++) mbar_wait_bounded(&S.bar[q], (par >> q) & 1u);
        par ^= 1u << sl;
        return ok;
    };
    __syncwarp();  // the previous item no longer reads the ring
    if (lane == 0) {
        fence_proxy_async_global();  // the copies see what was stored before the last barrier
        for (int c = 0; c < MNS && c < nch; c++) issue(c, c);
    }
    if (!acquire(0) || !acquire(1)) return false;
    // rows j, j + 1, j + 2 of the current output row
    const float* rc = &S.slot[1].s[0][0][2 * lane];
    const float* rn = rc + MBOX;
    const float* rl = &S.slot[2].s[0][0][2 * lane];
    Cell2 cur = loadCell2(rc), nxt = loadCell2(rn);
    Face<P2> yP;      // the row's reconstruction at its north face
    P2 fS[3];      // flux through its south face
    Diff2 dN;      // differences to the row above
    {
        const float* r0 = &S.slot[0].s[0][0][2 * lane];
        const float* r1 = r0 + MBOX;
        const Cell2 m2 = loadCell2(r0), m1 = loadCell2(r1);
        const Diff2 d0 = diffY(m2, r0, m1, r1), d1 = diffY(m1, r1, cur, rc);
        dN = diffY(cur, rc, nxt, rn);
        Face<P2> a, b, M;
        constructY2(m1, r1, d1, d0, a, b);
        constructY2(cur, rc, dN, d1, yP, M);
        faceFlux<1>(a, M, kappa, fS);
    }
    // the row's centre values (stage 2: U^n; rain maps or F, K, F^n when the
    // instantiation reads them ahead)
    P2 pre[6];
    auto loadCentre = [&](P2 (&d)[6], int jj) {
        const unsigned c = (unsigned)jj * pitch + ic;
        d[0] = ld2(P.A + c);
        d[1] = ld2(P.A + pl + c);
        d[2] = ld2(P.A + 2 * pl + c);
        if (RAINPRE) {
            d[3] = P.mapMode[0] != 0 ? ld2(P.map0[0] + c) : both(0.f);
            d[4] = P.mapMode[0] == 2 ? ld2(P.map1[0] + c) : both(0.f);
        } else if (INFPRE) {
            d[3] = ld2(C.Fin + c);
            d[4] = ld2(P.K + c);
            d[5] = ld2(P.FA + c);
        }
    };
#pragma unroll
    for (int q = 0; q < 6; q++) pre[q] = both(0.f);

    int sl = 1;  // slot of the chunk that holds row j + 1
    int by = (j0 - 2) / TH, rt = (j0 - 2) % TH;  // tile row, row in it
    bool act = on(by, bx);
    // the active cells' speeds as the speed pass rounds them, into the maximum m
    // of the warp: formed only where the fluxes' speeds, within 2e-7 of them,
    // come near it, and above the seed
    auto dtSpeeds = [&](P2 s, P2 hL, P2 qL, P2 hR, P2 qR, float& m, float seed) {
        auto top = [&](P2 v) { return act ? fmaxf(lo(v), inY ? hi(v) : 0.f) : 0.f; };
        if (!__any_sync(FULL, top(s) > fmaxf(m, seed) * (1.f - 1e-6f))) return;
        m = fmaxf(m, warpMax(top(pack2(faceSpeed(lo(hL), lo(qL), lo(hR), lo(qR), kappa),
                                       faceSpeed(hi(hL), hi(qL), hi(hR), hi(qR), kappa)))));
    };
    int src = STAGE == 2 && act ? sourceTile(P, by * P.nBX + bx) : -1;
    float ax = 0.f, ay = 0.f;
    bool wet = false;
    if (CLEAR && leader && act) clearTile(P, by * P.nBX + bx, euler);
    constexpr int UNROLL = STAGE == 1 ? 2 : 1;
#pragma unroll UNROLL
    for (int j = j0; j < j1; j++) {
        if (((j - j0) & 1) == 0) {
            // row j + 2 opens chunk k + 1 (k holds row j); rows below j are
            // done: their slot takes chunk k - 1 + MNS
            const int k = (j - j0) / 2 + 1;
            __syncwarp();
            sl = sl == MNS - 1 ? 0 : sl + 1;  // slot of chunk k + 1
            if (lane == 0 && k - 1 + MNS < nch) issue(k - 1 + MNS, sl < 2 ? sl + MNS - 2 : sl - 2);
            if (!acquire(sl)) return false;
            rl = &S.slot[sl].s[0][0][2 * lane];
        }
        if (STAGE == 2) loadCentre(pre, j);  // in flight during both directions' fluxes
        if (STAGE == 2 && FIX == 0) prefetchMaps(P, fl, (unsigned)j * pitch + ic);
        if (STAGE == 2 && pfB) prefetch_l2(pfB + (size_t)((unsigned)min(j + MPF, P.rows - 1) * pitch));
        const P2 eW = row2(rc, 3), eE = row2(rc, 4);
        P2 fN[3], sy, fx[3], fW0, fE0, sx;
        Face<P2> xL, xR;
        rowFacesX(cur, eW, eE, xL, xR);
        rowFluxX(xL, xR, kappa, fx, fW0, fE0, sx);
        if (DTS) dtSpeeds(sx, xL.h, xL.u, xR.h, xR.u, tmx, seedX);
        // y: reconstruction of row j + 1, flux through the north face of row j
        const Cell2 ld = loadCell2(rl);
        const Diff2 dNN = diffY(nxt, rn, ld, rl);
        Face<P2> yn, yM;
        constructY2(nxt, rn, dNN, dN, yn, yM);
        sy = faceFlux<1>(yP, yM, kappa, fN);
        if (DTS) dtSpeeds(sy, yP.h, yP.v, yM.h, yM.v, tmy, seedY);
        // divergence, with the bed-slope source in the momenta
        P2 d[3];
#pragma unroll
        for (int q = 0; q < 3; q++)
            d[q] = divergence(fx[q], vsub(fN[q], fS[q]), P.inv_dx, P.inv_dy);
        d[1] = addBed(d[1], cur.h, eW, eE, P.inv_dx);
        d[2] = addBed(d[2], cur.h, row2(rc, 5), row2(rc, 6), P.inv_dy);
        if (act) {
            if (!DTS) {
                ax = fmaxf(fmaxf(ax, lo(sx)), inY ? hi(sx) : 0.f);
                ay = fmaxf(fmaxf(ay, lo(sy)), inY ? hi(sy) : 0.f);
            }
            const unsigned c = (unsigned)j * pitch + (unsigned)i;
            if (led && edge) {
                float r = edgeInflow(P, j, i, lo(fW0), lo(fE0), lo(fS[0]), lo(fN[0]));
                if (inY) r += edgeInflow(P, j, i + 1, hi(fW0), hi(fE0), hi(fS[0]), hi(fN[0]));
                L.v[LED_BOUND] += STAGE == 1 ? r : C.wRate * r;
            }
            if (STAGE == 1) {
                st2(P.D + c, d[0]);
                st2(P.D + pl + c, d[1]);
                st2(P.D + 2 * pl + c, d[2]);
            } else {
                float r[2][3];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (k == 1 && !inY) break;
                    auto at = [&](P2 a) { return k == 0 ? lo(a) : hi(a); };
                    const float hC = at(cur.h), u0 = at(cur.u), v0 = at(cur.v);
                    const float pk[8] = {at(pre[0]), at(pre[1]), at(pre[2]), at(pre[3]),
                                         at(pre[4]), at(pre[5]), at(pre[3]), at(pre[4])};
                    const CellSrc s = cellSources<2, INFPRE, false, FIX, RAINPRE>(
                        P, C, src, j, i + k, at(d[0]), at(d[1]), at(d[2]), hC, u0, v0, 0.f, 0.f,
                        0.f, 0.f, pk);
                    wet |= cellResult<2, INFPRE, FIX>(P, C, j, i + k, s, hC, u0, v0, pk,
                                                      led ? &L : nullptr, r[k][0], r[k][1], r[k][2]);
                }
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    if (inY)
                        st2(P.A + q * pl + c, pack2(r[0][q], r[1][q]));
                    else
                        P.A[q * pl + c] = r[0][q];
                }
                if (j == 2 || j == P.ny - 3) {
                    writeGhostRows(P, P.A, j, i, r[0][0], r[0][1], r[0][2]);
                    if (inY) writeGhostRows(P, P.A, j, i + 1, r[1][0], r[1][1], r[1][2]);
                }
            }
        }
        if (++rt == TH || j + 1 == j1) {  // the item's last row of a tile row (warp-uniform)
            if (STAGE == 1 && !DTS) {
                tmx = fmaxf(tmx, ax);
                tmy = fmaxf(tmy, ay);
            }
            if (STAGE == 2 || euler) {  // speeds are non-negative: their bits order like the values
                const unsigned mx = __reduce_max_sync(group, __float_as_uint(ax));
                const unsigned my = __reduce_max_sync(group, __float_as_uint(ay));
                const unsigned any = __reduce_or_sync(group, wet ? 1u : 0u);
                if (leader && act) {
                    const int tile = by * P.nBX + bx;
                    atomicMax(reinterpret_cast<unsigned*>(P.mx) + tile, mx);
                    atomicMax(reinterpret_cast<unsigned*>(P.my) + tile, my);
                    if (STAGE == 2 && (any || !(fl & F_TILE_ACC))) P.wet[tile] = 1;
                }
            }
            rt = 0;
            ax = ay = 0.f;
            wet = false;
            if (j + 1 < j1) {
                by++;
                act = on(by, bx);
                src = STAGE == 2 && act ? sourceTile(P, by * P.nBX + bx) : -1;
                if (CLEAR && leader && act) clearTile(P, by * P.nBX + bx, euler);
            }
        }
#pragma unroll
        for (int q = 0; q < 3; q++) fS[q] = fN[q];
        yP = yn;
        dN = dNN;
        cur = nxt;
        nxt = ld;
        rc = rn;
        rn = rl;
        rl += MBOX;
    }
    if (STAGE == 2 && edge) ghostColumns(P, P.A, seg, j0, j1, on);
    return true;
}

// Resident CTAs per SM the march is compiled for: 128 registers a thread.
// (4096^2 urban rain, stage 1 / stage 2: 153 / 222 us at 4, 177 / 233 us at 3
// with 168 registers; at 5 the 96 registers spill and both run slower than the
// kernel of one column per lane this one replaced.)  Two rows per loop
// iteration in stage 1 (167 us with one), one in stage 2 (243 us with two).
constexpr int MARCH_CTAS = 4;

// rows: rows per item; negative: as many, but at most a tile row's, aligned
// with it, while tiles are inactive.  (The fitted height gives every warp the same
// number of items, of which it skips those without an active tile: some warps
// then hold several and some none.  2600^2 rain maps, half of the tiles active:
// 291 us a step at the fitted height, 254 at 14 rows.)
template <int STAGE, uint32_t FIX = 0>
__global__ void __launch_bounds__(MT, MARCH_CTAS) k_march(const __grid_constant__ CUtensorMap tmIn,
                                                                  const __grid_constant__ CUtensorMap tmE,
                                                                  Params P, int rows, int pf) {
    __shared__ MarchRing rings[MW];
    __shared__ bool last;
    __shared__ float wmax[2][MW];
    __shared__ int sRows;
    if (P.st->stop || !useMarch(P)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ __align__(8) unsigned char cbuf[sizeof(StageConsts)];
    StageConsts& C = *reinterpret_cast<StageConsts*>(cbuf);
    MarchRing& S = rings[warp];
    if (tid == 0) {
        const bool some = P.st->nActive < ((P.nx - 4 + TW - 1) / TW) * ((P.ny - 4 + TH - 1) / TH);
        sRows = rows > 0 ? rows : some ? min(-rows, TH) : -rows;
        C = stageConsts<STAGE>(P);
        prefetch_tmap(&tmIn);
        prefetch_tmap(&tmE);
    }
    if (lane == 0) {
        for (int k = 0; k < MNS; k++) mbar_init(&S.bar[k], 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t par = 0u;
    const bool led = (cellFlags<FIX>(C.fl) & F_CHECKVOL) != 0;
    Led L;
    ledZero(L);
    float tmx = 0.f, tmy = 0.f;
    const int itemRows = sRows;
    const int nSeg = segCount(P.nx), nGroup = (P.ny - 4 + itemRows - 1) / itemRows;
    auto on = [&](int by, int bx) { return bx >= 0 && P.prevAct[by * P.nBX + bx] != 0; };
    for (int item = blockIdx.x * MW + warp; item < nSeg * nGroup; item += gridDim.x * MW) {
        const int seg = item % nSeg, j0 = 2 + itemRows * (item / nSeg);
        const int j1 = min(j0 + itemRows, P.ny - 2);
        // does the item hold an active tile? (lane q tests tile row q of its rows)
        const int bx0 = MSEG * seg / TW, bx1 = min(MSEG * seg + MSEG - 1, P.nx - 5) / TW;
        const int by0 = (j0 - 2) / TH, by1 = (j1 - 3) / TH;
        const int nb = bx1 - bx0 + 1;
        bool any = false;
        for (int q = lane; q < nb * (by1 - by0 + 1); q += 32)
            any |= on(by0 + q / nb, bx0 + q % nb);
        if (!__any_sync(FULL, any)) continue;
        if (!marchRows<STAGE, FIX, STAGE == 1, false>(P, C, &tmIn, &tmE, S, par, seg, j0, j1, on, led, L, tmx, tmy, pf != 0)) {
            if (lane == 0) atomicOr(&P.st->error, ERR_TMA_TIMEOUT);
            break;
        }
    }
    if (led) {
        if (STAGE == 1) {
            float r = L.v[LED_BOUND];
            for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(FULL, r, o);
            if (lane == 0 && r != 0.f) atomicAdd(&P.st->ledPend, (double)r);
            __threadfence();  // before the dt ticket: the last CTA folds ledPend
        } else {
            flushLed(L, P.st->led);
        }
    }
    if (STAGE == 1) {
        tmx = warpMax(tmx);
        tmy = warpMax(tmy);
        if (lane == 0) {
            wmax[0][warp] = tmx;
            wmax[1][warp] = tmy;
        }
        __syncthreads();
        if (tid == 0)
            for (int w = 0; w < MW; w++) {
                tmx = fmaxf(tmx, wmax[0][w]);
                tmy = fmaxf(tmy, wmax[1][w]);
            }
        finishDt(P, tmx, tmy, &last);
        resyncDeactivated(P);
    }
}

}  // namespace rift
