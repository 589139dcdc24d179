// rift_flow.cuh -- the step loop in one cooperative launch on the march's
// work items, for active sets larger than one tile per CTA.
//
// k_persist (rift_persist.cuh) is built around one 16 x 14 tile per CTA; with
// more tiles than CTAs its step falls back to whole-grid phases of per-tile
// code with a separate speed pass.  k_flow runs such steps on the warps of
// one CTA per SM, each warp on its own items of 60 columns (rift_march.cuh),
// with three phases between grid barriers:
//   flux    marchRows<1>: stage-1 divergence, speed maxima
//   update  dt in every CTA, then the rest of RK stage 1 (updateRows)
//   stage 2 marchRows<2>
// and, on the first step and when the active set changes, the grow before
// them (and, while gridded rain or surge meets inactive tiles, the re-wet
// tracking with a barrier at the start of every step).  The set seldom changes,
// so from the second step on the flux phase runs on the last step's set while
// spare warps compare every tile's activity with it; only when one differs does
// the step grow the set and repeat its flux phase (measured: the grow and its
// barrier take 6 to 7 us of a step.  A list that stays also keeps a row on the
// same warp: 1400^2 rain maps, half of the tiles active, 127 -> 118 us a step).
//
// Items: with every tile active, the grid cut into rows fitted to the warps
// (marchItemRows).  Otherwise the grow lists the (segment, tile row) pairs that
// hold an active tile, and each is cut into as many pieces as there are warps
// to take them: a lone warp needs about 0.6 us per row, so a sparse set is
// spread thin.
//
// dt takes the speeds as the per-tile schedule's speed pass rounds them
// (faceSpeed), so both give the same dt; the fluxes' own differ in the last
// bit.  They are formed only for faces near the maximum and above 15/16 of the
// last step's (1117 x 1531 rain: 94 us a step, 96 without that seed).
//
// What bounds it (us per step, GB300).  512^2 rain, 1221 tiles: 22.7 (34 with
// the per-tile phases; 24.2 with tracking code in it, of which flux 5, dt 1.0,
// update 3.1, stage 2 7 and three barriers of 1.3 to 1.8 with the wait for the
// slowest CTA on top): latency.
// 1024^2 rain: 50 (86) = 12 + 1.0 + 8.7 + 17 + barriers and waits 10: issue in
// the flux passes, L2 in the update (52 bytes per cell).
#pragma once
#include "rift_grow.cuh"
#include "rift_march.cuh"
#include "rift_persist.cuh"

namespace rift {

constexpr int FLOW_WARPS = 16;
constexpr int FLOW_T = FLOW_WARPS * 32;
constexpr uint32_t FLOW_SMEM = FLOW_WARPS * sizeof(MarchRing);

// The rest of Integrate_1_k (grid.cu:856-922) on rows [j0, j1) of segment seg,
// once dt is known: U* and F* from U^n and the stored divergence.  CLEAR: see
// clearTile.  Euler mode: sets the wet flags of the tiles with wet cells, which
// the caller cleared a grid barrier before (other warps hold rows of the same
// tiles: a clear here would undo what they set).  One warp, the lanes and
// columns of marchRows; two rows of loads in flight.
template <uint32_t FIX, bool CLEAR, class On>
__device__ __forceinline__ void updateRows(const Params& P, const StageConsts& C, int seg, int j0,
                                           int j1, On on, bool led, Led& L) {
    constexpr bool RAINPRE = (FIX & F_RAIN_G) != 0;
    constexpr bool INFPRE = (FIX & F_INFIL) != 0;
    const int lane = threadIdx.x & 31;
    const int i = MSEG * seg + 2 * lane;
    const bool own = lane >= 1 && lane <= 30;
    const bool inX = own && i <= P.nx - 3, inY = own && i + 1 <= P.nx - 3;
    const int bx = inX ? (i - 2) / TW : -1;
    const unsigned pitch = (unsigned)P.pitch;
    const size_t pl = (size_t)P.planeSize;
    const bool edge = seg == 0 || MSEG * (seg + 1) + 1 >= P.nx - 3;
    const bool euler = FIX ? (FIX & F_EULER) != 0 : C.euler;
    struct In {
        P2 a[3], d[3], n, x[2];
    };
    auto load = [&](In& r, unsigned c) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            r.a[q] = ld2(P.A + q * pl + c);
            r.d[q] = ld2(P.D + q * pl + c);
        }
        r.n = ld2(P.nman + c);
        r.x[0] = r.x[1] = both(0.f);
        if (RAINPRE) {
            if (P.mapMode[0] != 0) r.x[0] = ld2(P.map0[0] + c);
            if (P.mapMode[0] == 2) r.x[1] = ld2(P.map1[0] + c);
        } else if (INFPRE) {
            r.x[0] = ld2(C.Fin + c);
            r.x[1] = ld2(P.K + c);
        }
    };
    auto cells = [&](const In& r, int tile, int j) {
        const unsigned c = (unsigned)j * pitch + (unsigned)i;
        bool wet = false;
        float u[2][3];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (k == 1 && !inY) break;
            auto at = [&](P2 a) { return k == 0 ? lo(a) : hi(a); };
            const float pk[8] = {at(r.n), 0.f, 0.f, at(r.x[0]), at(r.x[1]), 0.f, at(r.x[0]), at(r.x[1])};
            const CellSrc s = cellSources<1, INFPRE, false, FIX, RAINPRE>(
                P, C, tile, j, i + k, at(r.d[0]), at(r.d[1]), at(r.d[2]), at(r.a[0]), at(r.a[1]),
                at(r.a[2]), 0.f, 0.f, 0.f, 0.f, pk);
            wet |= cellResult<1, INFPRE, FIX>(P, C, j, i + k, s, at(r.a[0]), at(r.a[1]), at(r.a[2]), pk,
                                              led ? &L : nullptr, u[k][0], u[k][1], u[k][2]);
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            if (inY)
                st2(P.B + q * pl + c, pack2(u[0][q], u[1][q]));
            else
                P.B[q * pl + c] = u[0][q];
        }
        if (j == 2 || j == P.ny - 3) {
            writeGhostRows(P, P.B, j, i, u[0][0], u[0][1], u[0][2]);
            if (inY) writeGhostRows(P, P.B, j, i + 1, u[1][0], u[1][1], u[1][2]);
        }
        return wet;
    };
    const unsigned group = __match_any_sync(FULL, bx);
    const bool leader = inX && lane == __ffs(group) - 1;
    int byOld = -1;
    for (int j = j0; j < j1; j += 2) {
        const int by = (j - 2) / TH, by2 = (j - 1) / TH;
        const bool a0 = on(by, bx), a1 = j + 1 < j1 && (by2 == by ? a0 : on(by2, bx));
        if (CLEAR && !euler && leader && a0 && by != byOld) clearTile(P, by * P.nBX + bx, false);
        if (CLEAR && !euler && leader && a1 && by2 != by) clearTile(P, by2 * P.nBX + bx, false);
        const int src0 = a0 ? sourceTile(P, by * P.nBX + bx) : -1;
        const int src1 = a1 ? (by2 == by ? src0 : sourceTile(P, by2 * P.nBX + bx)) : -1;
        byOld = a1 ? by2 : by;
        In r0, r1;
        const unsigned c = (unsigned)j * pitch + (unsigned)i;
        if (FIX == 0 && a0) prefetchMaps(P, C.fl, c);
        if (FIX == 0 && a1) prefetchMaps(P, C.fl, c + pitch);
        if (a0) load(r0, c);
        if (a1) load(r1, c + pitch);
        const bool w0 = a0 && cells(r0, src0, j);
        const bool w1 = a1 && cells(r1, src1, j + 1);
        if (euler) {
            const bool any0 = __reduce_or_sync(group, w0 ? 1u : 0u) != 0u;
            const bool any1 = __reduce_or_sync(group, w1 ? 1u : 0u) != 0u;
            const bool keep = !(cellFlags<FIX>(C.fl) & F_TILE_ACC);
            if (leader && a0 && (any0 || keep)) P.wet[by * P.nBX + bx] = 1;
            if (leader && a1 && (any1 || keep)) P.wet[by2 * P.nBX + bx] = 1;
        }
    }
    if (edge) ghostColumns(P, P.B, seg, j0, j1, on);
}

// flushLed for the whole CTA: one atomic per term.  (One per term and warp has
// 2432 of them queue at each address: 500 x 701 with a surge 43.7 us a step,
// 42.9 with one per CTA.)
__device__ __forceinline__ void flushLedBlock(Led& L, double* dst) {
    __shared__ float part[LED_N][FLOW_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < LED_N; k++) {
        float v = L.v[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0) part[k][warp] = v;
        L.v[k] = 0.f;
    }
    __syncthreads();
    if (warp < LED_N) {
        double sum = lane < FLOW_WARPS ? (double)part[warp][lane] : 0.0;
        for (int o = FLOW_WARPS / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
        if (lane == 0 && sum != 0.0) atomicAdd(&dst[warp], sum);
    }
}

// Step loop.  itemRows: rows per item while every tile is active.
// minTiles: the loop leaves (persistExit) when fewer tiles are scheduled.
template <uint32_t FIX = 0>
__global__ void __launch_bounds__(FLOW_T, 1) k_flow(const __grid_constant__ CUtensorMap tmA,
                                                    const __grid_constant__ CUtensorMap tmB,
                                                    const __grid_constant__ CUtensorMap tmE, Params P,
                                                    int maxSteps, int itemRows, int minTiles) {
    extern __shared__ __align__(128) unsigned char flowRaw[];
    __shared__ __align__(8) unsigned char cbuf[2][sizeof(StageConsts)];
    __shared__ double sDt, sT;
    __shared__ float wmax[2][FLOW_WARPS];
    __shared__ unsigned sStale[2];
    __shared__ float sSeed[2];
    __shared__ int sErr, sRedo;
    StageConsts& C1 = *reinterpret_cast<StageConsts*>(cbuf[0]);
    StageConsts& C2 = *reinterpret_cast<StageConsts*>(cbuf[1]);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    MarchRing& S = reinterpret_cast<MarchRing*>(flowRaw)[warp];
    DevState* st = P.st;
    GridBar* const T = P.gbar;
    const uint32_t fl = P.flags;
    const bool track = (cellFlags<FIX>(fl) & (F_RAIN_G | F_SURGE)) != 0;
    const bool spare = blockIdx.x == gridDim.x - 1;
    const bool led = (cellFlags<FIX>(fl) & F_CHECKVOL) != 0;
    Led L;
    ledZero(L);
    if (lane == 0) {
        for (int k = 0; k < MNS; k++) mbar_init(&S.bar[k], 1);
        fence_mbar_init();
    }
    if (tid == 0) {
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        prefetch_tmap(&tmE);
        sStale[0] = sStale[1] = 0u;
        sSeed[0] = sSeed[1] = 0.f;
        C1 = stageConsts<1>(P);  // (the flux phase reads what no step changes)
        C2 = stageConsts<2>(P);
    }
    uint32_t par = 0u;
    unsigned barTarget = 0u;
    double tNow = st->t, dtPrev = st->dt;
    const double tStop = st->t_stop;
    const int nSeg = segCount(P.nx), nW = FLOW_WARPS * (int)gridDim.x;
    const int gw = warp * (int)gridDim.x + (int)blockIdx.x;
    const int allTiles = ((P.nx - 4 + TW - 1) / TW) * ((P.ny - 4 + TH - 1) / TH);
    int nAct = 0, nDe = 0, nInact = st->nInact, nList = 0;
    unsigned long long cells = 0ull;  // spare CTA: interior cells of the active tiles
    if (blockIdx.x == 0 && tid == 0) st->persistExit = 0;
    __syncthreads();
    auto on = [&](int by, int bx) { return bx >= 0 && P.prevAct[by * P.nBX + bx] != 0; };
#define FLOW_SYNC()                              \
    if (!gridSync(P.gbar, barTarget, st)) return; \
    (void)0
    for (int step = 0; step < maxSteps; step++) {
        if (tNow >= tStop) {
            if (blockIdx.x == 0 && tid == 0) st->stop = 1;
            return;
        }
        if (step > 0 && (nAct > P.persistMax || nAct < minTiles)) {
            if (blockIdx.x == 0 && tid == 0) st->persistExit = 1;
            return;
        }
        const int pr = step & 1;
        // the grow is a no-op when no tile's activity changes: from the second
        // step on the flux phase runs on the last step's set and checks that
        bool rated = false;  // this step's source rates are formed
        bool grown = false;  // and its set is the grow's
        // the dt speeds are sought from 15/16 of the last step's maxima upward;
        // where none is found, once more from 0
        float seedX = sSeed[0], seedY = sSeed[1];
        // (inactive tiles without interior cells are never tracked into the set)
        const bool trackNow = track && (step == 0 ? nInact != 0 : nAct < allTiles);
        bool guess = step > 0;
        if (trackNow) {
            trackTiles(P);
            FLOW_SYNC();
        }
        if (blockIdx.x == 0 && tid == 0) beginStepResets(st);
    flux:
        if (!guess && !grown) {
            grown = true;
            if (tid < NT) growAppend<false, true>(P, T->staleb[pr], &T->itemCnt[pr]);
            FLOW_SYNC();
            nAct = (int)ld_relaxed_gpu((const unsigned*)&st->appendCnt[0]);
            nDe = (int)ld_relaxed_gpu((const unsigned*)&st->appendCnt[1]);
            nInact = (int)ld_relaxed_gpu((const unsigned*)&st->appendCnt[2]);
            nList = (int)ld_relaxed_gpu((const unsigned*)&T->itemCnt[pr]);
            if (tid == 0) {
                sStale[0] = ld_relaxed_gpu(&T->staleb[pr][0]);
                sStale[1] = ld_relaxed_gpu(&T->staleb[pr][1]);
            }
            for (int k = blockIdx.x * FLOW_T + tid; k < nList; k += gridDim.x * FLOW_T)
                P.itemStamp[P.items[k]] = 0;  // for the next grow
        } else if (guess) {
            nDe = 0;
        }
        const bool all = nAct == allTiles;
        // pieces of a listed item, and rows per piece
        const int cut = all ? 1 : max(1, min(TH / 2, nW / max(nList, 1)));
        const int rows = all ? itemRows : (TH + cut - 1) / cut;
        const int nItems = all ? nSeg * ((P.ny - 4 + rows - 1) / rows) : nList * cut;
        // fn(seg, j0, j1) on this warp's items, until it returns false
        auto items = [&](auto fn) {
            for (int k = gw; k < nItems; k += nW) {
                int seg, j0, j1;
                if (all) {
                    seg = k % nSeg;
                    j0 = 2 + rows * (k / nSeg);
                    j1 = min(j0 + rows, P.ny - 2);
                } else {
                    const int id = P.items[k / cut], by = id / nSeg;
                    seg = id % nSeg;
                    j0 = 2 + TH * by + rows * (k % cut);
                    j1 = min(min(j0 + rows, 2 + TH * (by + 1)), P.ny - 2);
                }
                if (j0 < j1 && !fn(seg, j0, j1)) return false;
            }
            return true;
        };
        // ---- flux (the last warp, which has the fewest items, forms this step's source rates first)
        if (gw == nW - 1 && !rated) beginStepRates(P, st);
        rated = true;
        float tmx = 0.f, tmy = 0.f;
        Led L1;  // stage 1's edge inflow rates: dt is not known yet
        ledZero(L1);
        bool ok = items([&](int seg, int j0, int j1) {
            return marchRows<1, 0, false, true>(P, C1, &tmA, &tmE, S, par, seg, j0, j1, on, led, L1, tmx, tmy,
                                          false, seedX, seedY);
        });
        if (!ok && lane == 0) atomicOr(&st->error, ERR_TMA_TIMEOUT);
        if (guess) {
            // tiles whose activity changed, on the warps without items (or on all)
            const int idle = nW - nItems;
            const bool few = idle < (int)gridDim.x;
            const int rank = few ? gw : gw - nItems, n = few ? nW : idle;
            bool diff = false;
            if (rank >= 0)
                for (int b = rank * 32 + lane; b < P.gridSize; b += n * 32)
                    diff |= tileGrows(P, b) != (P.prevAct[b] != 0);
            if (__any_sync(FULL, diff) && lane == 0) atomicOr(&T->changed[pr], 1);
        }
        resyncDeactivated(P, nDe);
        tmx = warpMax(tmx);
        tmy = warpMax(tmy);
        if (lane == 0) {
            wmax[0][warp] = tmx;
            wmax[1][warp] = tmy;
        }
        __syncthreads();
        if (tid < 2) {
            float m = 0.f;
            for (int w = 0; w < FLOW_WARPS; w++) m = fmaxf(m, wmax[tid][w]);
            atomicMax(guess ? &T->guess[pr][tid] : &T->maxb[pr][tid], __float_as_uint(m));
        }
        FLOW_SYNC();
        // ---- dt (Simulator::ComputeTimestep) and the stage constants, by
        // thread 0 of every CTA (which all see the same counts and maxima);
        // then stage 1's update
        if (tid == 0) {
            const unsigned* const m = guess ? T->guess[pr] : T->maxb[pr];
            const unsigned mx = ld_relaxed_gpu(&m[0]), my = ld_relaxed_gpu(&m[1]);
            const unsigned ch = ld_relaxed_gpu((const unsigned*)&T->changed[pr]);
            sErr = (int)ld_relaxed_gpu((const unsigned*)&st->error);
            sRedo = guess && ch != 0u ? 1 : __uint_as_float(mx) < seedX || __uint_as_float(my) < seedY ? 2 : 0;
            if (sRedo == 0) {
                const double dtNew = stepDtAt(P, tNow, __uint_as_float(max(mx, sStale[0])),
                                              __uint_as_float(max(my, sStale[1])));
                sDt = dtNew;
                sT = tNow + dtNew;
                C1 = stageConstsAt<1>(P, dtNew, dtPrev, sT);
                C2 = stageConstsAt<2>(P, dtNew, dtPrev, sT);
                sSeed[0] = 0.9375f * __uint_as_float(mx);
                sSeed[1] = 0.9375f * __uint_as_float(my);
            }
        }
        __syncthreads();
        if (sErr) return;  // a wait gave up before the barrier: every CTA sees it
        if (sRedo == 1) {  // the set changes
            guess = false;
            goto flux;
        }
        if (sRedo == 2) {  // no speed as high as the seed (the next maxima join these)
            seedX = seedY = 0.f;
            FLOW_SYNC();
            goto flux;
        }
        tNow = sT;
        dtPrev = sDt;
        L.v[LED_BOUND] += C1.wRate * L1.v[LED_BOUND];
        items([&](int seg, int j0, int j1) {
            updateRows<FIX, true>(P, C1, seg, j0, j1, on, led, L);
            return true;
        });
        FLOW_SYNC();
        // ---- stage 2; the spare CTA publishes dt and the grow's counts
        ok = items([&](int seg, int j0, int j1) {
            return marchRows<2, FIX, false, false>(P, C2, &tmB, &tmE, S, par, seg, j0, j1, on, led, L, tmx, tmy, false);
        });
        if (!ok && lane == 0) atomicOr(&st->error, ERR_TMA_TIMEOUT);
        if (spare && tid == 0) {
            publishDt(P, st, sDt);
            T->maxb[pr ^ 1][0] = T->maxb[pr ^ 1][1] = 0u;
            T->staleb[pr ^ 1][0] = T->staleb[pr ^ 1][1] = 0u;
            T->guess[pr ^ 1][0] = T->guess[pr ^ 1][1] = 0u;
            T->itemCnt[pr ^ 1] = T->changed[pr ^ 1] = 0;
            if (!guess) {
                cells = st->appendCells;
                publishGrow(st);
            } else {
                st->activeCells += cells;
                st->nDeact = 0;
            }
        }
        if (led) flushLedBlock(L, st->led);
        FLOW_SYNC();
    }
#undef FLOW_SYNC
}

}  // namespace rift
