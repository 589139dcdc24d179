// rift_ensemble.cuh -- many independent simulations (members: scenarios on
// domains of uneven size) stepped by one persistent cooperative kernel.
//
// Each member is an engine handle with its own buffers, DevState and dt.
// Every iteration of k_ensemble advances every live member by one of its own
// steps, in five phases separated by grid barriers (six with tracking):
//   T  (members with gridded rain or surge) re-wet tracking of inactive tiles
//   G  grow: the strips of all live members (chunked over the CTAs) append
//      each member's lists; the stale speed maxima of the tiles that are not
//      active.  Only on the first iteration, when an active set changed, and
//      while a member in Euler mode is live: otherwise S runs on the last sets
//      and checks them, as k_flow does.  (An Euler member's tile speeds are
//      folded in S, into entries that the grow has read and cleared.)
//   S  flux: the stage-1 divergence and the members' speed maxima; the start
//      of each member's step (one warp per member); U* re-sync of the tiles
//      that went inactive
//   D  dt: one thread per member -> dt, t, ledger, list sizes, liveness of
//      the member's next step; the wet flags of the Euler members' active
//      tiles are cleared (phase 1 sets those of the wet ones: warps share
//      tiles, so a clear has to lie a barrier away from it)
//   1  the rest of RK stage 1
//   2  stage 2 of the RK members.  An Euler member's step ends with phase 1,
//      which writes U^{n+1} and F in place: it reads its own cells only (the
//      fluxes are in the divergence planes).  Through U* and a copy of the tiles
//      back, three members of 512 x 600 to 900 x 850 cells took 188 us an
//      iteration, 106 in place.
// S, 1 and 2 run the march's code (rift_march.cuh, rift_flow.cuh) on the warps
// of one CTA per SM.  The members' 60-column segments, one under the other
// (of a member with inactive tiles the listed (segment, tile row) pairs), make
// one queue of rows, and each warp takes an equal run of it: cut into whole
// tile rows instead, 20 members of 96 to 480 cells a side made 1.1 rounds of
// items, that is two.  The arithmetic is the single-member code, so each member's results are those of
// a run of its own.  A member is live while t < t_stop and its step count is
// below the requested maximum; the kernel ends when no member is live.  Every
// wait is bounded (TMA mbarriers, grid barriers), as in k_persist.
//
// What bounds it: 20 members of 96 to 480 cells a side, uniform rain (1.58 M
// cells), 102 us per iteration (191 on per-tile queues with a grow in every
// iteration): flux 20.7, update 22, stage 2 29.9 (issue and the latency of a
// warp's chain, 15.5 rows a warp), dt 4, the rest barriers and waits.  A run of
// 8 steps also takes 109 us on the host (336 with a copy and a wait each way
// per member).
#pragma once
#include "rift_flow.cuh"

namespace rift {

constexpr int ENS_MAX = 1024;  // members per ensemble

struct EnsTimes {
    unsigned long long t0;              // globaltimer at the kernel's start (ns)
    unsigned long long tDone[ENS_MAX];  // globaltimer when each member finished its last step
};

// Device side of an ensemble.
struct EnsDev {
    GridBar bar;
    int live[2][ENS_MAX];  // liveness per step parity
    int nAlive[2];
    int nEuler[2];         // live members in Euler mode
    int itemCnt[ENS_MAX];  // the grow's count of a member's (segment, tile row) pairs
    int nItems[ENS_MAX];   // the pairs of the member's current set
    int all[ENS_MAX];      // every tile with interior cells is active
    unsigned stale[ENS_MAX][2];          // speed maxima of the inactive tiles (bits)
    unsigned long long cells[ENS_MAX];   // interior cells of the active tiles
    int changed[2];        // by step parity: an active set differs from the last step's
    int fail;              // a wait gave up: every CTA leaves
    StageConsts consts[ENS_MAX][2];  // each member's stage constants of the step (phase D)
    EnsTimes times;
};

// One member as the host sends it: the tensor maps of A, B and E (march
// boxes), its parameters and device state.
struct EnsMember {
    CUtensorMap maps[3];
    Params P;
    DevState st;
    int live;
};

__device__ __forceinline__ unsigned long long globalTimerNs() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct EnsArgs {
    const EnsMember* M;  // [n]
    EnsDev* dev;
    int n;
    int maxSteps;
    int polls;  // of a grid barrier, after which it gives up
};

// The members' device states from the block the host sent, and back: one
// copy each way for all members (a copy per member each way, with a wait
// each, took 330 us a run of 20 members).
__global__ void k_ens_begin(const EnsMember* M, EnsDev* D) {
    const EnsMember& m = M[blockIdx.x];
    copyState(m.P.st, &m.st);
    if (threadIdx.x == 0) {
        D->live[0][blockIdx.x] = m.live;
        if (m.live) atomicAdd(&D->nAlive[0], 1);
        if (m.live && (m.P.flags & F_EULER)) atomicAdd(&D->nEuler[0], 1);
    }
}
// When a wait gave up, the kernel left every live member between two of its
// steps: the error is each one's.
__global__ void k_ens_end(EnsMember* M, const EnsDev* D) {
    EnsMember& m = M[blockIdx.x];
    if (threadIdx.x == 0 && m.live && D->fail) m.P.st->error |= ERR_ENSEMBLE;
    __syncthreads();
    copyState(&m.st, m.P.st);
}

struct EnsSmem {
    int offs[ENS_MAX + 1];   // prefix of the current queue's per-member counts
    int offs2[ENS_MAX + 1];  // a second queue of the same phase
};
constexpr int ENS_T = FLOW_T;

// Exclusive prefix of per-member counts get(m) (0 for members not live)
// into offs[0..n]; all threads; offs[n] is the total.
template <class Get>
__device__ __forceinline__ void ensPrefix(int n, Get get, int* offs) {
    const int tid = threadIdx.x;
    constexpr int PER = (ENS_MAX + ENS_T - 1) / ENS_T;  // members per thread
    int v[PER], sum = 0;
    for (int q = 0; q < PER; q++) {
        const int m = tid * PER + q;
        v[q] = m < n ? get(m) : 0;
        sum += v[q];
    }
    // block scan of the per-thread sums (warp shuffles, then warp totals)
    __shared__ int wtot[ENS_T / 32];
    const int lane = tid & 31, w = tid >> 5;
    int x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wtot[w] = x;
    __syncthreads();
    int before = 0;
    for (int k = 0; k < w; k++) before += wtot[k];
    int run = before + x - sum;  // exclusive prefix of this thread
    for (int q = 0; q < PER; q++) {
        const int m = tid * PER + q;
        if (m <= n) offs[m] = run;
        run += v[q];
    }
    if (tid == ENS_T - 1) offs[n] = run;
    __syncthreads();
}

// Member of queue item g: offs[m] <= g < offs[m + 1] (binary search).
__device__ __forceinline__ int ensMember(const int* offs, int n, int g) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (offs[mid] <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}


// The grow item of thread tid for global strip gs of the concatenated strip
// space (prefix offs over the live members): growItem's flags on the
// member's own tile grid.
__device__ __forceinline__ GrowItem ensGrowItem(const EnsArgs& E, const int* offs, int gs,
                                                 bool valid, int& m) {
    GrowItem t;
    t.b = -1;
    t.v = false;
    t.cells = 0;
    t.strip = -1;
    for (int q = 0; q < GROW_LISTS; q++) t.f[q] = 0;
    m = valid ? ensMember(offs, E.n, gs) : 0;
    const int lane = threadIdx.x & 31, r = threadIdx.x & 15;
    const Params& P = E.M[m].P;
    if (valid) {
        t.strip = gs - offs[m];
        if (r < STRIP_TX * STRIP_TY) {
            const int sx = t.strip % P.nSX, sy = t.strip / P.nSX;
            const int bx = STRIP_TX * sx + r % STRIP_TX, by = STRIP_TY * sy + r / STRIP_TX;
            if (bx < P.nBX && by < P.nBY) {
                const int bb = by * P.nBX + bx;
                t.b = bb;
                t.v = tileGrows(P, bb);
                t.cells = tileCells(P, bb);
                t.f[0] = (t.v && t.cells > 0) ? 1 : 0;
                t.f[1] = (P.prevAct[bb] && !t.v) ? 1 : 0;
                t.f[2] = (!t.v && bb != 0) ? 1 : 0;
            }
        }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, t.f[0]);
    const unsigned grp = (bal >> (lane & 16)) & 0xffffu;
    t.f[3] = (valid && r == 0 && grp != 0u) ? 1 : 0;
    return t;
}

// Phase G for all live members: each CTA's chunk of the concatenated strips
// appends to the members' lists (one atomic per half-warp, member and list:
// the two halves of a warp may hold strips of two members) and folds the
// stale speeds of the tiles that are not active this step into the
// member's stale maxima.
__device__ void ensGrow(const EnsArgs& E, const int* offs) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int total = offs[E.n];
    const int L = (total + gridDim.x - 1) / gridDim.x;
    const int s0 = min(total, (int)blockIdx.x * L), s1 = min(total, s0 + L);
    const unsigned half = (lane < 16) ? 0x0000ffffu : 0xffff0000u;
    const int leader = lane & 16;
    for (int rb = s0; rb < s1; rb += ENS_T / 16) {
        const int gs = rb + tid / 16;
        int m;
        const GrowItem t = ensGrowItem(E, offs, gs, gs < s1, m);
        const Params& P = E.M[m].P;
        DevState* st = P.st;
        int* const lists[GROW_LISTS] = {P.act, P.deact, P.inact, P.strips};
        for (int q = 0; q < GROW_LISTS; q++) {
            const unsigned bal = __ballot_sync(0xffffffffu, t.f[q]) & half;
            int base = 0;
            if (lane == leader && bal) base = atomicAdd(&st->appendCnt[q], __popc(bal));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (t.f[q]) lists[q][base + __popc(bal & ((1u << lane) - 1u))] = q == 3 ? t.strip : t.b;
        }
        // cells of the scheduled tiles and stale speeds, per half-warp
        unsigned long long cells = t.f[0] ? (unsigned long long)t.cells : 0ull;
        float smx = 0.f, smy = 0.f;
        if (t.b >= 0) {
            if (t.v) {  // speeds are folded into a cleared entry
                P.mx[t.b] = 0.f;
                P.my[t.b] = 0.f;
            } else {
                smx = P.mx[t.b];
                smy = P.my[t.b];
            }
            if (t.f[0]) listItems(P, t.b, &E.dev->itemCnt[m]);
            P.prevAct[t.b] = (uint8_t)(t.v ? 1 : 0);
        }
        for (int o = 8; o > 0; o >>= 1) {
            cells += __shfl_xor_sync(0xffffffffu, cells, o);
            smx = fmaxf(smx, __shfl_xor_sync(0xffffffffu, smx, o));
            smy = fmaxf(smy, __shfl_xor_sync(0xffffffffu, smy, o));
        }
        if (lane == leader && gs < s1) {
            if (cells) atomicAdd(&st->appendCells, cells);
            if (smx > 0.f) atomicMax(&st->staleBits[0], __float_as_uint(smx));
            if (smy > 0.f) atomicMax(&st->staleBits[1], __float_as_uint(smy));
        }
    }
}

// A warp's copy, in shared memory, of the parameters of the member it works on
// (kept while the member stays the same: the runs of the queue seldom change)
// and of its stage constants.
struct EnsWarp {
    MarchRing ring;
    Params P;
    StageConsts C;
};
constexpr uint32_t ENS_SMEM = FLOW_WARPS * sizeof(EnsWarp);
template <class T>
__device__ __forceinline__ void warpCopy(T& dst, const T& src) {
    static_assert(sizeof(T) % 4 == 0, "copied in words");
    for (int k = threadIdx.x & 31; k < (int)(sizeof(T) / 4); k += 32)
        reinterpret_cast<unsigned*>(&dst)[k] = reinterpret_cast<const unsigned*>(&src)[k];
}

// Uniform rain has instantiations of its own.
template <uint32_t FIX>
struct Fixed {
    static constexpr uint32_t value = FIX;
};
template <class Fn>
__device__ __forceinline__ bool byFlags(const Params& P, Fn fn) {
    return (P.flags & CELL_FLAGS) == FIX_RAIN && P.nsrc == 0 ? fn(Fixed<FIX_RAIN>{}) : fn(Fixed<0>{});
}

// The ensemble's step loop (one cooperative launch).
__global__ void __launch_bounds__(ENS_T, 1) k_ensemble(EnsArgs E) {
    extern __shared__ __align__(128) unsigned char ensRaw[];
    __shared__ EnsSmem Q;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = E.n;
    EnsWarp& W = reinterpret_cast<EnsWarp*>(ensRaw)[warp];
    MarchRing& S = W.ring;
    int mine = -1;  // member whose parameters W.P holds
    EnsDev* D = E.dev;
    if (lane == 0) {
        for (int k = 0; k < MNS; k++) mbar_init(&S.bar[k], 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t par = 0u;
    unsigned barTarget = 0u;
    const int nW = FLOW_WARPS * (int)gridDim.x, gw = warp * (int)gridDim.x + (int)blockIdx.x;
    DevState* st0 = E.M[0].P.st;  // barrier timeouts are recorded in member 0
    if (blockIdx.x == 0 && tid == 0) D->times.t0 = globalTimerNs();  // before any member can finish
#define ENS_SYNC()                                                         \
    if (!gridSync(&D->bar, barTarget, st0, false, nullptr, E.polls)) {     \
        if (tid == 0) D->fail = 1;                                         \
        return;                                                            \
    }                                                                      \
    (void)0
    for (int step = 0;; step++) {
        const int cur = step & 1;
        if (D->nAlive[cur] == 0) return;  // every CTA reads the same count
        const int* live = D->live[cur];
        // ---- T: re-wet tracking of the members with gridded rain or surge
        // and inactive tiles (a member without an inactive list -- last
        // stepped by the persistent loop's tile table -- scans its tiles)
        ensPrefix(n, [&](int m) {
            if (!live[m] || !(E.M[m].P.flags & (F_RAIN_G | F_SURGE)) || (step > 0 && D->all[m])) return 0;
            const int k = E.M[m].P.st->nInact;
            return k >= 0 ? k : E.M[m].P.gridSize - 1;
        }, Q.offs);
        // (the same total and count in every CTA)
        bool guess = step > 0 && Q.offs[n] == 0 && D->nEuler[cur] == 0;
        if (Q.offs[n] > 0) {
            int of = -1;  // member of the factors
            float fac0 = 0.f, fac2 = 0.f;
            for (int g = gw; g < Q.offs[n]; g += nW) {
                const int m = ensMember(Q.offs, n, g);
                const Params& P = E.M[m].P;
                if (m != of) trackFactors(P, fac0, fac2);
                of = m;
                const bool listed = P.st->nInact >= 0;
                const int b = listed ? P.inact[g - Q.offs[m]] : g - Q.offs[m] + 1;
                if (listed || !P.prevAct[b]) trackTile(P, b, fac0, fac2);
            }
            ENS_SYNC();
        }
        // the other parity's counts were last read in the previous step
        if (tid == 0 && blockIdx.x == 0) D->nAlive[cur ^ 1] = D->nEuler[cur ^ 1] = D->changed[cur ^ 1] = 0;
        Led L;  // members keep no ledger (rift_ensemble_create)
        bool begun = false;
    flux:
        // ---- G: grow, stale maxima
        if (!guess) {
            for (int m = gw; m < n; m += nW)
                if (live[m] && lane == 0) {
                    DevState* st = E.M[m].P.st;
                    st->max_bits[0] = st->max_bits[1] = 0u;
                    if (step == 0) D->consts[m][0] = stageConsts<1>(E.M[m].P);  // S reads what no step changes
                }
            ensPrefix(n, [&](int m) { return live[m] ? E.M[m].P.nSX * E.M[m].P.nSY : 0; }, Q.offs);
            ensGrow(E, Q.offs);
            ENS_SYNC();  // the counts are final after the barrier
        }
        const int* const nPairs = guess ? D->nItems : D->itemCnt;
        auto isAll = [&](int m) {
            const Params& P = E.M[m].P;
            return guess ? D->all[m] != 0
                         : P.st->appendCnt[0] == ((P.nx - 4 + TW - 1) / TW) * ((P.ny - 4 + TH - 1) / TH);
        };
        ensPrefix(n, [&](int m) {
            if (!live[m]) return 0;
            return isAll(m) ? segCount(E.M[m].P.nx) * (E.M[m].P.ny - 4) : nPairs[m] * TH;
        }, Q.offs);
        const int nRows = Q.offs[n], nUse = min(nW, (nRows + 1) / 2);
        // fn(member, segment, j0, j1) on this warp's run of the queue, until it
        // returns false, with the member's stage constants k in W.C.  (all:
        // read from the sets, which D publishes; phases 1 and 2 follow D)
        auto items = [&](bool published, int kC, auto fn) {
            if (gw >= nUse) return;
            int r = (int)((long long)nRows * gw / nUse);
            const int end = (int)((long long)nRows * (gw + 1) / nUse);
            while (r < end) {
                const int m = ensMember(Q.offs, n, r), local = r - Q.offs[m];
                const Params& P = W.P;
                __syncwarp();
                if (m != mine) warpCopy(W.P, E.M[m].P);
                warpCopy(W.C, D->consts[m][kC]);
                mine = m;
                __syncwarp();
                if (W.P.flags & F_EULER) {  // phase 1 writes the step's result in place
                    if (lane == 0) {
                        W.P.B = W.P.A;
                        W.C.Fout = W.P.FA;
                    }
                    __syncwarp();
                }
                const bool all = published ? D->all[m] != 0 : isAll(m);
                const int H = all ? P.ny - 4 : TH, col = local / H, j = local % H, len = min(end - r, H - j);
                const int nSeg = segCount(P.nx), id = all ? col : P.items[col];
                const int j0 = 2 + j + (all ? 0 : TH * (id / nSeg)), j1 = min(j0 + len, P.ny - 2);
                if (j0 < j1 && !fn(m, id % nSeg, j0, j1)) {
                    if (lane == 0) {
                        atomicOr(&P.st->error, ERR_TMA_TIMEOUT);
                        D->fail = 1;
                    }
                    return;
                }
                r += len;
            }
        };
        // ---- S: start of each member's step (the last warps); the stage-1
        // fluxes give the speeds, and each cell's divergence (bed-slope source
        // folded in) waits in the member's divergence planes for the update
        // after dt; U* re-sync of the deactivated tiles
        if (!begun)
            for (int m = nW - 1 - gw; m < n; m += nW)
                if (live[m]) {
                    beginStepRates(E.M[m].P, E.M[m].P.st);
                    if (lane == 0) beginStepCounts(E.M[m].P.st);
                }
        begun = true;
        items(false, 0, [&](int m, int seg, int j0, int j1) {
            const Params& P = W.P;
            auto on = [&](int by, int bx) { return bx >= 0 && P.prevAct[by * P.nBX + bx] != 0; };
            float tmx = 0.f, tmy = 0.f;
            const bool ok = marchRows<1, 0, false, false>(P, W.C, &E.M[m].maps[0], &E.M[m].maps[2], S,
                                                   par, seg, j0, j1, on, false, L, tmx, tmy, false);
            tmx = warpMax(tmx);
            tmy = warpMax(tmy);
            if (lane == 0) {
                atomicMax(&P.st->max_bits[0], __float_as_uint(tmx));
                atomicMax(&P.st->max_bits[1], __float_as_uint(tmy));
            }
            return ok;
        });
        if (guess) {  // tiles whose activity changed
            ensPrefix(n, [&](int m) { return live[m] ? E.M[m].P.gridSize : 0; }, Q.offs2);
            bool diff = false;
            for (int g = gw * 32 + lane; g < Q.offs2[n]; g += nW * 32) {
                const int m = ensMember(Q.offs2, n, g), b = g - Q.offs2[m];
                diff |= tileGrows(E.M[m].P, b) != (E.M[m].P.prevAct[b] != 0);
            }
            if (__any_sync(FULL, diff) && lane == 0) atomicOr(&D->changed[cur], 1);
        } else {
            ensPrefix(n, [&](int m) { return live[m] ? D->itemCnt[m] : 0; }, Q.offs2);
            for (int k = blockIdx.x * ENS_T + tid; k < Q.offs2[n]; k += gridDim.x * ENS_T) {
                const int m = ensMember(Q.offs2, n, k);
                E.M[m].P.itemStamp[E.M[m].P.items[k - Q.offs2[m]]] = 0;  // for the next grow
            }
            __syncthreads();
            ensPrefix(n, [&](int m) { return live[m] ? E.M[m].P.st->appendCnt[1] : 0; }, Q.offs2);
            for (int g = blockIdx.x; g < Q.offs2[n]; g += gridDim.x) {
                const int m = ensMember(Q.offs2, n, g);
                resyncTile(E.M[m].P, E.M[m].P.deact[g - Q.offs2[m]]);
            }
        }
        if (guess) {
            ENS_SYNC();
            if (ld_relaxed_gpu((const unsigned*)&D->changed[cur]) != 0u) {
                guess = false;  // every CTA reads the same flag
                goto flux;
            }
            if (D->fail) return;
        } else {
            ENS_SYNC();
            if (D->fail) return;
        }
        // ---- D: dt of each member, list sizes, liveness of its next step
        for (int m = blockIdx.x + gridDim.x * tid; m < n; m += gridDim.x * ENS_T) {
            int next = 0;
            if (live[m]) {
                const Params& P = E.M[m].P;
                DevState* st = P.st;
                if (!guess) {  // the grow's sets
                    D->stale[m][0] = st->staleBits[0];
                    D->stale[m][1] = st->staleBits[1];
                    D->cells[m] = st->appendCells;
                    D->nItems[m] = D->itemCnt[m];
                    D->all[m] = isAll(m);
                    D->itemCnt[m] = 0;
                    st->staleBits[0] = st->staleBits[1] = 0u;
                    publishGrow(st);
                } else {
                    st->activeCells += D->cells[m];
                    st->nDeact = 0;
                }
                const float mx = __uint_as_float(max(st->max_bits[0], D->stale[m][0]));
                const float my = __uint_as_float(max(st->max_bits[1], D->stale[m][1]));
                st->max_bits[0] = st->max_bits[1] = 0u;
                computeDt(P, st, (double)mx, (double)my);
                // the step's stage constants, once per member (the FP64
                // conversions stay out of the item loops)
                D->consts[m][0] = stageConsts<1>(P);
                D->consts[m][1] = stageConsts<2>(P);
                next = (st->t < st->t_stop && st->steps_done < E.maxSteps) ? 1 : 0;
                if (!next) st->stop = 1;
            }
            D->live[cur ^ 1][m] = next;
            if (next) atomicAdd(&D->nAlive[cur ^ 1], 1);
            if (next && (E.M[m].P.flags & F_EULER)) atomicAdd(&D->nEuler[cur ^ 1], 1);
        }
        if (D->nEuler[cur] > 0) {
            ensPrefix(n, [&](int m) { return live[m] && (E.M[m].P.flags & F_EULER) ? E.M[m].P.gridSize : 0; },
                      Q.offs2);
            for (int g = blockIdx.x * ENS_T + tid; g < Q.offs2[n]; g += gridDim.x * ENS_T) {
                const int m = ensMember(Q.offs2, n, g), b = g - Q.offs2[m];
                const Params& P = E.M[m].P;
                if (P.prevAct[b] && tileCells(P, b) > 0) P.wet[b] = 0;
            }
        }
        ENS_SYNC();
        // ---- 1: the rest of RK stage 1 from U^n and the stored divergence
        items(true, 0, [&](int, int seg, int j0, int j1) {
            const Params& P = W.P;
            const StageConsts& C = W.C;
            auto on = [&](int by, int bx) { return bx >= 0 && P.prevAct[by * P.nBX + bx] != 0; };
            return byFlags(P, [&](auto fix) {
                updateRows<decltype(fix)::value, true>(P, C, seg, j0, j1, on, false, L);
                return true;
            });
        });
        ENS_SYNC();
        // ---- 2: RK stage 2 (an Euler member's step is done)
        items(true, 1, [&](int m, int seg, int j0, int j1) {
            const Params& P = W.P;
            const StageConsts& C = W.C;
            if (C.euler) return true;
            auto on = [&](int by, int bx) { return bx >= 0 && P.prevAct[by * P.nBX + bx] != 0; };
            float tmx = 0.f, tmy = 0.f;
            return byFlags(P, [&](auto fix) {
                return marchRows<2, decltype(fix)::value, false, false>(P, C, &E.M[m].maps[1],
                                                                 &E.M[m].maps[2], S, par, seg, j0, j1,
                                                                 on, false, L, tmx, tmy, false);
            });
        });
        ENS_SYNC();
        if (D->fail) return;
        // members whose last step this iteration was: its end on the device clock
        for (int m = blockIdx.x * ENS_T + tid; m < n; m += gridDim.x * ENS_T)
            if (live[m] && !D->live[cur ^ 1][m]) D->times.tDone[m] = globalTimerNs();
    }
#undef ENS_SYNC
}

}  // namespace rift
