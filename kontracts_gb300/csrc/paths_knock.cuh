// paths_knock.cuh — the path kernel for one-flow knock-outs (k_knock).
//
// Serves static schedules whose barriers are all armed at t = 0, whose one
// flow after t = 0 is dropped by any of them, on a uniform grid (up-and-out,
// down-and-out, double knock-out calls and puts). Such a path needs no event
// handler: it pays its flow at the last step unless the extremes of its
// log-spot crossed a barrier. A lane therefore steps KNOCK_ROUND Philox
// blocks without a test, keeping only the running maximum (and minimum), and
// looks at the barriers once per round; a knocked-out path wastes half a
// round on average. Lanes are at different steps (a finished lane takes its
// next path at the end of the round), so a warp keeps the shared Philox words
// of all the contract's blocks in shared memory. Paths are the same bit for
// bit as k_lean's, which tests the window after every block, batches the
// events of several lanes and walks a block with an event twice.
//
// What bounds it: the FMA pipe, as the bare loop (paths_sync.cuh); what is
// left is the finished lanes that wait for their round to end. Measured on
// the up-and-out call of 4M paths x 365 steps: 1315 us on k_lean, 823 us here.
#pragma once
#include "paths_lean.cuh"

namespace kx {

constexpr int KNOCK_TAB = 256;   // longest grid served: 4 * KNOCK_TAB steps
constexpr int KNOCK_ROUND = 8;   // Philox blocks (4 steps each) between two looks at the barriers

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ double max3(double a, double b, double c) { return fmax(a, fmax(b, c)); }
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ double min3(double a, double b, double c) { return fmin(a, fmin(b, c)); }

// The lane's path between two rounds. ys: the log-spots of its last block
// (ys[3]: where the next one starts); mx, mn: extremes of all its steps, mxp, mnp: of the blocks before the last.
template <class Real>
struct KnockLane {
    Real mx, mn, mxp, mnp;
    Real ys[4];
    int b;  // next block
    uint64_t pw;
};

template <class Real, bool UP, bool DN>
__device__ __forceinline__ void knock_round(KnockLane<Real> &L, const uint4 *tab, const PhiloxTail &keys, int nb,
                                            Real c0, Real c1) {
#pragma unroll 1
    for (int q = 0; q < KNOCK_ROUND; ++q) {
        if (L.b >= nb) break;
        const uint4 w = philox_tail(tab[L.b], L.pw, keys);
        Real zz[4];
        box_muller(w.x, w.y, zz[0], zz[1]);
        box_muller(w.z, w.w, zz[2], zz[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) L.ys[j] = gbm_step(j ? L.ys[j - 1] : L.ys[3], c0, c1, zz[j]);
        if (UP) {
            L.mxp = L.mx;
            L.mx = max3(max3(L.mx, L.ys[0], L.ys[1]), L.ys[2], L.ys[3]);
        }
        if (DN) {
            L.mnp = L.mn;
            L.mn = min3(min3(L.mn, L.ys[0], L.ys[1]), L.ys[2], L.ys[3]);
        }
        ++L.b;
    }
}

// What a warp needs of its contract only when a path starts or ends, kept in
// shared memory (the step loop has no registers to spare for it).
template <class Real>
struct KnockContract {
    const StaticDev *T;
    uint64_t pv_off;
    double pv0, df;  // the value of t = 0; the discount of the flow
    Real s0, hi, lo;
    uint32_t seed_lo;
    int last, flow, over;  // over: every path ends at t = 0
};

// The value of the one flow j paid at the last step with log-spot y
// (static_event's amounts), added to the flows of t = 0.
template <class Real>
__device__ __forceinline__ double knock_pay(const KnockContract<Real> &C, Real y) {
    const StaticDev &T = *C.T;
    const int j = C.flow;
    double amt = T.f_sign[j];
    if (T.f_fast[j] != FA_NONE) {
        const Real S = spot_of<Real>(C.s0, y);
        const Real K = (Real)T.f_k[j];
        Real r;
        switch (T.f_fast[j]) {
        case FA_CALL: r = fmax(S - K, Real(0)); break;
        case FA_PUT: r = fmax(K - S, Real(0)); break;
        case FA_SPOT: r = S; break;
        default: r = K; break;
        }
        amt = (double)(((T.f_neg >> j) & 1u) ? -r : r);
    }
    return __dadd_rn(C.pv0, __dmul_rn(amt, C.df));
}

template <class Real, int MINB>
__global__ void __launch_bounds__(KX_BLOCK, MINB) k_knock(const PathArgs A) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ uint4 tabs[KX_BLOCK / 32][KNOCK_TAB];
    uint4 *tab = tabs[threadIdx.x >> 5];
    __shared__ KnockContract<Real> contracts[KX_BLOCK / 32];
    KnockContract<Real> &K = contracts[threadIdx.x >> 5];
    // warp-uniform: the work item and its contract
    int cur = -1, pend = -1;
    uint64_t nx = 0, end = 0;
    bool drained = false;
    PhiloxTail keys{};
    int nb = 0;
    Real c0 = 0, c1 = 0;
    bool up = false, dn = false;
    // lane
    bool busy = false;
    uint32_t path = 0;
    KnockLane<Real> L{};
    uint32_t steps = 0;

    while (true) {
        // ---- hand paths to idle lanes ----
        unsigned idle = __ballot_sync(FULL, !busy);
        while (idle) {
            if (nx >= end) {
                int it = pend;
                if (it < 0) {
                    if (drained) break;
                    if (lane == 0) it = (int)atomicAdd(A.item_counter, 1u);
                    it = __shfl_sync(FULL, it, 0);
                    if (it >= (int)A.n_items) {
                        drained = true;
                        break;
                    }
                }
                const WorkItem w = fetch_item(A, it);
                if (w.contract != cur) {
                    if (cur >= 0 && idle != FULL) {  // finish the current contract first
                        pend = it;
                        break;
                    }
                    cur = w.contract;
                    const ContractDev &C = A.cons[cur];
                    const StaticDev &T = static_cast<const StaticDev *>(A.statics)[cur];
                    keys = philox_tail_keys(C.seed);
                    c0 = pick<Real>(C.uc0, C.uc0f);
                    c1 = pick<Real>(C.uc1, C.uc1f);
                    // step 0 is the same for every path: barriers armed and tested, flows of t = 0 paid
                    const double *D = A.disc + C.disc_off;
                    const Real s0 = pick<Real>(C.s0[0], C.s0f[0]);
                    SLane sl{0u, T.all_flows, 0, 0.0};
                    static_event<Real>(T, D, s0, Real(0), 0, sl);
                    Real hi, lo;
                    static_window<Real>(T, sl.live, hi, lo);
                    up = (sl.live & T.up_mask) != 0u;
                    dn = (sl.live & ~T.up_mask) != 0u;
                    const int last = T.ev_step[T.n_ev - 1];
                    nb = (last + 3) / 4;
                    __syncwarp();
                    if (lane == 0)
                        K = KnockContract<Real>{&T, C.pv_off, sl.pv, D[last], s0, hi, lo, (uint32_t)C.seed, last,
                                                __ffs(T.ev_pay[T.n_ev - 1]) - 1, sl.rem == 0u ? 1 : 0};
                    for (int b = lane; b < nb; b += 32) tab[b] = philox_block_words((uint32_t)b, C.stream, C.seed);
                    __syncwarp();
                    L.b = nb;
                }
                pend = -1;
                nx = w.first;
                end = w.first + w.count;
                if (K.over) {  // knocked out (or paid in full) at t = 0
                    for (uint64_t p = nx + lane; p < end; p += 32) A.pv[K.pv_off + p] = K.pv0;
                    nx = end;
                }
                continue;
            }
            const int nidle = __popc(idle);
            const uint64_t avail = end - nx;
            const int take = avail < (uint64_t)nidle ? (int)avail : nidle;
            const int rank = __popc(idle & lt);
            if (!busy && rank < take) {
                path = (uint32_t)nx + (uint32_t)rank;
                busy = true;
                L.ys[3] = Real(0);
                L.mx = Real(-INFINITY);
                L.mn = Real(INFINITY);
                L.b = 0;
                L.pw = philox_path_word(path, K.seed_lo);
            }
            nx += (uint64_t)take;
            idle = __ballot_sync(FULL, !busy);
        }
        if (__ballot_sync(FULL, busy) == 0u) {
            if (drained && pend < 0 && nx >= end) break;
            continue;
        }
        // ---- one round (an idle lane has b == nb and steps nothing) ----
        const int b_in = L.b;
        if (up && !dn) knock_round<Real, true, false>(L, tab, keys, nb, c0, c1);
        else if (dn && !up) knock_round<Real, false, true>(L, tab, keys, nb, c0, c1);
        else knock_round<Real, true, true>(L, tab, keys, nb, c0, c1);
        __syncwarp();
        // ---- paths that ended: knocked out, or at the last step ----
        if (busy) {
            const bool expired = L.b >= nb;
            const int last = K.last;
            Real yl = L.ys[3], mx = L.mx, mn = L.mn;
            if (expired && last < 4 * nb) {  // the steps of the last block that the path has
                const int r = last - 4 * (nb - 1);
                yl = r == 1 ? L.ys[0] : r == 2 ? L.ys[1] : L.ys[2];
                const Real a = L.ys[0], b = r >= 2 ? L.ys[1] : a, c = r >= 3 ? L.ys[2] : a;
                mx = fmax(L.mxp, max3(a, b, c));
                mn = fmin(L.mnp, min3(a, b, c));
            }
            const bool hit = (up && mx >= K.hi) || (dn && mn <= K.lo);
            if (hit || expired) {
                A.pv[K.pv_off + path] = hit ? K.pv0 : knock_pay<Real>(K, yl);
                // a knocked-out path counts the rounds it survived
                steps += hit ? 4u * (unsigned)b_in : (unsigned)last;
                busy = false;
                L.b = nb;
            }
        }
    }
    unsigned long long tot = steps;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(FULL, tot, o);
    if (lane == 0 && tot) atomicAdd(A.steps_done, tot);
}

// k_knock in a precision.
const void *knock_kernel(bool f64);

}  // namespace kx
