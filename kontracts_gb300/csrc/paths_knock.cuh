// paths_knock.cuh — the path kernel for one-flow knock-outs and knock-ins
// (k_knock).
//
// Serves GBM contracts on a uniform grid with one flow after t = 0, closed
// form, paid at the last step, that barriers armed at t = 0 drop (up-and-out,
// down-and-out, double knock-out) or that one barrier must be crossed to
// acquire (up-and-in, down-and-in). Such a path needs no event handler: only
// the extremes of its log-spot against the barriers.
//
// A block of threads holds up to knock_list paths and walks them segment by
// segment (some Philox blocks of 4 steps), 32 paths a warp in step; the
// survivors of a segment move to the front of the next list, so the warps stay
// full while paths are knocked out. The steps after a path's hit, up to the
// segment's end, are all that is simulated in vain. Every lane of a warp is at
// the same step: the shared Philox words are one broadcast read, and the step
// loop holds the bare simulation and one three-input maximum per two steps.
// A knock-in walks its paths to the end the same way, without lists.
// Paths are the same bit for bit as k_lean's, which tests the window after
// every block, batches the events of several lanes and walks a block with an
// event twice.
//
// What bounds it: the FMA pipe, as the bare loop (PhiloxTail): a warp's block
// of 4 steps takes 121 cycles, 115 in the bare loop; the steps simulated in
// vain are 11 % more (8.53e8 for 7.68e8 on the call below). Measured on the up-and-out call of 4M paths x 365
// steps: 1315 us on k_lean, 823 us with a lane per path that takes its next
// path at the end of a round of 8 blocks, 676 us here; the down-and-in put of
// 1,000,001 paths x 189 steps: 477 us on k_lean, 141 us here.
#pragma once
#include "paths_lean.cuh"

namespace kx {

constexpr int KNOCK_TAB = 256;  // longest grid served: 4 * KNOCK_TAB steps
// Philox blocks between two looks at the barriers, for a path of nb blocks: a
// sixth of it. Shorter segments simulate less in vain but their barriers and
// list moves cost more (92 blocks: 5 at a time 786 us, 8 708, 12 704, 16 680;
// 126 blocks and fewer hits: 16 as good as 12); a short path still gets looked at.
__device__ __forceinline__ int knock_segment(int nb) { return min(16, max(4, (nb + 5) / 6)); }
template <class Real>
constexpr int knock_list() { return sizeof(Real) == 4 ? 2048 : 1024; }  // paths a block holds (32 / 24 KB, twice)

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

// Steps of the Philox blocks whose shared words are e0 .. e1 - 1: the log-spot
// and, where a barrier is up (down), the maximum (minimum) so far.
template <class Real, bool UP, bool DN>
__device__ __forceinline__ void knock_blocks(const uint4 *e0, const uint4 *e1, uint64_t pw, const PhiloxTail &keys,
                                             Real c0, Real c1, Real &y, Real &mx, Real &mn) {
#pragma unroll 2
    for (const uint4 *e = e0; e < e1; ++e) {
        const uint4 w = philox_tail(*e, pw, keys);
        Real zz[4], ys[4];
        box_muller(w.x, w.y, zz[0], zz[1]);
        box_muller(w.z, w.w, zz[2], zz[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            y = gbm_step(y, c0, c1, zz[j]);
            ys[j] = y;
        }
        if (UP) mx = max3(max3(mx, ys[0], ys[1]), ys[2], ys[3]);
        if (DN) mn = min3(min3(mn, ys[0], ys[1]), ys[2], ys[3]);
    }
}

// The same with the barriers' sides as (warp-uniform) arguments, `rest` steps
// (0 to 3) of the block after them included.
template <class Real>
__device__ __forceinline__ void knock_walk(bool up, bool dn, const uint4 *e0, const uint4 *e1, int rest, uint64_t pw,
                                           const PhiloxTail &keys, Real c0, Real c1, Real &y, Real &mx, Real &mn) {
    if (up && !dn) knock_blocks<Real, true, false>(e0, e1, pw, keys, c0, c1, y, mx, mn);
    else if (dn && !up) knock_blocks<Real, false, true>(e0, e1, pw, keys, c0, c1, y, mx, mn);
    else knock_blocks<Real, true, true>(e0, e1, pw, keys, c0, c1, y, mx, mn);
    if (rest) {
        const uint4 w = philox_tail(*e1, pw, keys);
        Real zz[4];
        box_muller(w.x, w.y, zz[0], zz[1]);
        box_muller(w.z, w.w, zz[2], zz[3]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (j < rest) {
                y = gbm_step(y, c0, c1, zz[j]);
                mx = fmax(mx, y);
                mn = fmin(mn, y);
            }
    }
}

// The value of the one flow j paid at the last step with log-spot y
// (static_event's amounts), added to the flows of t = 0.
template <class Real>
__device__ __forceinline__ double knock_pay(const StaticDev &T, int j, Real s0, double df, Real y, double pv0) {
    double amt = T.f_sign[j];
    if (T.f_fast[j] != FA_NONE) {
        const Real S = spot_of<Real>(s0, y);
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
    return __dadd_rn(pv0, __dmul_rn(amt, df));
}

template <class Real, int MINB>
__global__ void __launch_bounds__(KX_BLOCK, MINB) k_knock(const PathArgs A) {
    constexpr int CAP = knock_list<Real>();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ uint4 tab[KNOCK_TAB + 1];
    __shared__ uint32_t lp[2][CAP];  // the paths alive, ...
    __shared__ Real ly[2][CAP];      // ... and their log-spots
    __shared__ uint32_t alive[2];
    __shared__ uint32_t item;
    int cur = -1;
    PhiloxTail keys{};
    Real c0 = 0, c1 = 0, s0 = 1, hi = 0, lo = 0;
    uint32_t seed_lo = 0;
    uint64_t pv_off = 0;
    double pv0 = 0.0, df = 0.0;
    int last = 0, flow = 0;
    bool up = false, dn = false, over = false;  // over: every path is settled at t = 0
    const StaticDev *T = nullptr;
    unsigned long long steps = 0;
    while (true) {
        __syncthreads();  // the last item's lists and table are done with
        if (threadIdx.x == 0) item = atomicAdd(A.item_counter, 1u);
        __syncthreads();
        if (item >= A.n_items) break;
        const WorkItem w = fetch_item(A, (int)item);
        if (w.contract != cur) {
            cur = w.contract;
            const ContractDev &C = A.cons[cur];
            T = static_cast<const StaticDev *>(A.statics) + cur;
            keys = philox_tail_keys(C.seed);
            seed_lo = (uint32_t)C.seed;
            c0 = pick<Real>(C.uc0, C.uc0f);
            c1 = pick<Real>(C.uc1, C.uc1f);
            s0 = pick<Real>(C.s0[0], C.s0f[0]);
            pv_off = C.pv_off;
            const double *D = A.disc + C.disc_off;
            last = T->ev_step[T->n_ev - 1];
            flow = __ffs(T->ev_pay[T->n_ev - 1]) - 1;
            df = D[last];
            // step 0 is the same for every path
            if (T->knock_in) {
                static_window<Real>(*T, T->ev_arm[0], hi, lo);
                up = (T->ev_arm[0] & T->up_mask) != 0u;
                dn = !up;
                pv0 = 0.0;
                over = false;
            } else {  // barriers armed and tested, flows of t = 0 paid
                SLane sl{0u, T->all_flows, 0, 0.0};
                static_event<Real>(*T, D, s0, Real(0), 0, sl);
                static_window<Real>(*T, sl.live, hi, lo);
                up = (sl.live & T->up_mask) != 0u;
                dn = (sl.live & ~T->up_mask) != 0u;
                pv0 = sl.pv;
                over = sl.rem == 0u;
            }
            for (int b = threadIdx.x; b < (last + 3) / 4; b += KX_BLOCK)
                tab[b] = philox_block_words((uint32_t)b, C.stream, C.seed);
            __syncthreads();
        }
        const uint32_t first = (uint32_t)w.first, n = (uint32_t)w.count;
        const int nb = last / 4, rest = last % 4, seg = knock_segment(nb);
        if (over || T->knock_in) {
            for (uint32_t i0 = (uint32_t)warp * 32u; i0 < n; i0 += KX_BLOCK) {
                const uint32_t path = first + i0 + (uint32_t)lane;
                double v = pv0;
                if (!over) {
                    Real y = Real(0), mx = Real(0), mn = Real(0);  // t = 0: y = 0
                    knock_walk<Real>(up, dn, tab, tab + nb, rest, philox_path_word(path, seed_lo), keys, c0, c1, y, mx, mn);
                    if (up ? mx >= hi : mn <= lo) v = knock_pay<Real>(*T, flow, s0, df, y, pv0);
                }
                if (i0 + (uint32_t)lane < n) A.pv[pv_off + path] = v;
            }
            if (threadIdx.x == 0 && !over) steps += (unsigned long long)n * (unsigned)last;
            continue;
        }
        int q = 0;  // list in use
        uint32_t m = n;
        for (int b = 0; m != 0u;) {
            const int b1 = min(nb, b + seg);
            const bool end = b1 == nb;  // the segment with the last step
            if (threadIdx.x == 0) alive[q ^ 1] = 0u;
            __syncthreads();
            for (uint32_t i0 = (uint32_t)warp * 32u; i0 < m; i0 += KX_BLOCK) {
                const uint32_t i = i0 + (uint32_t)lane;
                const bool on = i < m;
                uint32_t path = first + i;
                Real y = Real(0);
                if (b && on) {
                    path = lp[q][i];
                    y = ly[q][i];
                }
                Real mx = Real(-INFINITY), mn = Real(INFINITY);
                knock_walk<Real>(up, dn, tab + b, tab + b1, end ? rest : 0, philox_path_word(path, seed_lo), keys, c0, c1,
                                 y, mx, mn);
                const bool hit = (up && mx >= hi) || (dn && mn <= lo);
                if (end) {
                    if (on) A.pv[pv_off + path] = hit ? pv0 : knock_pay<Real>(*T, flow, s0, df, y, pv0);
                } else {
                    if (on && hit) A.pv[pv_off + path] = pv0;
                    const unsigned keep = __ballot_sync(FULL, on && !hit);
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&alive[q ^ 1], (uint32_t)__popc(keep));
                    at = __shfl_sync(FULL, at, 0) + (uint32_t)__popc(keep & ((1u << lane) - 1u));
                    if (on && !hit) {
                        lp[q ^ 1][at] = path;
                        ly[q ^ 1][at] = y;
                    }
                }
            }
            __syncthreads();
            // every path that entered the segment, knocked out in it or not
            if (threadIdx.x == 0) steps += (unsigned long long)m * (unsigned)(end ? last - 4 * b : 4 * (b1 - b));
            if (end) break;
            q ^= 1;
            m = alive[q];
            b = b1;
        }
    }
    if (threadIdx.x == 0 && steps) atomicAdd(A.steps_done, steps);
}

// k_knock in a precision.
const void *knock_kernel(bool f64);

}  // namespace kx
