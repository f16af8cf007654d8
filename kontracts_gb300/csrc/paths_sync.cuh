// paths_sync.cuh — the path kernel for static schedules without barriers
// (k_sync): European and Bermudan payoffs, averages, running extrema.
//
// No price condition can end or change such a path, so the lanes of a warp
// walk their 32 paths in step: the schedule's events, the accumulator window
// and the Philox block are the same for all of them, and the step loop holds
// nothing but the model step and the accumulator. k_lean serves these
// contracts too, but pays for its freedom to stop each lane elsewhere: the
// hand-out of paths, the window and limit tests, the event ballots and a
// second walk of every block with an event. Every path is the same bit for
// bit (the model step, the accumulator and the events are k_lean's own).
//
// What bounds it: the FMA pipe (15 wide multiplies of a Philox block at 4
// cycles a warp, 14 products of Box-Muller, the steps and, for an average, the
// exponential's product and Kahan's four additions per step), with the XU and
// the issue slots close behind. The loop is unrolled over two Philox blocks:
// their independent chains are what the scheduler overlaps. Measured: 9.5e11
// steps/s for averages (500,003 paths x 328 steps in 172 us; 313 us, 5.2e11, on
// k_lean).
#pragma once
#include "paths_lean.cuh"

namespace kx {

// e^y of one step's log-spot. TAME: the caller knows that no e^y of the block is
// subnormal (y > -80), and e^y = 2^(y log2 e) is taken from the hardware's 2^x.
template <bool TAME>
__device__ __forceinline__ float block_exp(float y) {
    if (!TAME) return fast_exp<float>(y);
    return ex2_approx(__fmul_rn(y, 1.4426950408889634f));  // log2 e
}
template <bool TAME>
__device__ __forceinline__ double block_exp(double y) { return exp(y); }

template <class Real, int AK, bool TAME>
__device__ __forceinline__ void block_acc(const Real (&ys)[4], int n, Real s0, Real &av, Real &ac) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j < n) acc_add<Real, AK>(AK, av, ac, mul_rn(s0, block_exp<TAME>(ys[j])));
}

// Where a path's normals come from: Philox and Box-Muller in registers, or
// (SH, FP64) a table of the launch's normals that k_normals wrote. GB300 runs
// FP64 at 1/64 of its FP32 rate, so a pair of FP64 normals costs two to three
// Heston steps, and reading it back is free next to that: a launch whose
// contracts all draw the same stream (the candidates of a calibration, the
// reprices of a bump) draws it once.
template <class Real, bool SH>
struct SyncDraws {
    uint4 *tab;  // SYNC_TAB entries of this warp
    uint64_t pw;
    const double *z;  // SH: draw 0 of this lane's path
    uint64_t ld;
    // the first n (of four) normals of block b
    __device__ __forceinline__ void block(const PhiloxTail &keys, const uint4 *e, int b, int n, Real (&zz)[4]) const {
        if (SH) {
            const double *p = z + (uint64_t)(4 * b) * ld;
#pragma unroll
            for (int j = 0; j < 4; ++j) zz[j] = j < n ? (Real)p[(uint64_t)j * ld] : Real(0);
        } else {
            const uint4 w = philox_tail(*e, pw, keys);
            box_muller(w.x, w.y, zz[0], zz[1]);
            if (n > 2) box_muller(w.z, w.w, zz[2], zz[3]);
            else zz[2] = zz[3] = Real(0);
        }
    }
};

// One whole Philox block of a path: SPB steps with the coefficients (c0, c1)
// of R (UNI: uc0, uc1), every step's spot added to the accumulator (AK >= 0).
template <class Real, int MODEL, bool UNI, int AK, bool TAME, bool SH>
__device__ __forceinline__ void sync_block(const SyncDraws<Real, SH> &draws, const uint4 *e, int b,
                                           const PhiloxTail &keys, const StepRec<Real> *Rk, Real uc0, Real uc1,
                                           const HestonPar<Real> &hp, Real s0, Real &y, Real &v, Real &av, Real &ac) {
    constexpr int SPB = lean_spb<MODEL>();
    Real zz[4], ys[4];
    draws.block(keys, e, b, 4, zz);
#pragma unroll
    for (int j = 0; j < SPB; ++j) {
        Real c0 = uc0, c1 = uc1;
        if (!UNI) {
            const StepRec<Real> rec = Rk[j];
            c0 = rec.c0;
            c1 = rec.c1;
        }
        lean_model_step<Real, MODEL>(hp, c0, c1, zz, j, y, v);
        ys[j] = y;
    }
    if (AK >= 0) block_acc<Real, AK, TAME>(ys, SPB, s0, av, ac);
}

// The normals a path takes for a block of which `left` draws remain to its last step: from a table
// those alone (its last row may be the first of them), in registers a pair or a whole block.
__host__ __device__ constexpr int walk_normals(int left, bool table) {
    return table ? (left < 4 ? left : 4) : left <= 2 ? 2 : 4;
}
static_assert(walk_normals(1, true) == 1 && walk_normals(2, true) == 2 && walk_normals(3, true) == 3 && walk_normals(9, true) == 4,
              "a table is read to its end, not past it");

constexpr int SYNC_TAB = 32;  // Philox blocks whose shared words a warp keeps at a time

// The paths first .. first + 31 of a contract (one a lane), from step 0 to
// the last event of the schedule. AK: the accumulator's kind, -1 for none.
template <class Real, int MODEL, int AK, bool SH>
struct SyncWalk {
    static constexpr int SPB = lean_spb<MODEL>();
    const StaticDev &T;
    const KxProgram *P;
    const StepRec<Real> *R;
    const double *D;
    const PhiloxTail keys;
    SyncDraws<Real, SH> draws;
    uint64_t seed;
    uint32_t stream;
    int last;    // step of the last event
    int af, at;  // the accumulator's window
    bool uniform;
    Real s0, uc0, uc1;
    HestonPar<Real> hp;

    // whole blocks b0 .. b1 - 1, no event inside them, all or none of their steps in the window
    template <bool UNI, int A, bool TAME>
    __device__ __forceinline__ void blocks(int b0, int b1, Real &y, Real &v, Real &av, Real &ac) const {
        const uint4 *e = draws.tab + b0 % SYNC_TAB, *const end = e + (b1 - b0);
        const StepRec<Real> *Rk = R + 1 + b0 * SPB;
        int b = b0;
#pragma unroll 2
        for (; e < end; ++e) {
            sync_block<Real, MODEL, UNI, A, TAME, SH>(draws, e, b, keys, Rk, uc0, uc1, hp, s0, y, v, av, ac);
            if (!UNI) Rk += SPB;
            if (SH) ++b;
        }
    }
    template <int A>
    __device__ __forceinline__ void blocks(int b0, int b1, Real &y, Real &v, Real &av, Real &ac) const {
        if (MODEL == M_GBM && sizeof(Real) == 4 && A >= 0 && uniform) {
            // no FP32 normal exceeds sqrt(66 ln 2) = 6.77, so no step of these blocks goes lower than this:
            // one look at the segment instead of one at every block (an Asian block 161 -> 146 cycles a warp)
            const Real low = y - Real((b1 - b0) * SPB) * (fabs(uc0) + Real(6.8) * fabs(uc1));
            if (__all_sync(0xffffffffu, low > Real(-80))) {
                blocks<true, A, true>(b0, b1, y, v, av, ac);
                return;
            }
        }
        if (uniform) blocks<true, A, false>(b0, b1, y, v, av, ac);
        else blocks<false, A, false>(b0, b1, y, v, av, ac);
    }

    // the path's value; y: its log-spot at the last event
    __device__ __forceinline__ double walk(Real v0, SLane sl, Real av, Real ac, bool &fresh, Real &y) const {
        const int lane = threadIdx.x & 31;
        Real v = v0;
        y = Real(0);
        const int n_blocks = (last + SPB - 1) / SPB;
        int b = 0;
        while (b < n_blocks) {
            // the words of the next SYNC_TAB blocks (kept from path to path when they are all there are)
            const int t1 = min(n_blocks, b - b % SYNC_TAB + SYNC_TAB);
            if (!SH && b % SYNC_TAB == 0 && !(fresh && n_blocks <= SYNC_TAB)) {
                __syncwarp();
                draws.tab[lane] = philox_block_words((uint32_t)(b + lane), stream, seed);
                __syncwarp();
                fresh = true;
            }
            // whole blocks up to the next event step (lim), the table's end and a window edge
            const int lim = sl.e < T.n_ev ? min(T.ev_step[sl.e], last) : last;
            int b1 = min(t1, lim / SPB);
            const int k = b * SPB + 1;  // first step of block b
            bool in = false;
            if (AK >= 0) {
                const int w0 = max(af, 1);
                if (k >= w0 && k <= at) {  // inside: up to the last block wholly in the window
                    in = true;
                    b1 = min(b1, at / SPB);
                } else if (k < w0) {  // before: up to the block of its first step
                    b1 = min(b1, (w0 - 1) / SPB);
                }
            }
            if (b1 > b) {
                if (AK >= 0 && in) blocks<AK>(b, b1, y, v, av, ac);
                else blocks<-1>(b, b1, y, v, av, ac);
                b = b1;
                if (b * SPB == lim) static_event<Real, (AK >= 0)>(T, D, s0, y, lim, sl, P, av, ac);
                continue;
            }
            // a block with an event or a window edge inside, step by step (a one-step path uses one pair)
            Real zz[4];
            const int left = (last - k + 1) * lean_draws<MODEL>();
            if (left <= 2) draws.block(keys, draws.tab + b % SYNC_TAB, b, walk_normals(left, SH), zz);
            else draws.block(keys, draws.tab + b % SYNC_TAB, b, SH ? walk_normals(left, true) : 4, zz);
#pragma unroll
            for (int j = 0; j < SPB; ++j) {
                if (k + j <= last) {
                    const StepRec<Real> rec = R[k + j];
                    lean_model_step<Real, MODEL>(hp, uniform ? uc0 : rec.c0, uniform ? uc1 : rec.c1, zz, j, y, v);
                    if (AK >= 0 && k + j >= af && k + j <= at) acc_add<Real, AK>(AK, av, ac, spot_of<Real>(s0, y));
                    if (sl.e < T.n_ev && T.ev_step[sl.e] == k + j)
                        static_event<Real, (AK >= 0)>(T, D, s0, y, k + j, sl, P, av, ac);
                }
            }
            ++b;
        }
        return sl.pv;
    }
};

// The value of a contract of Europeans (one event, at step k) on a path with
// log-spot y there.
template <class Real>
__device__ __forceinline__ double sync_european(const PathArgs &A, int c, Real y, int k) {
    const ContractDev &C = A.cons[c];
    const StaticDev &T = static_cast<const StaticDev *>(A.statics)[c];
    SLane sl{0u, T.all_flows, 0, 0.0};
    static_event<Real>(T, A.disc + C.disc_off, pick<Real>(C.s0[0], C.s0f[0]), y, k, sl);
    return sl.pv;
}

template <class Real, int MODEL, int MINB, bool ACC, bool SH>
__global__ void __launch_bounds__(KX_BLOCK, MINB) k_sync(const PathArgs A) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    constexpr bool HESTON = MODEL == M_HESTON;
    __shared__ uint4 tabs[KX_BLOCK / 32][SYNC_TAB];
    uint4 *tab = tabs[threadIdx.x >> 5];
    int cur = -1, last = 0, kind = ACC_SUM;
    PhiloxTail keys{};
    SLane sl{0u, 0u, 0, 0.0};  // after step 0
    Real av = 0, ac = 0, v0 = 0;
    bool fresh = false;
    unsigned long long steps = 0;
    // in a small launch (no more items than warps) a warp's one item is its own number, so it never
    // waits for an atomic (100,000 one-step paths: 12.5 -> 10.2 us)
    __shared__ int taken[KX_BLOCK / 32];
    if (lane == 0) taken[threadIdx.x >> 5] = 0;
    while (true) {
        int it = 0;
        if (lane == 0) {
            const int warps = (int)(gridDim.x * (KX_BLOCK / 32));
            int &t = taken[threadIdx.x >> 5];
            if ((int)A.n_items > warps) it = (int)atomicAdd(A.item_counter, 1u);
            else it = t == 0 ? (int)(blockIdx.x * (KX_BLOCK / 32) + (threadIdx.x >> 5)) : (int)A.n_items;
            t = 1;
        }
        it = __shfl_sync(FULL, it, 0);
        if (it >= (int)A.n_items) break;
        const WorkItem w = fetch_item(A, it);
        const ContractDev &C = A.cons[w.contract];
        const StaticDev &T = static_cast<const StaticDev *>(A.statics)[w.contract];
        const KxProgram *P = A.progs + C.prog;
        const double *D = A.disc + C.disc_off;
        const Real s0 = pick<Real>(C.s0[0], C.s0f[0]);
        const int af = ACC && T.acc_on ? T.acc_from : 1, at = ACC && T.acc_on ? T.acc_to : 0;
        if (w.contract != cur) {
            cur = w.contract;
            fresh = false;
            keys = philox_tail_keys(C.seed);
            kind = ACC ? T.acc_kind : (int)ACC_SUM;
            v0 = HESTON ? (Real)fmax(pick<Real>(C.v0, C.v0f), Real(0)) : Real(0);
            // step 0, the same for every path (S = s0): its flows and its spot in the accumulator
            sl = SLane{0u, T.all_flows, 0, 0.0};
            av = kind == ACC_MAX ? Real(-INFINITY) : kind == ACC_MIN ? Real(INFINITY) : Real(0);
            ac = Real(0);
            if (ACC && af <= 0 && 0 <= at) acc_add<Real>(kind, av, ac, spot_of<Real>(s0, Real(0)));
            static_event<Real, ACC>(T, D, s0, Real(0), 0, sl, P, av, ac);
            last = sl.rem == 0u || T.n_ev == 0 ? 0 : min(T.ev_step[T.n_ev - 1], C.n_times - 1);
        }
        HestonPar<Real> hp{};
        if (HESTON)
            hp = HestonPar<Real>{pick<Real>(C.r, C.rf), pick<Real>(C.kappa, C.kappaf), pick<Real>(C.theta, C.thetaf),
                                 pick<Real>(C.sigma_v, C.sigma_vf), pick<Real>(C.rho, C.rhof),
                                 pick<Real>(C.rho_perp, C.rho_perpf), C.heston_scheme};
        const StepRec<Real> *R = reinterpret_cast<const StepRec<Real> *>(A.steps) + C.step_off;
        const Real uc0 = pick<Real>(C.uc0, C.uc0f), uc1 = pick<Real>(C.uc1, C.uc1f);
        const uint64_t end = w.first + w.count, pv_off = C.pv_off;
        steps += (unsigned long long)w.count * (unsigned)last;
        const bool uni = C.uniform != 0;
        for (uint64_t p0 = w.first; p0 < end; p0 += 32) {
            const uint64_t path = p0 + lane;
            // (a lane past the item's end walks its last path again and stores nothing)
            const uint64_t own = path < end ? path : end - 1;
            const SyncDraws<Real, SH> draws{tab, philox_path_word((uint32_t)own, C.seed),
                                            SH ? A.zs + (own - C.path_base) : nullptr, A.zs_ld};
            double pv;
            Real y;
            if (!ACC)
                pv = SyncWalk<Real, MODEL, -1, SH>{T, P, R, D, keys, draws, C.seed, C.stream, last, af, at, uni, s0, uc0, uc1, hp}
                         .walk(v0, sl, av, ac, fresh, y);
            else if (kind == ACC_SUM)  // the kind is warp-uniform
                pv = SyncWalk<Real, MODEL, ACC_SUM, SH>{T, P, R, D, keys, draws, C.seed, C.stream, last, af, at, uni, s0, uc0, uc1, hp}
                         .walk(v0, sl, av, ac, fresh, y);
            else if (kind == ACC_MAX)
                pv = SyncWalk<Real, MODEL, ACC_MAX, SH>{T, P, R, D, keys, draws, C.seed, C.stream, last, af, at, uni, s0, uc0, uc1, hp}
                         .walk(v0, sl, av, ac, fresh, y);
            else
                pv = SyncWalk<Real, MODEL, ACC_MIN, SH>{T, P, R, D, keys, draws, C.seed, C.stream, last, af, at, uni, s0, uc0, uc1, hp}
                         .walk(v0, sl, av, ac, fresh, y);
            if (path < end) {
                A.pv[pv_off + path] = pv;
                if (!ACC)  // the Europeans that share this contract's paths
                    for (int q = 1; q <= C.more; ++q)
                        A.pv[A.cons[cur + q].pv_off + path] = sync_european<Real>(A, cur + q, y, last);
            }
        }
    }
    if (lane == 0 && steps) atomicAdd(A.steps_done, steps);
}

// Several averages on one draw (k_sync_scen): the contracts of a group.
constexpr int SYNC_SCEN = 7;
const void *sync_scen_kernel();

// The FP64 normals of paths path_base .. path_base + n - 1 of a stream, draw d
// of path i at out[d * n + i]: one thread a Philox block, the paths of a block
// side by side.
__global__ void k_normals(double *out, uint64_t n, uint32_t draws, uint64_t seed, uint32_t stream, uint32_t path_base);

// k_sync for a model and precision; acc: the contracts may keep an
// accumulator; shared: FP64 normals read from PathArgs::zs.
const void *sync_kernel(int model, bool f64, bool acc, bool shared);

}  // namespace kx
