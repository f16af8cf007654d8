// paths_sync.cu — instantiations of k_sync (static schedules without barriers),
// the table of normals that FP64 launches of one stream share, and the walk of
// several averages on one draw.
#include "paths_sync.cuh"

namespace kx {

__global__ void __launch_bounds__(256) k_normals(double *out, uint64_t n, uint32_t draws, uint64_t seed,
                                                 uint32_t stream, uint32_t path_base) {
    const uint32_t blocks = (draws + 3) / 4;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n * blocks;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = (uint32_t)(t / n);
        const uint64_t i = t - (uint64_t)b * n;
        const uint4 w = philox4x32_10(make_uint4(b, path_base + (uint32_t)i, 0u, stream), (uint32_t)seed,
                                      (uint32_t)(seed >> 32));
        double z[4];
        box_muller(w.x, w.y, z[0], z[1]);
        box_muller(w.z, w.w, z[2], z[3]);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (4 * b + j < draws) out[(uint64_t)(4 * b + j) * n + i] = z[j];
    }
}

template <class Real, int MODEL, int MINB, bool SH>
static const void *sync_pick(bool acc) {
    return acc ? (const void *)&k_sync<Real, MODEL, MINB, true, SH> : (const void *)&k_sync<Real, MODEL, MINB, false, SH>;
}

const void *sync_kernel(int model, bool f64, bool acc, bool shared) {
    if (model == KX_MODEL_GBM) {
        if (!f64) return sync_pick<float, M_GBM, 4, false>(acc);
        return shared ? sync_pick<double, M_GBM, 2, true>(acc) : sync_pick<double, M_GBM, 2, false>(acc);
    }
    if (!f64) return sync_pick<float, M_HESTON, 4, false>(acc);
    return shared ? sync_pick<double, M_HESTON, 2, true>(acc) : sync_pick<double, M_HESTON, 2, false>(acc);
}

// Several averages on one draw (FP32, GBM): the reprices of a central
// difference walk the same normals under other spots, volatilities and rates.
// A lane draws its path's block once and walks up to W contracts with it, the
// leader and the C.more after it; each has its own log-spot and Kahan sum, so
// every value is k_sync's bit for bit. What bounds it: per block 74 cycles of
// the FMA pipe for the draw and 32 per contract (k_sync: 106 each). The seven
// reprices of an Asian call's Greeks, 252 steps: 200,000 paths 345 -> 172 us,
// 1,000,000 paths 1654 -> 694 us (3 blocks an SM 724, 2: 763; groups of 4: 946).
static __global__ void __launch_bounds__(KX_BLOCK, 4) k_sync_scen(const PathArgs A) {
    constexpr int W = SYNC_SCEN;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    __shared__ uint4 tabs[KX_BLOCK / 32][SYNC_TAB];
    uint4 *tab = tabs[threadIdx.x >> 5];
    unsigned long long steps = 0;
    while (true) {
        int it = 0;
        if (lane == 0) it = (int)atomicAdd(A.item_counter, 1u);
        it = __shfl_sync(FULL, it, 0);
        if (it >= (int)A.n_items) break;
        const WorkItem w = fetch_item(A, it);
        const ContractDev &C = A.cons[w.contract];
        const StaticDev &T = static_cast<const StaticDev *>(A.statics)[w.contract];
        const int more = C.more, last = T.ev_step[0], af = T.acc_from, at = T.acc_to;
        const int n_blocks = (last + 3) / 4;
        const PhiloxTail keys = philox_tail_keys(C.seed);
        float s0[W], c0[W], c1[W], reach = 0.0f;
#pragma unroll
        for (int q = 0; q < W; ++q) {  // (a walk past the group repeats its last and stores nothing)
            const ContractDev &Q = A.cons[w.contract + min(q, more)];
            s0[q] = Q.s0f[0];
            c0[q] = Q.uc0f;
            c1[q] = Q.uc1f;
            reach = fmaxf(reach, fabsf(c0[q]) + 6.8f * fabsf(c1[q]));
        }
        const uint64_t end = w.first + w.count;
        steps += (unsigned long long)w.count * (unsigned)last * (unsigned)(1 + more);
        bool fresh = false;
        for (uint64_t p0 = w.first; p0 < end; p0 += 32) {
            const uint64_t path = p0 + lane, own = path < end ? path : end - 1;
            const SyncDraws<float, false> draws{tab, philox_path_word((uint32_t)own, C.seed), nullptr, 0};
            float y[W], av[W], ac[W];
#pragma unroll
            for (int q = 0; q < W; ++q) {
                y[q] = av[q] = ac[q] = 0.0f;
                if (af <= 0) acc_add<float, ACC_SUM>(ACC_SUM, av[q], ac[q], spot_of<float>(s0[q], 0.0f));
            }
            for (int b = 0; b < n_blocks;) {
                const int t1 = min(n_blocks, b - b % SYNC_TAB + SYNC_TAB);
                if (b % SYNC_TAB == 0 && !(fresh && n_blocks <= SYNC_TAB)) {
                    __syncwarp();
                    tab[lane] = philox_block_words((uint32_t)(b + lane), C.stream, C.seed);
                    __syncwarp();
                    fresh = true;
                }
                const int k = 4 * b + 1;  // first step of block b
                int b1 = min(t1, min(last, at) / 4);  // whole blocks inside the window and before the event
                float low = y[0];
#pragma unroll
                for (int q = 1; q < W; ++q) low = fminf(low, y[q]);
                // as SyncWalk::blocks: no step goes lower than this, so no exponential is subnormal
                if (k >= max(af, 1) && b1 > b && __all_sync(FULL, low - (float)(4 * (b1 - b)) * reach > -80.0f)) {
                    for (; b < b1; ++b) {
                        float zz[4];
                        draws.block(keys, tab + b % SYNC_TAB, b, 4, zz);
#pragma unroll
                        for (int q = 0; q < W; ++q) {
                            float ys[4], v = 0.0f;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                lean_model_step<float, M_GBM>(HestonPar<float>{}, c0[q], c1[q], zz, j, y[q], v);
                                ys[j] = y[q];
                            }
                            block_acc<float, ACC_SUM, true>(ys, 4, s0[q], av[q], ac[q]);
                        }
                    }
                    continue;
                }
                float zz[4];
                draws.block(keys, tab + b % SYNC_TAB, b, 4, zz);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k + j <= last) {
#pragma unroll
                        for (int q = 0; q < W; ++q) {
                            float v = 0.0f;
                            lean_model_step<float, M_GBM>(HestonPar<float>{}, c0[q], c1[q], zz, j, y[q], v);
                            if (k + j >= af && k + j <= at)
                                acc_add<float, ACC_SUM>(ACC_SUM, av[q], ac[q], spot_of<float>(s0[q], y[q]));
                        }
                    }
                ++b;
            }
            float fin[3][W];
#pragma unroll
            for (int q = 0; q < W; ++q) {
                fin[0][q] = y[q];
                fin[1][q] = av[q];
                fin[2][q] = ac[q];
            }
            if (path < end) {
#pragma unroll 1
                for (int q = 0; q <= more; ++q) {
                    const ContractDev &Q = A.cons[w.contract + q];
                    const StaticDev &TQ = static_cast<const StaticDev *>(A.statics)[w.contract + q];
                    SLane sl{0u, TQ.all_flows, 0, 0.0};
                    static_event<float, true>(TQ, A.disc + Q.disc_off, Q.s0f[0], fin[0][q], last, sl, A.progs + Q.prog,
                                              fin[1][q], fin[2][q]);
                    A.pv[Q.pv_off + path] = sl.pv;
                }
            }
        }
    }
    if (lane == 0 && steps) atomicAdd(A.steps_done, steps);
}

const void *sync_scen_kernel() { return (const void *)&k_sync_scen; }

}  // namespace kx
