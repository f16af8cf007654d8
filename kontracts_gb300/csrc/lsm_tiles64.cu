// lsm_tiles64.cu — the backward induction of FP64 American options whose tiles
// are all resident at once, eight blocks per tile (see lsm.cu for the algorithm
// and for larger calls, lsm_tiles.cu for the FP32 form of the same scheme).
//
// What bounds it: the FP64 pipe (64 cycles per warp instruction on each SM
// quarter). One block per tile kept 8,192 paths on one SM: 94 of a date's 114 us
// on 13 SMs at 100,000 paths. Here a block has one of a tile's eight column
// warps' paths (a column: the paths one thread of k_lsm_backward adds up), its
// eight warps take four paths of every column each, and
//  - A^T A is summed and factored for all dates beforehand, on all SMs;
//  - the regression functions evaluated for A^T A serve the date's A^T y and the
//    next decision: the weighted ones are kept in memory (an exponential and a
//    division are some 50 FP64 operations), powers are formed from the spot;
//  - the products with y go through shared memory and warp q adds those of sum
//    q in the order of the paths, so the M chains of 32 additions run on
//    different SM quarters;
//  - every block adds all warps' totals and solves, as in lsm_tiles.cu.
// Every sum keeps the order of k_lsm_backward: same bits. 50 dates, kernels with
// the forward simulation, k_lsm_backward and this: 3 monomials 20,000 paths 5710
// -> 836 us, 200,000 paths 6809 -> 2678 us; 4 weighted Laguerre functions 17,194
// -> 1053 us and 18,379 -> 3817 us. Taken while a tile's eight blocks are
// resident, two to an SM (38 tiles, 311,296 paths; at 300,000 paths 7258 -> 3381
// us and 18,809 -> 4965 us).
#include "lsm_common.cuh"

namespace kx {

constexpr int LSM64_PPT = LSM_PPT / LSM_SPLIT64.sets;  // paths per thread
static_assert(LSM_SPLIT64.parts * 32 == LSM_BLOCK && LSM_SPLIT64.sets * 32 == LSM_BLOCK, "a column warp per block");

__device__ __forceinline__ unsigned long long lsm_cell_of(double x) {
    const unsigned long long v = (unsigned long long)__double_as_longlong(x);
    return v == LSM_EMPTY ? 0x7fffffffffffffffull : v;  // a NaN that would read as an empty cell
}

// Sums of A and the in-the-money count of a tile at every regression date:
// block (tile, it), the loop of lsm_tile_paths without the values.
template <int M, int B>
__global__ void __launch_bounds__(LSM_BLOCK) k_lsm_gram64(const LsmArgs *__restrict__ cases, int n_cases) {
    constexpr int NA = M * (M + 1) / 2;
    __shared__ double red[(NA + 1) * 8];
    const LsmArgs &A = cases[lsm_case_of(cases, n_cases, blockIdx.x)];
    const unsigned tile = blockIdx.x - A.first_tile, j = threadIdx.x;
    const uint64_t i0 = (uint64_t)tile * LSM_TILE + j;
    const LsmPay<double> terms = lsm_pay_terms<double>(A.pay);
    for (int it = (int)blockIdx.y; it < A.n_ex - 1; it += (int)gridDim.y) {
        const int gram = A.n_ex - 2 - it;
        const double *S = reinterpret_cast<const double *>(A.S) + (uint64_t)gram * A.ld;
        double *phi = B == KX_LSM_LAGUERRE ? A.phi + (uint64_t)gram * M * A.ld : nullptr;
        double acc[NA + 1];
#pragma unroll
        for (int q = 0; q <= NA; ++q) acc[q] = 0.0;
#pragma unroll 1
        for (int k0 = 0; k0 < LSM_PPT; k0 += 4) {
            double s[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t i = i0 + (uint64_t)(k0 + k) * LSM_BLOCK;
                s[k] = i < A.n_paths ? __ldg(S + i) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t i = i0 + (uint64_t)(k0 + k) * LSM_BLOCK;
                if (i >= A.n_paths) break;
                if (lsm_payoff_terms<double>(terms, s[k]) > 0.0) {
                    double pw[M];
                    lsm_basis<M, B>(s[k], A.x_scale, pw);
                    if (B == KX_LSM_LAGUERRE) {
#pragma unroll
                        for (int r = 0; r < M; ++r) phi[(uint64_t)r * A.ld + i] = pw[r];
                    }
                    int q = 0;
#pragma unroll
                    for (int r = 0; r < M; ++r)
#pragma unroll
                        for (int c = r; c < M; ++c) acc[q++] += __dmul_rn(pw[r], pw[c]);
                    acc[NA] += 1.0;
                }
            }
        }
        // block_sums: the lanes of a warp, then the 8 warps in order
#pragma unroll
        for (int q = 0; q <= NA; ++q) {
            double v = acc[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((j & 31u) == 0u) red[q * 8 + (j >> 5)] = v;
        }
        __syncthreads();
        if (j <= NA) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[j * 8 + w];
            reinterpret_cast<double *>(A.gram)[((size_t)it * (NA + 1) + j) * A.n_tiles + tile] = t;
        }
        __syncthreads();
    }
}

// The sum over tiles of one quantity by the T threads t (lsm_sum_rows): `row`
// gives a tile's sum; every lane of the group returns the total.
template <int T, class F>
__device__ __forceinline__ double lsm_tiles_sum(unsigned n, int t, const F &row) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    for (unsigned b = t, u = 0; b < n; b += T, u = (u + 1) & 3u) {
        const double x = row(b);
#pragma unroll
        for (unsigned v = 0; v < 4; ++v)
            if (v == u) s4[v] += x;
    }
    double v = (s4[0] + s4[1]) + (s4[2] + s4[3]);
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// solve_gauss_warp up to the right-hand side, for every case and date at once
// (the record of k_lsm_factor, in doubles).
template <int M>
__global__ void __launch_bounds__(LSM_BLOCK) k_lsm_factor64(const LsmArgs *__restrict__ cases, unsigned *) {
    constexpr int NA = M * (M + 1) / 2, NS = NA + M + 1, T = NS * 16 <= LSM_BLOCK ? 16 : 8;
    static_assert(2 * (8 + M * M) <= LSM_FACTOR, "record");
    __shared__ double sums[LSM_BLOCK / T];
    const LsmArgs &A = cases[blockIdx.x];
    if (A.n_tiles == 0) return;
    for (int it = (int)blockIdx.y; it < A.n_ex - 1; it += (int)gridDim.y) {
        const int q = threadIdx.x / T, t = threadIdx.x % T;
        const double *rows = reinterpret_cast<const double *>(A.gram) + ((size_t)it * (NA + 1) + q) * A.n_tiles;
        const double v = lsm_tiles_sum<T>(q <= NA ? A.n_tiles : 0u, t, [&](unsigned b) { return rows[b]; });
        if (t == 0) sums[q] = v;
        __syncthreads();
        if (threadIdx.x < 32) {
            const unsigned FULL = 0xffffffffu;
            const int lane = (int)threadIdx.x;
            double a[M], f[M];
            int row = lane;
#pragma unroll
            for (int c = 0; c < M; ++c) a[c] = f[c] = 0.0;
            if (lane < M) {
                int k = 0;
#pragma unroll
                for (int r = 0; r < M; ++r)
#pragma unroll
                    for (int c = r; c < M; ++c) {
                        if (r == lane) a[c] = sums[k];
                        if (c == lane) a[r] = sums[k];
                        ++k;
                    }
            }
            const bool fit = sums[NA] >= (double)M;  // lsm.rs:190-194
            bool singular = false;
#pragma unroll
            for (int col = 0; col < M; ++col) {
                int piv = col;
                double best = fabs(__shfl_sync(FULL, a[col], col));
#pragma unroll
                for (int r = col + 1; r < M; ++r) {
                    const double x = fabs(__shfl_sync(FULL, a[col], r));
                    if (x > best) { best = x; piv = r; }
                }
                if (best < 1e-12) { singular = true; break; }
                double pr[M];
#pragma unroll
                for (int c = 0; c < M; ++c) {
                    const double from_piv = __shfl_sync(FULL, a[c], piv), from_col = __shfl_sync(FULL, a[c], col);
                    if (lane == col) a[c] = from_piv;
                    else if (lane == piv) a[c] = from_col;
                    pr[c] = from_piv;
                    const double f_piv = __shfl_sync(FULL, f[c], piv), f_col = __shfl_sync(FULL, f[c], col);
                    if (lane == col) f[c] = f_piv;  // a row takes its factors along
                    else if (lane == piv) f[c] = f_col;
                }
                const int r_piv = __shfl_sync(FULL, row, piv), r_col = __shfl_sync(FULL, row, col);
                if (lane == col) row = r_piv;
                else if (lane == piv) row = r_col;
                if (lane > col && lane < M) {
                    const double factor = __ddiv_rn(a[col], pr[col]);
#pragma unroll
                    for (int c = col; c < M; ++c) a[c] = __dsub_rn(a[c], __dmul_rn(factor, pr[c]));
                    f[col] = factor;
                }
            }
            double *rec = reinterpret_cast<double *>(A.factor + (size_t)it * LSM_FACTOR);
            if (lane == 0) {
                rec[0] = fit ? 1.0 : 0.0;
                rec[1] = singular ? 1.0 : 0.0;
            }
            if (lane < M) {
                rec[2 + lane] = (double)row;
                double *L = rec + 8 + lane * (lane - 1) / 2;
                double *U = rec + 8 + M * (M - 1) / 2 + lane * M - lane * (lane - 1) / 2;
#pragma unroll
                for (int c = 0; c < M; ++c) {
                    if (c < lane) L[c] = f[c];
                    else U[c - lane] = a[c];
                }
            }
        }
        __syncthreads();
    }
}

// Grid: the tiles of all cases times 8, all resident. prod: the products of a
// date, [M][LSM_PPT][32].
template <int M, int B>
__global__ void __launch_bounds__(LSM_BLOCK, 2)
    k_lsm_tiles64(const LsmArgs *__restrict__ cases, int n_cases, unsigned *err, unsigned spin_limit) {
    constexpr int NA = M * (M + 1) / 2, NS = NA + M + 1, T = NS * 16 <= LSM_BLOCK ? 16 : 8;
    constexpr int PARTS = LSM_SPLIT64.parts, PPT = LSM64_PPT;
    constexpr unsigned GATHER = (M * T + 31) / 32 * 32;  // threads of the warps that gather
    extern __shared__ __align__(16) double lsm_prod[];
    __shared__ double sums[LSM_BLOCK / T], coef[8], rec[LSM_FACTOR / 2];
    const unsigned gtile = blockIdx.x / PARTS, part = blockIdx.x % PARTS;
    const LsmArgs &A = cases[lsm_case_of(cases, n_cases, gtile)];
    const unsigned tile = gtile - A.first_tile, n_tiles = A.n_tiles;
    const int n_ex = A.n_ex;
    const unsigned j = threadIdx.x, lane = j & 31u, set = j >> 5;
    const uint64_t np = A.n_paths, ld = A.ld;
    const uint64_t i0 = (uint64_t)tile * LSM_TILE + part * 32u + lane + (uint64_t)(set * PPT) * LSM_BLOCK;
    const double *S = reinterpret_cast<const double *>(A.S);
    const LsmPay<double> terms = lsm_pay_terms<double>(A.pay);
    auto path = [&](int p) { return i0 + (uint64_t)p * LSM_BLOCK; };
    // spots, payoffs and regression functions of the decision date (u) and the regression date (g)
    double su[PPT], pu[PPT], fu[PPT][M], sg[PPT], pg[PPT], fg[PPT][M], val[PPT];
    auto load = [&](int row) {
#pragma unroll
        for (int p = 0; p < PPT; ++p) sg[p] = row >= 0 && path(p) < np ? __ldg(S + (uint64_t)row * ld + path(p)) : 0.0;
        if (B == KX_LSM_LAGUERRE) {
#pragma unroll
            for (int r = 0; r < M; ++r)
#pragma unroll
                for (int p = 0; p < PPT; ++p)  // written where the payoff is positive, used there alone
                    fg[p][r] = row >= 0 && path(p) < np ? __ldg(A.phi + ((uint64_t)row * M + r) * ld + path(p)) : 0.0;
        }
    };
    auto prepare = [&] {
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            pg[p] = lsm_payoff_terms<double>(terms, sg[p]);
            if (B == KX_LSM_MONOMIAL) lsm_basis<M, B>(sg[p], 1.0, fg[p]);
        }
    };
    auto shift = [&] {  // the regression date becomes the decision date
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            su[p] = sg[p];
            pu[p] = pg[p];
            if (B == KX_LSM_LAGUERRE) {
#pragma unroll
                for (int r = 0; r < M; ++r) fu[p][r] = fg[p][r];
            }
        }
    };
#pragma unroll
    for (int p = 0; p < PPT; ++p) sg[p] = path(p) < np ? __ldg(S + (uint64_t)(n_ex - 1) * ld + path(p)) : 0.0;
#pragma unroll
    for (int p = 0; p < PPT; ++p)
#pragma unroll
        for (int r = 0; r < M; ++r) fg[p][r] = 0.0;
    prepare();
    shift();
    load(n_ex - 2);
    prepare();
    for (int it = 0; it < n_ex; ++it) {
        const int upd = n_ex - 1 - it, gram = upd - 1;  // it = 0: the payoff at the last date
        const bool fin = gram < 0, have = it > 0 && coef[7] != 0.0;
        const double disc_u = it > 0 ? A.disc[upd] : 0.0, disc_g = fin ? 0.0 : A.disc[gram];
        const double frec = !fin && j < LSM_FACTOR / 2
                                ? __ldg(reinterpret_cast<const double *>(A.factor + (size_t)it * LSM_FACTOR) + j)
                                : 0.0;
        double cu[M];
#pragma unroll
        for (int r = 0; r < M; ++r) cu[r] = coef[r];
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            if (it == 0) {
                val[p] = pu[p];
                continue;
            }
            const double discounted = val[p] * disc_u;
            double cont = discounted;
            if (have) {
                if (B == KX_LSM_MONOMIAL) {
                    cont = lsm_continuation<M, B>(cu, su[p], 1.0);
                } else {
                    cont = 0.0;
#pragma unroll
                    for (int r = 0; r < M; ++r) cont = __dadd_rn(cont, __dmul_rn(cu[r], fu[p][r]));
                }
            }
            val[p] = pu[p] > 0.0 && pu[p] > cont ? pu[p] : discounted;
        }
        if (fin) {
            const double d0 = A.disc[n_ex - 1];
#pragma unroll
            for (int p = 0; p < PPT; ++p)
                if (path(p) < np) A.pv[path(p)] = val[p] * d0;
            return;
        }
#pragma unroll
        for (int p = 0; p < PPT; ++p) {  // a path that is not in the money adds zeros
            const bool itm = pg[p] > 0.0 && path(p) < np;
            const double y = val[p] * disc_g;
#pragma unroll
            for (int r = 0; r < M; ++r)
                lsm_prod[(r * LSM_PPT + set * PPT + p) * 32 + lane] = itm ? __dmul_rn(fg[p][r], y) : 0.0;
        }
        if (j < LSM_FACTOR / 2) rec[j] = frec;
        __syncthreads();
        unsigned long long *cells = A.cells + (size_t)it * M * n_tiles * PARTS;
        if (set < M) {
            double v = 0.0;
#pragma unroll 8
            for (int k = 0; k < LSM_PPT; ++k) v += lsm_prod[(set * LSM_PPT + k) * 32 + lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) {
                unsigned long long *cell = cells + ((size_t)set * n_tiles + tile) * PARTS + part;
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(cell), "l"(lsm_cell_of(v)) : "memory");
            }
        }
        shift();
        load(gram - 1);  // in flight behind the exchange
        bool ok = true;
        if (j < GATHER) {
            if (n_tiles * PARTS >= LSM_COUNT_BLOCKS) {
                // the count is a hint without ordering: the cells say for themselves that they are there
                unsigned *count = A.arrived + (size_t)it * LSM_ARRIVED;
                if (j == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
                if (lane == 0) ok = lsm_count_wait(count, n_tiles * PARTS - 1u, err, spin_limit);
                __syncwarp();
            }
            const int q = (int)j / T, t = (int)j % T;
            const double v = lsm_tiles_sum<T>(q < M ? n_tiles : 0u, t, [&](unsigned b) {
                const unsigned long long *src = cells + ((size_t)q * n_tiles + b) * PARTS;
                unsigned long long w[PARTS];
#pragma unroll
                for (int u = 0; u < PARTS; ++u) w[u] = LSM_EMPTY;
                for (unsigned polls = 0; ok;) {
                    bool all = true;
#pragma unroll
                    for (int u = 0; u < PARTS; ++u)
                        if (w[u] == LSM_EMPTY) w[u] = lsm_cell_load(src + u);
#pragma unroll
                    for (int u = 0; u < PARTS; ++u) all = all && w[u] != LSM_EMPTY;
                    if (all) break;
                    if (++polls > spin_limit || ((polls & 63u) == 0u && *(volatile unsigned *)err != 0u)) ok = false;
                }
                double x = __longlong_as_double((long long)w[0]);
#pragma unroll
                for (int u = 1; u < PARTS; ++u) x += __longlong_as_double((long long)w[u]);  // the 8 warps in order
                return x;
            });
            if (t == 0) sums[q] = v;
        }
        prepare();
        if (__syncthreads_or(!ok)) {
            if (j == 0) atomicOr(err, 1u);
            return;
        }
        if (j < 32) {  // the rest of solve_gauss_warp
            const bool fit = rec[0] != 0.0, singular = rec[1] != 0.0;
            const double *L = rec + 8, *U = L + M * (M - 1) / 2;
            double y[M], x[M];
#pragma unroll
            for (int i = 0; i < M; ++i) y[i] = sums[(int)rec[2 + i] & 7];
#pragma unroll
            for (int c = 0; c < M; ++c)
#pragma unroll
                for (int i = c + 1; i < M; ++i) y[i] = __dsub_rn(y[i], __dmul_rn(L[i * (i - 1) / 2 + c], y[c]));
#pragma unroll
            for (int i = M - 1; i >= 0; --i) {
                const double *u = U + i * M - i * (i - 1) / 2;
#pragma unroll
                for (int c = i + 1; c < M; ++c) y[i] = __dsub_rn(y[i], __dmul_rn(u[c - i], x[c]));
                x[i] = __ddiv_rn(y[i], u[0]);
            }
            if (j == 0) {
#pragma unroll
                for (int r = 0; r < M; ++r) coef[r] = fit && !singular ? x[r] : 0.0;
                coef[7] = fit ? 1.0 : 0.0;
            }
        }
        __syncthreads();
    }
}

template <int M>
static LsmTileKernels tile_kernels_m(int basis) {
    if (basis == KX_LSM_LAGUERRE)
        return {{(const void *)k_lsm_tiles64<M, KX_LSM_LAGUERRE>, nullptr}, k_lsm_gram64<M, KX_LSM_LAGUERRE>, k_lsm_factor64<M>};
    return {{(const void *)k_lsm_tiles64<M, KX_LSM_MONOMIAL>, nullptr}, k_lsm_gram64<M, KX_LSM_MONOMIAL>, k_lsm_factor64<M>};
}
LsmTileKernels lsm_tile_kernels64(int m, int basis) {
    switch (m) {
    case 2: return tile_kernels_m<2>(basis);
    case 3: return tile_kernels_m<3>(basis);
    case 4: return tile_kernels_m<4>(basis);
    case 5: return tile_kernels_m<5>(basis);
    default: return tile_kernels_m<6>(basis);
    }
}

}  // namespace kx
