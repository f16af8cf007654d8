// lsm_tiles.cu — the backward induction of FP32 American options whose tiles are
// all resident at once (see lsm.cu for the algorithm and for larger calls).
#include "lsm_common.cuh"

namespace kx {

// ---------------------------------------------------------------------------
// FP32 calls whose tiles all fit on the chip at once: a block owns a tile of
// one case, or a part of one, for the whole backward induction (k_lsm_tiles).
//
// What bounds it: the chain of one date — the last block's sums become
// visible, every block adds them and solves, and applies the decision to its
// tile — a few microseconds of latency, against 0.03 us/tile of traffic. So
//  - the tile's values, and the spots of the decision and regression dates,
//    stay in shared memory; the spots of the date after next are copied in
//    (cp.async) behind the work on this one, so no global read is waited for;
//  - every block adds all tiles' sums and solves the system itself: two hops
//    through L2 per date (a coordinator's count, its publication) less, and
//    the solve stays in each SM's instruction cache because it runs there at
//    every date;
//  - the matrix A^T A of a date depends on the spots alone, so it is summed and
//    factored for all dates at once beforehand; the chain keeps A^T y (m sums
//    of m(m+1)/2 + m + 1) and the substitutions;
//  - a sum is published as one 8-byte store into a cell of its own (one row
//    per date, cleared to LSM_EMPTY before the launch), so the cell's content
//    says that it is there: no fence, nothing reset or reused;
//  - LSM_GRP paths per thread are worked on side by side without branches.
// The order of every sum is that of k_lsm_backward (per thread over its paths,
// xor tree over the lanes, fixed trees over warps and tiles): same bits.
// 50 dates, 4 Laguerre functions, all kernels with the forward simulation
// (k_lsm_backward; all sums in the chain; A^T A ahead; arrivals counted; tiles
// split over blocks, fewer operations per path): 20,000 paths 998, 433, 332,
// 320, 206 us, 100,000 paths 1010, 503, 380, 357, 246 us, 1,000,000 paths
// 1227, 756, 713, 506, 482 us. Of a date's 13,000 cycles at 1,000,000 paths the
// paths take 6,150, the warp sums 500, the exchange 4,000 and the solve 2,300;
// at 20,000 paths 2,450, 400, 1,900 and 2,250.
constexpr int LSM_GRP = 8;  // paths a thread has in hand: two sub-chunks
static_assert(LSM_GRP % 4 == 0 && LSM_TILE % (LSM_BLOCK * LSM_GRP) == 0, "whole groups per tile");

// lsm_payoff_terms of several spots: the choice of a term's form once for all,
// a lone long call or put without the sum over terms.
template <int N>
__device__ __forceinline__ void lsm_payoff_group(const LsmPay<float> &t, const float (&S)[N], float (&v)[N]) {
    if (t.n == 1 && !(t.sign[0] < 0.0f) && (t.kind[0] == FA_PUT || t.kind[0] == FA_CALL)) {
        const float k = t.k[0];
        if (t.kind[0] == FA_PUT) {
#pragma unroll
            for (int p = 0; p < N; ++p) v[p] = fmaxf(k - S[p], 0.0f);
        } else {
#pragma unroll
            for (int p = 0; p < N; ++p) v[p] = fmaxf(S[p] - k, 0.0f);
        }
        return;
    }
#pragma unroll
    for (int p = 0; p < N; ++p) v[p] = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= t.n) break;
        const float k = t.k[q], sg = t.sign[q];
        if (t.kind[q] == FA_NONE) {
#pragma unroll
            for (int p = 0; p < N; ++p) v[p] += sg;
            continue;
        }
        float r[N];
        switch (t.kind[q]) {
        case FA_CALL:
#pragma unroll
            for (int p = 0; p < N; ++p) r[p] = fmaxf(S[p] - k, 0.0f);
            break;
        case FA_PUT:
#pragma unroll
            for (int p = 0; p < N; ++p) r[p] = fmaxf(k - S[p], 0.0f);
            break;
        case FA_SPOT:
#pragma unroll
            for (int p = 0; p < N; ++p) r[p] = S[p];
            break;
        default:
#pragma unroll
            for (int p = 0; p < N; ++p) r[p] = k;
            break;
        }
#pragma unroll
        for (int p = 0; p < N; ++p) v[p] += sg < 0.0f ? -r[p] : r[p];
    }
}

// The xor-tree sums over a warp's lanes of NS values per lane: each step hands
// half of the values to the other half of the lanes, so a step costs half of
// the one before (31 shuffles for 32 values instead of 160); every sum adds the
// same pairs as a full butterfly. Lane l ends with the sum of value
// l >> (5 - log2 NP), NP the power of two that holds NS.
template <int NP>
__device__ __forceinline__ float lsm_warp_sums(float (&a)[NP]) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = NP; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float send = up ? a[i] : a[i + n / 2], keep = up ? a[i + n / 2] : a[i];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int k = NP; k < 32; k <<= 1, o >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    return a[0];
}

__device__ __forceinline__ void lsm_cell_store(unsigned long long *p, ff x) {
    unsigned long long v = ((unsigned long long)__float_as_uint(x.lo) << 32) | __float_as_uint(x.hi);
    if (v == LSM_EMPTY) v = 0x7fffffff7fffffffull;  // a NaN pair that would read as an empty cell
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// lsm_sum_rows_ff over the cells of one date, cells[(q * n + tile) * C ...],
// each waited for until it is there: a thread re-reads only what is still
// empty, at most spin_limit times, and stops when another block reported an
// error. C = 1 or 4: a tile's sum or its four quarters in float-float
// (block_sums_ff's tree cut at that level, finished here). False when the
// calling thread gave up.
template <int NS, int NQ, int C>
__device__ __forceinline__ bool lsm_gather_ff(const unsigned long long *cells, unsigned n, ff *dst, unsigned *err,
                                              unsigned spin_limit) {
    constexpr int T = NS * 16 <= LSM_BLOCK ? 16 : 8;  // as lsm_sum_rows_ff of all NS sums
    static_assert(NQ <= NS && NS * T <= LSM_BLOCK, "threads per sum");
    constexpr int U = C == 4 ? 4 : 8;  // tiles read at once (a multiple of the 4 chains)
    const int q = threadIdx.x / T, t = threadIdx.x % T;
    ff s4[4] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
    bool ok = true;
    if (q < NQ) {
        const unsigned long long *src = cells + (size_t)q * n * C;
        for (unsigned b0 = t; b0 < n && ok; b0 += U * T) {
            unsigned long long w[U * C];
#pragma unroll
            for (int u = 0; u < U * C; ++u) w[u] = LSM_EMPTY;
            for (unsigned polls = 0;;) {
                bool all = true;
#pragma unroll
                for (int u = 0; u < U * C; ++u)
                    if (b0 + u / C * T < n && w[u] == LSM_EMPTY) w[u] = lsm_cell_load(src + (b0 + u / C * T) * C + u % C);
#pragma unroll
                for (int u = 0; u < U * C; ++u) all = all && (b0 + u / C * T >= n || w[u] != LSM_EMPTY);
                if (all) break;
                if (++polls > spin_limit || ((polls & 63u) == 0u && *(volatile unsigned *)err != 0u)) {
                    ok = false;
                    break;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (b0 + u * T >= n) continue;
                auto cell = [&](int k) {
                    return ff{__uint_as_float((unsigned)w[u * C + k]), __uint_as_float((unsigned)(w[u * C + k] >> 32))};
                };
                ff v = cell(0);
                if constexpr (C == 4) v = ff_add(ff_add(v, cell(1)), ff_add(cell(2), cell(3)));
                s4[u & 3] = ff_add(s4[u & 3], v);
            }
        }
    }
    if (q / (32 / T) * (32 / T) >= NQ) return ok;  // a warp without a sum
    __syncwarp();
    ff v = ff_add(ff_add(s4[0], s4[1]), ff_add(s4[2], s4[3]));
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
        const ff other{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = (t & o) ? ff_add(other, v) : ff_add(v, other);
    }
    if (q < NQ && t == 0) dst[q] = v;
    return ok;
}

// The float-float sums of one tile: warp sums `a` of NQ values, the 8 warps' totals added in the fixed tree of
// block_sums_ff; threads q < NQ return sum q.
template <int NQ, int NP>
__device__ __forceinline__ ff lsm_tile_sums(float (&a)[NP], float *rf) {
    static_assert(LSM_BLOCK == 256, "8 warps: a 3-level tree");
    constexpr int SH = NP == 32 ? 0 : NP == 16 ? 1 : NP == 8 ? 2 : NP == 4 ? 3 : 4;
    const unsigned j = threadIdx.x, lane = j & 31u;
    const float wsum = lsm_warp_sums<NP>(a);
    if ((lane & ((1u << SH) - 1u)) == 0u && (lane >> SH) < NQ) rf[(lane >> SH) * 8 + (j >> 5)] = wsum;
    __syncthreads();
    if (j >= NQ) return ff{0.0f, 0.0f};
    const float *r = rf + j * 8;
    return ff_add(ff_add(two_sum(r[0], r[1]), two_sum(r[2], r[3])), ff_add(two_sum(r[4], r[5]), two_sum(r[6], r[7])));
}

// The regression functions of an in-the-money path, zeros of any other.
template <int M, int B>
__device__ __forceinline__ void lsm_basis_itm(bool itm, float s, float inv_scale, float (&pw)[M]) {
    lsm_basis_f32<M, B>(itm ? s * inv_scale : 0.0f, pw);
    if (B == KX_LSM_MONOMIAL) {
        pw[0] = itm ? 1.0f : 0.0f;
    } else {
#pragma unroll
        for (int r = 0; r < M; ++r) pw[r] = itm ? pw[r] : 0.0f;
    }
}

__host__ __device__ constexpr int lsm_pow2(int n) { return n <= 2 ? 2 : n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32; }

// A tile's sums of A and its in-the-money count at every regression date:
// they depend on the spots alone, so all dates are summed at once before the
// induction instead of one after another in its chain. Block (tile, it);
// bound by the FMA pipe (about 30 operations per path and date).
template <int M, int B>
__global__ void __launch_bounds__(LSM_BLOCK) k_lsm_gram(const LsmArgs *__restrict__ cases, int n_cases) {
    constexpr int NA = M * (M + 1) / 2, NP = lsm_pow2(NA + 1);
    __shared__ float rf[(NA + 1) * 8];
    const LsmArgs &A = cases[lsm_case_of(cases, n_cases, blockIdx.x)];
    const unsigned tile = blockIdx.x - A.first_tile, j = threadIdx.x;
    const uint64_t t0 = (uint64_t)tile * LSM_TILE;
    const unsigned left = (unsigned)min((uint64_t)LSM_TILE, A.n_paths - t0);
    const float inv_scale = A.inv_scale_f;
    const LsmPay<float> terms = lsm_pay_terms<float>(A.pay);
    constexpr int GS = LSM_GRP / 4;
    for (int it = (int)blockIdx.y; it < A.n_ex - 1; it += (int)gridDim.y) {
        const float *S = reinterpret_cast<const float *>(A.S) + (uint64_t)(A.n_ex - 2 - it) * A.ld + t0;
        float acc[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] = 0.0f;
        float4 x[LSM_TILE / LSM_SUB];
#pragma unroll
        for (int sc = 0; sc < (int)(LSM_TILE / LSM_SUB); ++sc) {
            const unsigned e = sc * LSM_SUB + 4u * j;
            x[sc] = e < left ? __ldg(reinterpret_cast<const float4 *>(S + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int g = 0; g < (int)(LSM_TILE / LSM_SUB) / GS; ++g) {
            float sg[LSM_GRP], pay[LSM_GRP];
#pragma unroll
            for (int h = 0; h < GS; ++h) {
                const float4 y = x[g * GS + h];
                sg[4 * h] = y.x, sg[4 * h + 1] = y.y, sg[4 * h + 2] = y.z, sg[4 * h + 3] = y.w;
            }
            lsm_payoff_group<LSM_GRP>(terms, sg, pay);
#pragma unroll
            for (int p = 0; p < LSM_GRP; ++p) {
                const bool itm = pay[p] > 0.0f && (g * GS + p / 4) * LSM_SUB + 4u * j + (p & 3) < left;
                const float one = itm ? 1.0f : 0.0f;
                float pw[M];
                lsm_basis_itm<M, B>(itm, sg[p], inv_scale, pw);
                constexpr int R0 = B == KX_LSM_MONOMIAL ? 1 : 0;
                if (B == KX_LSM_MONOMIAL) {  // a product that is a power is that power, rounded
#pragma unroll
                    for (int s = 0; s < M; ++s) acc[s] = __fadd_rn(acc[s], pw[s]);
                }
                int q = R0 * M;
#pragma unroll
                for (int r = R0; r < M; ++r)
#pragma unroll
                    for (int s = r; s < M; ++s, ++q)
                        acc[q] = B == KX_LSM_MONOMIAL && r == 1 && s + 1 < M ? __fadd_rn(acc[q], pw[s + 1])
                                                                             : __fmaf_rn(pw[r], pw[s], acc[q]);
                acc[NA] = __fadd_rn(acc[NA], one);
            }
        }
        const ff sum = lsm_tile_sums<NA + 1>(acc, rf);
        if (j < NA + 1) lsm_cell_store(A.gram + ((size_t)it * (NA + 1) + j) * A.n_tiles + tile, sum);
        __syncthreads();
    }
}

// solve_gauss_warp_ff up to the right-hand side, for every case and date at
// once (block (case, it)): the tiles' sums of A added in tile order, the
// elimination with its row exchanges. Record: [0] enough paths for a fit, [1] a
// pivot below the bound, [2 + i] the row of A^T y that ends in row i, then the
// factors L[i][c < i] and the rows U[i][c >= i] in float-float.
static_assert(8 + 2 * LSM_MAXM * LSM_MAXM <= LSM_FACTOR, "record");
template <int M>
__global__ void __launch_bounds__(LSM_BLOCK) k_lsm_factor(const LsmArgs *__restrict__ cases, unsigned *err) {
    constexpr int NA = M * (M + 1) / 2, NS = NA + M + 1;
    __shared__ ff sums[NA + 1];
    const LsmArgs &A = cases[blockIdx.x];
    if (A.n_tiles == 0) return;
    for (int it = (int)blockIdx.y; it < A.n_ex - 1; it += (int)gridDim.y) {
        lsm_gather_ff<NS, NA + 1, 1>(A.gram + (size_t)it * (NA + 1) * A.n_tiles, A.n_tiles, sums, err, 0u);
        __syncthreads();
        if (threadIdx.x < 32) {
            const int lane = (int)threadIdx.x;
            ff a[M], f[M];
            int row = lane;
#pragma unroll
            for (int c = 0; c < M; ++c) a[c] = f[c] = ff{0.0f, 0.0f};
            if (lane < M) {
                int q = 0;
#pragma unroll
                for (int r = 0; r < M; ++r)
#pragma unroll
                    for (int c = r; c < M; ++c) {
                        if (r == lane) a[c] = sums[q];
                        if (c == lane) a[r] = sums[q];
                        ++q;
                    }
            }
            const bool fit = sums[NA].hi >= (float)M;  // lsm.rs:190-194
            bool singular = false;
#pragma unroll
            for (int col = 0; col < M; ++col) {
                int piv = col;
                ff best = ff_abs(ff_shfl(a[col], col));
#pragma unroll
                for (int r = col + 1; r < M; ++r) {
                    const ff v = ff_abs(ff_shfl(a[col], r));
                    if (ff_gt(v, best)) { best = v; piv = r; }
                }
                if (best.hi < 1e-12f) { singular = true; break; }
                ff pr[M];
#pragma unroll
                for (int c = 0; c < M; ++c) {
                    const ff from_piv = ff_shfl(a[c], piv), from_col = ff_shfl(a[c], col);
                    if (lane == col) a[c] = from_piv;
                    else if (lane == piv) a[c] = from_col;
                    pr[c] = from_piv;
                    const ff f_piv = ff_shfl(f[c], piv), f_col = ff_shfl(f[c], col);  // a row takes its factors along
                    if (lane == col) f[c] = f_piv;
                    else if (lane == piv) f[c] = f_col;
                }
                const int r_piv = __shfl_sync(0xffffffffu, row, piv), r_col = __shfl_sync(0xffffffffu, row, col);
                if (lane == col) row = r_piv;
                else if (lane == piv) row = r_col;
                if (lane > col && lane < M) {
                    const ff factor = ff_div(a[col], pr[col]);
#pragma unroll
                    for (int c = col; c < M; ++c) a[c] = ff_sub(a[c], ff_mul(factor, pr[c]));
                    f[col] = factor;
                }
            }
            float *rec = A.factor + (size_t)it * LSM_FACTOR;
            if (lane == 0) {
                rec[0] = fit ? 1.0f : 0.0f;
                rec[1] = singular ? 1.0f : 0.0f;
            }
            if (lane < M) {
                rec[2 + lane] = __int_as_float(row);
                ff *L = reinterpret_cast<ff *>(rec + 8) + lane * (lane - 1) / 2;
                ff *U = reinterpret_cast<ff *>(rec + 8) + M * (M - 1) / 2 + lane * M - lane * (lane - 1) / 2;
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

// The rest of solve_gauss_warp_ff: the right-hand side through the recorded
// factors and the back substitution, the same operations on the same values.
template <int M>
__device__ __forceinline__ void lsm_solve_factored(const float *rec, const ff *b, float *coef) {
    const bool fit = rec[0] != 0.0f, singular = rec[1] != 0.0f;
    const ff *L = reinterpret_cast<const ff *>(rec + 8), *U = L + M * (M - 1) / 2;
    ff y[M], x[M];
#pragma unroll
    for (int i = 0; i < M; ++i) y[i] = b[__float_as_int(rec[2 + i])];
#pragma unroll
    for (int c = 0; c < M; ++c)
#pragma unroll
        for (int i = c + 1; i < M; ++i) y[i] = ff_sub(y[i], ff_mul(L[i * (i - 1) / 2 + c], y[c]));
#pragma unroll
    for (int i = M - 1; i >= 0; --i) {
        const ff *u = U + i * M - i * (i - 1) / 2;
#pragma unroll
        for (int c = i + 1; c < M; ++c) y[i] = ff_sub(y[i], ff_mul(u[c - i], x[c]));
        x[i] = ff_div(y[i], u[0]);
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < M; ++r) coef[r] = fit && !singular ? x[r].hi : 0.0f;  // hi = the float nearest hi + lo
        coef[7] = fit ? 1.0f : 0.0f;
    }
}

// P blocks per tile, each with its 256 / P columns (a column: the paths one
// thread of k_lsm_backward adds up, 4 groups of LSM_GRP), SETS threads per
// column. A column's sums go through its groups in order, so the threads of a
// column do everything but those additions at once and then take turns at
// them. Grid: the tiles of all cases times P, all resident.
//
// One block per tile with one thread per column spends 7,400 cycles of a date
// on the 8,192 paths. P = 4, SETS = 4 spends 2,400 on them and is taken while
// every block has an SM of its own (38 tiles of 152 SMs: 311,296 paths; 50
// dates, 4 Laguerre functions: 20,000 paths 297 -> 212 us, 200,000 paths 355
// -> 254 us). Beyond, the exchange between more blocks takes back what the
// split gives: P = 2, SETS = 4 at 500,000 paths 402 -> 379 us with 4 functions,
// 314 -> 314 us with 3; SETS = 2 at 1,000,000 paths 480 -> 488 us.
template <int M, int B, int P, int SETS>
__global__ void __launch_bounds__(LSM_BLOCK / P *SETS, P == 1 && SETS == 1 ? 2 : 1)
    k_lsm_tiles(const LsmArgs *__restrict__ cases, int n_cases, unsigned *err, unsigned spin_limit) {
    constexpr int NA = M * (M + 1) / 2;
    constexpr int NS = NA + M + 1, NP = lsm_pow2(M);
    constexpr int GS = LSM_GRP / 4;                     // sub-chunks of a group
    constexpr int COLS = LSM_BLOCK / P, NT = COLS * SETS;
    constexpr int GP = LSM_TILE / (LSM_BLOCK * LSM_GRP) / SETS;  // groups per thread
    constexpr int SLOTS = GP * GS * NT;                 // float4 of one array of the block's paths
    extern __shared__ __align__(16) float4 lsm_smem[];  // [2][SLOTS] spots, [SLOTS] values
    __shared__ float rf[M * 8], turn[SETS > 1 ? M * COLS : 1];
    __shared__ ff sums[M];
    __shared__ __align__(8) float coef[8], rec[LSM_FACTOR];
    const unsigned gtile = blockIdx.x / P, part = blockIdx.x % P;
    const LsmArgs &A = cases[lsm_case_of(cases, n_cases, gtile)];
    const unsigned tile = gtile - A.first_tile, n_tiles = A.n_tiles;
    const int n_ex = A.n_ex;
    const unsigned j = threadIdx.x, col = part * COLS + j % COLS, set = j / COLS;
    const uint64_t t0 = (uint64_t)tile * LSM_TILE, ld = A.ld;
    const unsigned left = (unsigned)min((uint64_t)LSM_TILE, A.n_paths - t0);
    const float *S = reinterpret_cast<const float *>(A.S) + t0;
    const float inv_scale = A.inv_scale_f;
    const LsmPay<float> terms = lsm_pay_terms<float>(A.pay);
    float4 *const V = lsm_smem + 2 * SLOTS;
    // the first of the 4 paths in slot k of this thread (sub-chunk set * GP * GS + k)
    auto path0 = [&](int k) { return (set * (GP * GS) + k) * LSM_SUB + 4u * col; };
    auto fetch = [&](int row, int k) {  // the spots of slot k at exercise date `row`
        const unsigned e = path0(k);
        if (row >= 0 && e < left)  // rows are padded to 64 elements: the 16 bytes are there
            lsm_cp16(lsm_smem + ((n_ex - 1 - row) & 1) * SLOTS + k * NT + j, S + (uint64_t)row * ld + e);
    };
    for (int k = 0; k < GP * GS; ++k) {
        fetch(n_ex - 1, k);
        fetch(n_ex - 2, k);
    }
    for (int it = 0; it < n_ex; ++it) {
        const int upd = n_ex - 1 - it, gram = upd - 1;  // it = 0: the payoff at the last date
        const bool fin = gram < 0, have = it > 0 && coef[7] != 0.0f;
        const float disc_u = it > 0 ? A.disc_f[upd] : 0.0f, disc_g = fin ? 0.0f : A.disc_f[gram];
        float cu[M];
#pragma unroll
        for (int r = 0; r < M; ++r) cu[r] = coef[r];
        // the factored system of this date: read now, needed after the sums
        const float frec = !fin && j < LSM_FACTOR ? __ldg(A.factor + (size_t)it * LSM_FACTOR + j) : 0.0f;
        lsm_cp_wait_all();  // only this thread's own copies are read
        float4 *const bu = lsm_smem + (it & 1) * SLOTS, *const bg = lsm_smem + ((it + 1) & 1) * SLOTS;
        auto read = [&](const float4 *b, int g, float(&x)[LSM_GRP]) {
#pragma unroll
            for (int h = 0; h < GS; ++h) {
                const float4 y = b[(g * GS + h) * NT + j];
                x[4 * h] = y.x, x[4 * h + 1] = y.y, x[4 * h + 2] = y.z, x[4 * h + 3] = y.w;
            }
        };
        // the decision of date upd on group g: the new values, then the group's slots of `su` are free
        auto decide = [&](int g) {
            float su[LSM_GRP], pay[LSM_GRP], val[LSM_GRP];
            read(bu, g, su);
            lsm_payoff_group<LSM_GRP>(terms, su, pay);
            if (it == 0) {
#pragma unroll
                for (int p = 0; p < LSM_GRP; ++p) val[p] = pay[p];
            } else {
                float dv[LSM_GRP];
                read(V, g, dv);
#pragma unroll
                for (int p = 0; p < LSM_GRP; ++p) dv[p] *= disc_u;
                if (have) {
#pragma unroll
                    for (int p = 0; p < LSM_GRP; ++p) {
                        float phi[M];
                        lsm_basis_f32<M, B>(su[p] * inv_scale, phi);
                        float cont = 0.0f;
                        if (B == KX_LSM_MONOMIAL) {
#pragma unroll
                            for (int r = M - 1; r >= 0; --r) cont = cont * phi[1] + cu[r];
                        } else {
#pragma unroll
                            for (int r = 0; r < M; ++r) cont += cu[r] * phi[r];
                        }
                        val[p] = pay[p] > 0.0f && pay[p] > cont ? pay[p] : dv[p];
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < LSM_GRP; ++p) val[p] = pay[p] > 0.0f && pay[p] > dv[p] ? pay[p] : dv[p];
                }
            }
            if (fin) {
                double *pv = A.pv + t0;
                const double d0 = A.disc[n_ex - 1];
#pragma unroll
                for (int p = 0; p < LSM_GRP; ++p) {
                    const unsigned e = path0(g * GS + p / 4) + (p & 3);
                    if (e < left) pv[e] = (double)val[p] * d0;
                }
                return;
            }
#pragma unroll
            for (int h = 0; h < GS; ++h) {
                V[(g * GS + h) * NT + j] = make_float4(val[4 * h], val[4 * h + 1], val[4 * h + 2], val[4 * h + 3]);
                fetch(gram - 1, g * GS + h);
            }
        };
        // group g's terms of A^T y at date gram; a path that is not in the money has y = 0
        auto terms_of = [&](int g, float(&pw)[LSM_GRP][M], float(&yf)[LSM_GRP]) {
            float sg[LSM_GRP], pay[LSM_GRP], val[LSM_GRP];
            read(bg, g, sg);
            read(V, g, val);
            lsm_payoff_group<LSM_GRP>(terms, sg, pay);
#pragma unroll
            for (int p = 0; p < LSM_GRP; ++p) {
                const bool itm = pay[p] > 0.0f && (int)(p & 3) < (int)(left - path0(g * GS + p / 4));
                yf[p] = itm ? __fmul_rn(val[p], disc_g) : 0.0f;
                lsm_basis_f32<M, B>(itm ? sg[p] * inv_scale : 0.0f, pw[p]);
            }
        };
        float acc[NP];
        auto add = [&](const float(&pw)[LSM_GRP][M], const float(&yf)[LSM_GRP]) {
#pragma unroll
            for (int p = 0; p < LSM_GRP; ++p) {
                if (B == KX_LSM_MONOMIAL) acc[0] = __fadd_rn(acc[0], yf[p]);
#pragma unroll
                for (int r = B == KX_LSM_MONOMIAL ? 1 : 0; r < M; ++r) acc[r] = __fmaf_rn(pw[p][r], yf[p], acc[r]);
            }
        };
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] = 0.0f;
        if constexpr (SETS == 1) {
#pragma unroll 1
            for (int g = 0; g < GP && path0(g * GS) < left; ++g) {
                decide(g);
                if (fin) continue;
                float pw[LSM_GRP][M], yf[LSM_GRP];
                terms_of(g, pw, yf);
                add(pw, yf);
            }
            if (fin) return;  // no copy is in flight: date 0's spots were waited for above
        } else {
            static_assert(GP == 1, "a group per thread");
            float pw[LSM_GRP][M], yf[LSM_GRP];
            decide(0);
            if (fin) return;
            terms_of(0, pw, yf);
#pragma unroll 1
            for (unsigned k = 0; k < SETS; ++k) {
                if (set == k) {
                    if (k > 0) {
#pragma unroll
                        for (int r = 0; r < M; ++r) acc[r] = turn[r * COLS + j % COLS];
                    }
                    add(pw, yf);
                    if (k + 1 < SETS) {
#pragma unroll
                        for (int r = 0; r < M; ++r) turn[r * COLS + j % COLS] = acc[r];
                    }
                }
                if (k + 1 < SETS) __syncthreads();
            }
        }
        if (j < LSM_FACTOR) rec[j] = frec;
        if (set == SETS - 1) {
            constexpr int SH = NP == 8 ? 2 : NP == 4 ? 3 : 4;
            const unsigned lane = j & 31u;
            const float wsum = lsm_warp_sums<NP>(acc);
            if ((lane & ((1u << SH) - 1u)) == 0u && (lane >> SH) < M) rf[(lane >> SH) * 8 + (j % COLS) / 32] = wsum;
        }
        __syncthreads();
        unsigned long long *cells = A.cells + (size_t)it * M * n_tiles * P;
        if (j < M) {  // this block's part of block_sums_ff's tree
            const float *r = rf + j * 8;
            ff v = two_sum(r[0], r[1]);
            if constexpr (P == 1)
                v = ff_add(ff_add(v, two_sum(r[2], r[3])), ff_add(two_sum(r[4], r[5]), two_sum(r[6], r[7])));
            lsm_cell_store(cells + ((size_t)j * n_tiles + tile) * P + part, v);
        }
        bool ok = true;
        if (n_tiles * P >= LSM_COUNT_BLOCKS && j < 32 * LSM_GATHER_WARPS<NS, M>) {
            // the count is a hint without ordering: the cells say for themselves that they are there
            unsigned *count = A.arrived + (size_t)it * LSM_ARRIVED;
            if (j == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            if ((j & 31u) == 0u) ok = lsm_count_wait(count, n_tiles * P - 1u, err, spin_limit);
            __syncwarp();
        }
        ok = lsm_gather_ff<NS, M, P>(cells, n_tiles, sums, err, spin_limit) && ok;
        if (__syncthreads_or(!ok)) {
            if (j == 0) atomicOr(err, 1u);
            lsm_cp_wait_all();
            return;
        }
        if (j < 32) lsm_solve_factored<M>(rec, sums, coef);
        __syncthreads();
    }
}

#define LSM_TILE_VARIANTS(M, B) {(const void *)k_lsm_tiles<M, B, 4, 4>, (const void *)k_lsm_tiles<M, B, 1, 1>}
template <int M>
static LsmTileKernels tile_kernels_m(int basis) {
    if (basis == KX_LSM_LAGUERRE)
        return {LSM_TILE_VARIANTS(M, KX_LSM_LAGUERRE), k_lsm_gram<M, KX_LSM_LAGUERRE>, k_lsm_factor<M>};
    return {LSM_TILE_VARIANTS(M, KX_LSM_MONOMIAL), k_lsm_gram<M, KX_LSM_MONOMIAL>, k_lsm_factor<M>};
}
LsmTileKernels lsm_tile_kernels(int m, int basis) {
    switch (m) {
    case 2: return tile_kernels_m<2>(basis);
    case 3: return tile_kernels_m<3>(basis);
    case 4: return tile_kernels_m<4>(basis);
    case 5: return tile_kernels_m<5>(basis);
    default: return tile_kernels_m<6>(basis);
    }
}

}  // namespace kx
