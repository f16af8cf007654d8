// lsm_common.cuh — what the Longstaff-Schwartz kernels of lsm.cu, lsm_tiles.cu
// and lsm_tiles64.cu share: a case's arguments, its payoff and regression
// basis, and how its paths are cut into tiles.
#pragma once

#include "device_common.cuh"
#include "ffloat.cuh"
#include "engine.hpp"

namespace kx {

constexpr int LSM_BLOCK = 256;
// Block reduction scratch (doubles): red[q * 8 + w] the 8 warps' sums of up to
// 32 quantities q, the block's sums at red[LSM_RED_OUT + q].
constexpr int LSM_RED_OUT = (LSM_BLOCK / 32) * 32;
constexpr int LSM_MAXM = 6;
constexpr int LSM_COEF = 12;  // coef[d * LSM_COEF + j], j < m; [7] = have-fit flag; doubles 8..11 hold
                              // the coefficients and the flag as floats (float index j, 7)

// The payoff as up to 4 closed-form terms (kinds FA_*, FA_NONE = the constant
// sign), in both precisions, converted once on the host.
struct LsmPayTab {
    int ok, n;
    uint8_t kind[4];
    double kd[4], sd[4];
    float kf[4], sf[4];
};

struct LsmArgs {
    const KxProgram *P;  // bound payoff program (root flows only)
    const void *steps;   // StepRec<Real>[n_times]
    const double *disc;  // disc[d] = exp(-rate (t_{d+1} - t_d)), d < n_ex - 1; disc[n_ex - 1] = exp(-rate t_0)
    int n_times;         // 1 + n_ex
    int n_ex;
    uint64_t n_paths;
    uint64_t seed;
    int model;
    int scheme;
    double s0, v0, kappa, theta, sigma_v, rho, rho_perp, r;
    double x_scale;    // regressor x = S / x_scale (the model's spot): Laguerre basis, FP32 fits
    // the same parameters rounded to FP32 on the host (GB300's FP64 pipe runs
    // at ~1/64 of FP32: no thread converts a double), inv_scale_f = 1 / x_scale
    float s0_f, v0_f, kappa_f, theta_f, sigma_v_f, rho_f, rho_perp_f, r_f, inv_scale_f;
    const float *disc_f;  // (float) disc[d]
    LsmPayTab pay;
    const double *z64;
    const float *z32;
    uint64_t z_dpp;
    void *S;           // Real[n_ex][ld]
    uint64_t ld;       // row stride of S: n_paths rounded up to 64 (every row 256-byte aligned)
    void *value;       // Real[n_paths]: realised value at the current date
    double *pv;        // final per-path values
    double *partial;   // [n_tiles][LSM_NSUM]: a tile's normal equations
    double *coef;      // [n_ex][LSM_COEF]
    unsigned *sync;    // [0] iterations solved and published, [1] tiles of the current iteration done
    unsigned n_tiles;
    unsigned first_tile;         // tiles of the call before this case's
    // k_lsm_gram / k_lsm_tiles, one entry per iteration it < n_ex - 1 (regression date n_ex - 2 - it):
    unsigned long long *gram;    // [n_ex - 1][m(m+1)/2 + 1][n_tiles] a tile's sums of A and the count,
                                 // float-float or FP64
    float *factor;               // [n_ex - 1][LSM_FACTOR] the factored system
    double *phi;                 // FP64, weighted basis: [n_ex - 1][m][ld] the functions of paths in the money
    unsigned long long *cells;   // [n_ex - 1][m][n_tiles][parts] sums of A^T y, the same
    unsigned *arrived;           // [n_ex - 1][LSM_ARRIVED] blocks that published, counted from ~0u
};

// Value of the exercised contract at exercise step k (lsm.rs:238-251): the
// lowered payoff has only flows acquired at once, so each flow's discount to
// the exercise date is exp(0) = 1 and the value is the sum of the amounts.
template <class Real>
__device__ __forceinline__ Real lsm_payoff(const KxProgram &P, Real S, int k) {
    Real v = Real(0);
    AccView<Real> none{nullptr, 0};
    for (int j = 0; j < P.n_leaf; ++j) {
        const KxLeaf &F = P.leaf[j];
        uint32_t e = 0;
        v += F.kind == AK_CONST ? (Real)F.sign
             : F.fast           ? fast_amount<Real>(P, F, S)
                                : eval_code<Real>(P, F.code_off, F.code_len, none, 0u, k, S, e);
    }
    return v;
}

// The payoff as up to 4 closed-form terms in the path precision, converted
// once per thread (no double is converted per path on GB300's slow FP64
// pipe); `ok` is false when some term needs the interpreter.
template <class Real>
struct LsmPay {
    bool ok;
    int n;
    uint8_t kind[4];  // FA_NONE: the constant sign[q]
    Real k[4], sign[4];
};

// Host side: the closed-form terms of a bound payoff program.
inline LsmPayTab lsm_pay_tab(const KxProgram &P) {
    LsmPayTab t{};
    t.ok = P.n_leaf <= 4;
    t.n = 0;
    for (int j = 0; j < P.n_leaf && t.ok; ++j) {
        const KxLeaf &F = P.leaf[j];
        if (F.kind != AK_CONST && !F.fast) t.ok = false;
        t.kind[t.n] = F.kind == AK_CONST ? (uint8_t)FA_NONE : F.fast;
        t.kd[t.n] = F.kind == AK_CONST ? 0.0 : P.cpool[F.fast_k];
        t.sd[t.n] = (double)F.sign;
        t.kf[t.n] = (float)t.kd[t.n];
        t.sf[t.n] = (float)t.sd[t.n];
        ++t.n;
    }
    return t;
}

template <class Real>
__device__ __forceinline__ Real pick(double d, float f) {
    if constexpr (sizeof(Real) == 4) return f;
    else return d;
}

template <class Real>
__device__ __forceinline__ LsmPay<Real> lsm_pay_terms(const LsmPayTab &T) {
    LsmPay<Real> t;
    t.ok = T.ok;
    t.n = T.n;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        t.kind[q] = T.kind[q];
        t.k[q] = pick<Real>(T.kd[q], T.kf[q]);
        t.sign[q] = pick<Real>(T.sd[q], T.sf[q]);
    }
    return t;
}

// lsm_payoff by the closed-form terms (the same operations as fast_amount).
template <class Real>
__device__ __forceinline__ Real lsm_payoff_terms(const LsmPay<Real> &t, Real S) {
    Real v = Real(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= t.n) break;
        Real r;
        switch (t.kind[q]) {
        case FA_NONE: v += t.sign[q]; continue;
        case FA_CALL: r = fmax(S - t.k[q], Real(0)); break;
        case FA_PUT: r = fmax(t.k[q] - S, Real(0)); break;
        case FA_SPOT: r = S; break;
        default: r = t.k[q]; break;
        }
        v += t.sign[q] < Real(0) ? -r : r;
    }
    return v;
}

template <class Real>
__device__ __forceinline__ Real lsm_pay(const LsmPay<Real> &t, const KxProgram &P, Real S, int k) {
    return t.ok ? lsm_payoff_terms<Real>(t, S) : lsm_payoff<Real>(P, S, k);
}

// The same with the choice made by the caller (GEN: the interpreter), so
// that a kernel specialised for closed-form payoffs contains no call.
template <class Real, bool GEN>
__device__ __forceinline__ Real lsm_pay_g(const LsmPay<Real> &t, const KxProgram &P, Real S, int k) {
    if constexpr (GEN) return lsm_payoff<Real>(P, S, k);
    else return lsm_payoff_terms<Real>(t, S);
}

// Regression basis at spot s: monomials 1, s, ..., s^(M-1) (lsm.rs:273-278),
// or weighted Laguerre polynomials e^(-x/2) L_j(x), x = s / x_scale, with
// L_0 = 1, L_1 = 1 - x, (j + 1) L_(j+1) = (2j + 1 - x) L_j - j L_(j-1).
// Every product and sum is rounded separately (no FMA), as on the host.
template <int M, int B>
__device__ __forceinline__ void lsm_basis(double s, double x_scale, double (&phi)[M]) {
    if (B == KX_LSM_MONOMIAL) {
        phi[0] = 1.0;
#pragma unroll
        for (int j = 1; j < M; ++j) phi[j] = __dmul_rn(phi[j - 1], s);
    } else {
        const double x = __ddiv_rn(s, x_scale);
        const double w = exp(__dmul_rn(-0.5, x));
        double lm = 1.0, l = __dsub_rn(1.0, x);
        phi[0] = w;
        if (M > 1) phi[1] = __dmul_rn(w, l);
#pragma unroll
        for (int j = 1; j + 1 < M; ++j) {
            const double ln = __ddiv_rn(__dsub_rn(__dmul_rn(__dsub_rn((double)(2 * j + 1), x), l), __dmul_rn((double)j, lm)),
                                        (double)(j + 1));
            lm = l;
            l = ln;
            phi[j + 1] = __dmul_rn(w, l);
        }
    }
}

// FP32 paths: the basis of x = s / x_scale in FP32 (monomials x^j or the
// weighted Laguerre functions); the regression is invariant to the scale, so
// the fitted continuation is that of the reference's basis, while FP32 keeps
// the per-path work off the slow FP64 pipe. FP64 is used only across threads
// (block sums, cross-block sums) and for the solve.
template <int M, int B>
__device__ __forceinline__ void lsm_basis_f32(float x, float (&phi)[M]) {
    if (B == KX_LSM_MONOMIAL) {
        phi[0] = 1.0f;
#pragma unroll
        for (int j = 1; j < M; ++j) phi[j] = phi[j - 1] * x;
    } else {
        const float w = __expf(-0.5f * x);
        float lm = 1.0f, l = 1.0f - x;
        phi[0] = w;
        if (M > 1) phi[1] = w * l;
#pragma unroll
        for (int j = 1; j + 1 < M; ++j) {
            const float ln = (((float)(2 * j + 1) - x) * l - (float)j * lm) * (1.0f / (float)(j + 1));
            lm = l;
            l = ln;
            phi[j + 1] = w * l;
        }
    }
}

// Continuation value sum_j c_j phi_j(s): Horner from the top coefficient for
// monomials (poly_eval, lsm.rs:293-295), the plain sum for Laguerre.
template <int M, int B>
__device__ __forceinline__ double lsm_continuation(const double (&c)[M], double s, double x_scale) {
    double cont = 0.0;
    if (B == KX_LSM_MONOMIAL) {
#pragma unroll
        for (int j = M - 1; j >= 0; --j) cont = __dadd_rn(__dmul_rn(cont, s), c[j]);
    } else {
        double phi[M];
        lsm_basis<M, B>(s, x_scale, phi);
#pragma unroll
        for (int j = 0; j < M; ++j) cont = __dadd_rn(cont, __dmul_rn(c[j], phi[j]));
    }
    return cont;
}

// Tiles: the paths of a case are cut into tiles of LSM_TILE consecutive
// paths (FP32: in sub-chunks of 4 * LSM_BLOCK paths, thread j takes the 4
// consecutive paths 4j .. 4j + 3 of each; FP64: thread j takes paths j,
// j + LSM_BLOCK, ...); a tile's
// normal equations are reduced in a fixed order (FP32 per thread and across a
// warp's lanes, FP64 across warps) and the tiles are added in tile order. The
// order depends only on the path count, so one case alone and in a batch, on
// any grid, gives the same bits.
constexpr int LSM_PPT = 32;
constexpr unsigned LSM_TILE = LSM_BLOCK * LSM_PPT;
constexpr int LSM_NSUM = 32;                    // stride of a partial (>= m(m+1)/2 + m + 1 for m <= 6)
constexpr unsigned LSM_SPIN_LIMIT = 1u << 22;   // polls of a wait (32 ns apart at least) before giving up;
                                                // KX_LSM_SPIN_LIMIT in the environment overrides it (tests)
constexpr int LSM_MAX_CASES = 1024;             // cases of one backward launch
constexpr int LSM_MAX_COORD = 16;               // coordinator blocks of one backward launch

inline unsigned lsm_tiles(uint64_t n_paths) { return (unsigned)((n_paths + LSM_TILE - 1) / LSM_TILE); }

// Per-thread asynchronous 16-byte copies global -> shared (through L2, not
// L1: the values are written by other SMs between iterations).
__device__ __forceinline__ void lsm_cp16(void *smem_dst, const void *gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void lsm_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void lsm_cp_wait_all_but() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void lsm_cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr int LSM_SUB = 4 * LSM_BLOCK;  // paths of an FP32 sub-chunk (4 per thread)
// The kernels of a call with a resident block (or more) per tile, by basis: the
// sums of A for all dates, their factorisation, the induction (cooperative).
struct LsmTileKernels {
    const void *tiles[2];  // FP32: by LSM_SPLITS; FP64: the first
    void (*gram)(const LsmArgs *, int);
    void (*factor)(const LsmArgs *, unsigned *);
};
// The splits of k_lsm_tiles: blocks per tile and threads per column.
struct LsmSplit {
    int parts, sets;
};
constexpr LsmSplit LSM_SPLITS[2] = {{4, 4}, {1, 1}};
constexpr LsmSplit LSM_SPLIT64 = {8, 8};
constexpr int LSM_ARRIVED = 32;   // words between two dates' counts: a line each
constexpr int LSM_FACTOR = 88;    // floats of a factored system (FP64: 44 doubles)
constexpr size_t LSM_TILE_SMEM = 3 * (size_t)LSM_TILE * sizeof(float);  // two dates' spots, the values
inline size_t lsm_tile64_smem(int m) { return (size_t)m * LSM_PPT * 32 * sizeof(double); }
LsmTileKernels lsm_tile_kernels(int m, int basis);
LsmTileKernels lsm_tile_kernels64(int m, int basis);

constexpr unsigned long long LSM_EMPTY = ~0ull;
// Blocks from which each waits on the count before it reads the cells. Every
// block reading every cell until the last is there is n_tiles^2 reads a round:
// the gather of 13, 61 and 122 tiles took 3,700, 10,700 and 13,000 cycles
// (2,200 with 3 tiles).
constexpr unsigned LSM_COUNT_BLOCKS = 16;

__device__ __forceinline__ unsigned long long lsm_cell_load(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// The case of a tile of the call: the last one that starts at or before it.
__device__ __forceinline__ int lsm_case_of(const LsmArgs *cases, int n_cases, unsigned tile) {
    int c = 0;
    for (int lo = 0, hi = n_cases; lo < hi;) {
        const int mid = (lo + hi) / 2;
        if (cases[mid].first_tile <= tile) {
            c = mid;
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    return c;
}

// Waits until `want` more than ~0u has been counted; false when it gave up.
__device__ __forceinline__ bool lsm_count_wait(const unsigned *count, unsigned want, const unsigned *err,
                                               unsigned spin_limit) {
    for (unsigned polls = 0;;) {
        unsigned v;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v == want) return true;
        if (++polls > spin_limit || ((polls & 63u) == 0u && *(volatile const unsigned *)err != 0u)) return false;
    }
}

// Warps of a block that gather NQ sums (the threads per sum are those of all NS).
template <int NS, int NQ>
constexpr unsigned LSM_GATHER_WARPS = (NQ * (NS * 16 <= LSM_BLOCK ? 16 : 8) + 31) / 32;

}  // namespace kx
