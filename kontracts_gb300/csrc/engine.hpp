// engine.hpp — host-side device context shared by the CUDA translation units.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "capi_util.hpp"
#include "frontend.hpp"

namespace kx {

void cuda_check(cudaError_t e, const char *what);
#define KX_CUDA(call) ::kx::cuda_check((call), #call)

// Device memory; when there is none left, the context's memory that calls can
// do without (Ctx::normals, Ctx::lsm_extra) is given back and the request made
// once more.
void *device_alloc(size_t bytes);

// Growable device buffer owned by the context.
struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
    void ensure(size_t bytes);
    // for memory the caller can do without: false when the device has no room for it, or it is more
    // than KX_EXTRA_SCRATCH bytes (an environment variable; unset: no limit). The buffer is then empty.
    bool try_ensure(size_t bytes);
    void release();
    template <class T>
    T *as() const { return static_cast<T *>(p); }
};

// Growable page-locked host buffer: copies from and to it are true
// asynchronous DMA (a pageable source costs a staging copy per call).
struct PinnedBuf {
    void *p = nullptr;
    size_t cap = 0;
    void ensure(size_t bytes);
    template <class T>
    T *as() const { return static_cast<T *>(p); }
};

struct DrawStore {  // host normals for KX_RNG_SHARED_DRAWS
    DevBuf z64, z32;
    bool is64 = false;
    uint64_t n_paths = 0, dpp = 0;
    bool set = false;
};

struct Ctx {
    std::atomic<bool> ready{false};  // set once, after every field below is valid
    int device = 0;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    std::string name;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t ev2 = nullptr, ev3 = nullptr;  // around the statistics, which queue behind a path launch
    // scratch owned by the context
    DevBuf progs, steps, disc, thr, cons, items, counters, pv, chunks, chunk_out, misc, vr, lsm_paths, lsm_value,
        grid_tabs, statics, mlmc, plan, stats_in;
    // and what a call can do without: the normals several FP64 walks share (at most 1 GiB), and what the
    // resident American kernels keep beside the stored spots (the weighted basis, at most 1 GiB, and sums)
    DevBuf normals, lsm_extra;
    // host staging of a call's uploads and downloads (path plan, statistics)
    PinnedBuf plan_stage, stats_stage, count_stage;
    DrawStore draws;
    kx_launch_stats last{};
    const char *last_kernel = "";  // the kernel of the last call's (last) launch over paths
    // a path launch (ev0 .. ev1) that nothing has waited for yet: the call waits once, for its
    // statistics, and its counters (item counter, error word, steps as u64; 16 bytes on the
    // device) come back with them
    bool paths_pending = false, pending_has_err = false;
    const uint32_t *pending_dev = nullptr;
    bool kahan_stats = false;  // this call's plain statistics in compensated FP32 (KX_PREC_FP32_KAHAN)
    std::mutex mu;
};

// Waits for a pending path launch and reads its time, steps and error word
// (settle_paths: the stream has been waited for, `counters` are the launch's on
// the host). Raises the launch's error.
void finish_paths(Ctx &c);
void settle_paths(Ctx &c, const uint32_t *counters);

// Per-call bookkeeping of the launch statistics.
void begin_call(Ctx &c);
void end_call(Ctx &c);

// Lazily initialised process context; throws KX_NO_DEVICE without a GPU.
// Thread-safe: the first callers race only for a set-up mutex, one of them
// creates the stream and events, the others wait and then see the result.
Ctx &ctx();

// Persistent grid size for a kernel with `block` threads and `smem` bytes.
int persistent_blocks(const void *kernel, int block, size_t smem);

double now_ms();

// Deterministic statistics of per-path values: returns (n, mean, M2)
// merged over fixed chunks of [begin, begin + n) of `values` (device), with
// values[i] = sum_s w[s] * base[s * stride + i] when ns > 1.
struct Stats {
    double n = 0, mean = 0, m2 = 0;
};
struct StatsJob {
    uint64_t begin = 0, n = 0;
    int ns = 1;
    double w[8] = {1, 0, 0, 0, 0, 0, 0, 0};
};
std::vector<Stats> device_stats(Ctx &c, const double *values, uint64_t stride, const std::vector<StatsJob> &jobs);
kx_price_result finish(const Stats &s);

// Path-kernel valuation of several contracts on one grid with one model and
// seed (engine.cu).
std::vector<Stats> batch_paths(Ctx &c, const std::vector<const Program *> &progs, const Model &m,
                               const kx_mc_config &cfg, const std::vector<double> &grid);

// Portfolio prices (hard barriers) with pathwise sensitivities (adjoint.cu).
void portfolio_adjoint(Ctx &c, size_t n, const kx_program *const *progs, const kx_model *models,
                       const kx_mc_config *cfgs, kx_price_result *out, kx_sens *sens);

}  // namespace kx
