// paths_sync.cu — instantiations of k_sync (static schedules without barriers)
// and the table of normals that launches of one stream share.
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

}  // namespace kx
