// paths_sync.cu — instantiations of k_sync (static schedules without barriers).
#include "paths_sync.cuh"

namespace kx {

template <class Real, int MODEL, int MINB>
static const void *sync_pick(bool acc) {
    return acc ? (const void *)&k_sync<Real, MODEL, MINB, true> : (const void *)&k_sync<Real, MODEL, MINB, false>;
}

const void *sync_kernel(int model, bool f64, bool acc) {
    if (model == KX_MODEL_GBM) return f64 ? sync_pick<double, M_GBM, 2>(acc) : sync_pick<float, M_GBM, 4>(acc);
    return f64 ? sync_pick<double, M_HESTON, 2>(acc) : sync_pick<float, M_HESTON, 4>(acc);
}

}  // namespace kx
