// paths_knock.cu — instantiations of k_knock (one-flow knock-outs, GBM).
#include "paths_knock.cuh"

namespace kx {

const void *knock_kernel(bool f64) {
    return f64 ? (const void *)&k_knock<double, 3> : (const void *)&k_knock<float, 4>;
}

}  // namespace kx
