// Device code of the engine run on inputs of the tests' choice
// (test_gpu_device_math.py builds and loads this file): each check counts the
// inputs on which the engine's form and CUDA's own function differ.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../kontracts_gb300/csrc/lsm_common.cuh"

namespace {

using kx::lsm_basis_f32;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// The first weighted regression function at x, bits b0 .. b0 + n - 1 of x, against __expf(-x / 2).
__global__ void k_basis_weight(uint32_t b0, uint32_t n, unsigned long long *bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(b0 + (uint32_t)i);
        float phi[3];
        lsm_basis_f32<3, KX_LSM_LAGUERRE>(x, phi);
        if (!same(phi[0], __expf(-0.5f * x))) atomicAdd(bad, 1ull);
    }
}

// Runs `launch(counter)` and returns the count, or -1 - the CUDA error.
template <class F>
long long counted(F launch) {
    unsigned long long *bad = nullptr, h = 0;
    cudaError_t e = cudaMalloc(&bad, sizeof h);
    if (e == cudaSuccess) e = cudaMemset(bad, 0, sizeof h);
    if (e == cudaSuccess) {
        launch(bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&h, bad, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return e == cudaSuccess ? (long long)h : -1 - (long long)e;
}

}  // namespace

extern "C" {

long long check_basis_weight(uint32_t b0, uint32_t n) {
    return counted([&](unsigned long long *bad) { k_basis_weight<<<1024, 256>>>(b0, n, bad); });
}

}
