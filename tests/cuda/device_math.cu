// Device code of the engine run on inputs of the tests' choice
// (test_gpu_device_math.py builds and loads this file): each check counts the
// inputs on which the engine's form and CUDA's own function differ.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../kontracts_gb300/csrc/lsm_common.cuh"
#include "../../kontracts_gb300/csrc/paths_sync.cuh"

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

// The FP32 normals of every first word (with second words spread over their range) against the
// same pair with CUDA's logarithm.
__global__ void k_normal_pairs(unsigned long long *bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (1ull << 32);
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = (uint32_t)i, b = a * 0x9E3779B9u;
        float z0, z1, s, c;
        kx::box_muller(a, b, z0, z1);
        const float r = kx::sqrt_approx(-2.0f * __logf(fmaf(__uint2float_rn(a), 0x1p-32f, 0x1p-33f)));
        __sincosf(6.283185307179586f * fmaf(__uint2float_rn(b), 0x1p-32f, 0x1p-33f - 0.5f), &s, &c);
        if (!same(z0, -r * c) || !same(z1, -r * s)) atomicAdd(bad, 1ull);
    }
}

// e^y without subnormal results at the FP32 values of magnitude bits b0 .. b0 + n - 1 and of the
// sign, against __expf.
__global__ void k_tame_exp(uint32_t sign, uint32_t b0, uint32_t n, unsigned long long *bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float y = __uint_as_float((b0 + (uint32_t)i) | (sign << 31));
        if (!same(kx::block_exp<true>(y), __expf(y))) atomicAdd(bad, 1ull);
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

long long check_normal_pairs() {
    return counted([&](unsigned long long *bad) { k_normal_pairs<<<4096, 256>>>(bad); });
}

long long check_tame_exp(uint32_t sign, uint32_t b0, uint32_t n) {
    return counted([&](unsigned long long *bad) { k_tame_exp<<<1024, 256>>>(sign, b0, n, bad); });
}

}
