// Device code of the engine run on inputs of the tests' choice
// (test_gpu_device_math.py builds and loads this file): each check counts the
// inputs on which the engine's form and CUDA's own function differ.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../kontracts_gb300/csrc/discount.cuh"
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

__device__ uint64_t mix(uint64_t z) {  // SplitMix64's finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Amounts times discount factors of one kind against the FP64 product: 0 spread over all
// mantissas, 1 and 2 products whose lost part is exactly half (76 and 77 bits wide), 3 one unit
// beside it, 4 mantissas of ones (carries into the exponent), 5 amounts that are zero, subnormal,
// infinite or not numbers, 6 factors that are zero, negative, tiny, huge or not finite.
__global__ void k_discount(int kind, uint32_t n, unsigned long long *bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = mix(2 * i + 1), q = mix(2 * i + 2);
        uint32_t m = (uint32_t)r & 0x7FFFFFu, e = 1u + (uint32_t)(r >> 32) % 254u;
        uint64_t d = q & 0xFFFFFFFFFFFFFull, de = 512u + (q >> 52) % 1025u;
        if (kind >= 1 && kind <= 3) {
            m |= 1u;
            uint32_t inv = 1u;  // 1 / (2^23 + m) mod 2^24, by Newton's iteration
            for (int t = 0; t < 5; ++t) inv *= 2u - ((m | 0x800000u) * inv);
            const uint32_t bits = kind == 1 ? 23u : 24u;
            const uint32_t low = ((1u << (bits - 1u)) * inv) & ((1u << bits) - 1u);
            d = (d & ~(uint64_t)((1u << bits) - 1u)) | low;
            if (kind == 3) d += (i & 1u) ? 1u : (uint64_t)-1;
            d &= 0xFFFFFFFFFFFFFull;
        } else if (kind == 4) {
            m = 0x7FFFFFu - (uint32_t)(r >> 40) % 4u;
            d = 0xFFFFFFFFFFFFFull - (q >> 40) % 4u;
        } else if (kind == 5) {
            e = (i & 1u) ? 0u : 255u;
            if (i % 3u == 0u) m = 0u;
        } else if (kind == 6) {
            de = (i % 5u == 0u) ? 0u : (i % 5u == 1u) ? 2047u : (i % 5u == 2u) ? 511u : (i % 5u == 3u) ? 1537u : 0x800u | 1000u;
            if (i % 7u == 0u) d = 0u;
        }
        const float x = __uint_as_float(m | (e << 23) | ((uint32_t)(r >> 63) << 31));
        const double df = __longlong_as_double((long long)(d | (de << 52)));
        const double got = kx::discount_product(x, df, kx::discount_bits(df)), want = __dmul_rn((double)x, df);
        const bool ok = got != got ? want != want : __double_as_longlong(got) == __double_as_longlong(want);
        if (!ok) atomicAdd(bad, 1ull);
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

long long check_discount(int kind, uint32_t n) {
    return counted([&](unsigned long long *bad) { k_discount<<<1024, 256>>>(kind, n, bad); });
}

}
