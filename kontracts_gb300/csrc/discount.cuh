// discount.cuh — an FP32 amount times its FP64 discount factor, rounded as the
// FP64 product, in integer arithmetic (k_flows_walk).
#pragma once
#include <cstdint>

namespace kx {

// A discount factor as a 53-bit integer and an exponent, for discount_product.
struct DiscountBits {
    uint64_t mant;
    int expo;  // biased exponent field, or 0: use FP64
};
__device__ __forceinline__ DiscountBits discount_bits(double df) {
    const uint64_t b = (uint64_t)__double_as_longlong(df);
    const int e = (int)(b >> 52);
    if (e < 512 || e > 1536) return DiscountBits{0, 0};  // negative, tiny, huge, not finite
    return DiscountBits{(b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull, e};
}
// (out of line, so that the product below does not compute it beside its own)
__device__ __noinline__ double discount_fp64(float x, double df) { return (double)x * df; }
// (double)x * df rounded to nearest-even: the 24-bit significand of x times the
// 53-bit one of df is 76 or 77 bits, of which the top 53 are kept.
__device__ __forceinline__ double discount_product(float x, double df, const DiscountBits &d) {
    const uint32_t b = __float_as_uint(x), e8 = (b >> 23) & 0xFFu, sign = b & 0x80000000u;
    if ((b << 1) == 0u && d.expo) return __hiloint2double((int)sign, 0);
    if (e8 == 0u || e8 == 255u || !d.expo) return discount_fp64(x, df);
    const uint32_t m = (b & 0x7FFFFFu) | 0x800000u;
    const uint64_t lo = (uint64_t)m * (uint32_t)d.mant;
    const uint64_t hi = (uint64_t)m * (uint32_t)(d.mant >> 32) + (lo >> 32);  // the product: hi 2^32 + low word
    const uint32_t low = (uint32_t)lo;
    const uint32_t up = (uint32_t)(hi >> 44);        // 1: 77 bits
    const uint32_t sh = 9u - up;                     // bits taken from the low word
    const uint64_t mant = (hi << sh) | (low >> (32u - sh));
    const uint32_t rest = low << sh;                 // what is rounded away, from the top of the word
    const uint64_t inc = rest > 0x80000000u || (rest == 0x80000000u && (mant & 1u)) ? 1u : 0u;
    const uint64_t ef = (uint64_t)(e8 + (uint32_t)d.expo + up - 127u);
    const uint64_t bits = ((ef - 1u) << 52) + mant + inc;  // mant's leading bit adds 1 to the field; so does a carry
    return __longlong_as_double((long long)(bits | ((uint64_t)sign << 32)));
}
__device__ __forceinline__ double discount_product(double x, double df, const DiscountBits &) { return x * df; }

}  // namespace kx
