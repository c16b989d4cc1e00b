// The reference's rounding of whitened values to multiples of 1e-4,
//     floor(x / 0.0001 + 0.5) * 0.0001   in double, stored as float
// (packages/ms3/p_whiten.cpp:31-41), in six FP32 operations with the same bits for
// |x| < kQuantizeRange.
//
// For a float x the double quotient equals x * 10000 (at most 38 significant bits), so
// the integer is f = floor(10000 x + 0.5) in exact arithmetic.  Rounding 10000 x + 0.5
// down to a float (one FMA) does not change its floor, since below 2^23 every integer
// is a float, and adding 1.5 * 2^23 rounding down drops the fraction.  The double product
// f * 0.0001 rounded to float is f / 10000 rounded once (for |f| < 2^23 that lies 2^-40
// or more, relative, from a float tie), formed as a product by 1e-4 and one
// exact-remainder correction.
#pragma once

#include <cfenv>
#include <cmath>

namespace ms3gpu {

constexpr float kQuantizeRange = 400.0f;

// |x| < kQuantizeRange
__host__ __device__ inline float quantize_1e4_small(float x) {
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
#ifdef __CUDA_ARCH__
    const float f = __fadd_rn(__fadd_rd(__fmaf_rd(x, 10000.0f, 0.5f), kMagic), -kMagic);
    const float q = __fmul_rn(f, 1e-4f);
    return __fmaf_rn(__fmaf_rn(-q, 10000.0f, f), 1e-4f, q);
#else
    const int mode = std::fegetround();
    std::fesetround(FE_DOWNWARD);
    const volatile float t = std::fma(x, 10000.0f, 0.5f);
    const volatile float n = t + kMagic;
    std::fesetround(mode);
    const float f = n - kMagic;
    const float q = f * 1e-4f;
    return std::fma(std::fma(-q, 10000.0f, f), 1e-4f, q);
#endif
}

}  // namespace ms3gpu
