// The IEEE quotient y / b of many doubles by one divisor.
//
// With r = RN(1 / b) and a quotient estimate q within one ulp of y / b, the
// remainder rem = y - q b is exact in one FMA and RN(q + rem r) is the correctly
// rounded quotient (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990, theorem on
// division).  q = y r + y rl, with rl = (1 - b r) r the reciprocal's own
// rounding error, is within one ulp for every mantissa.  One reciprocal serves
// all values: four FMA-pipe operations per value instead of a division of its
// own.  The remainder is exact and nothing overflows while |y| and |b| lie within
// [2^-500, 2^500), and for y = +0 every operation gives +0.  Other values (-0,
// infinities and NaN among them) are divided with the ordinary operator.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace ms3gpu {

// 2^-500 <= |y| < 2^500, from the exponent field
__host__ __device__ inline bool quotient_range(double y) {
#ifdef __CUDA_ARCH__
    const uint32_t hi = (uint32_t)__double2hiint(y);
#else
    uint64_t bits;
    std::memcpy(&bits, &y, 8);
    const uint32_t hi = (uint32_t)(bits >> 32);
#endif
    return (hi & 0x7FF00000u) - (523u << 20) < (1000u << 20);
}

struct Reciprocal {
    double r, rl;
    bool in_range;
};

__host__ __device__ inline Reciprocal reciprocal_of(double b) {
    Reciprocal c;
#ifdef __CUDA_ARCH__
    c.r = __drcp_rn(b);
    c.rl = __dmul_rn(__fma_rn(-b, c.r, 1.0), c.r);
#else
    c.r = 1.0 / b;
    c.rl = std::fma(-b, c.r, 1.0) * c.r;
#endif
    c.in_range = quotient_range(b);
    return c;
}

// y / b for |y| and |b| in range, or y = +0 and b > 0 in range
__host__ __device__ inline double quotient_in_range(double y, double b, const Reciprocal& c) {
#ifdef __CUDA_ARCH__
    const double q = __fma_rn(y, c.r, __dmul_rn(y, c.rl));
    const double rem = __fma_rn(-q, b, y);
    return __fma_rn(rem, c.r, q);
#else
    const double q = std::fma(y, c.r, y * c.rl);
    const double rem = std::fma(-q, b, y);
    return std::fma(rem, c.r, q);
#endif
}

}  // namespace ms3gpu
