// Host run of div_by.cuh: quotients by one divisor against the ordinary
// division, bit for bit.  Prints the number of values tried and of differences.
#include <cinttypes>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "div_by.cuh"

static uint64_t state = 1;
static uint64_t next64() {  // splitmix64
    uint64_t z = (state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double from_bits(uint64_t b) {
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}
// mantissas where rounding errors are largest: near 1, near 2, and random ones
static double value(int span) {
    uint64_t m = next64() & 0xFFFFFFFFFFFFFull;
    switch (next64() & 7) {
        case 0: m = next64() & 0xFF; break;
        case 1: m = 0xFFFFFFFFFFFFFull - (next64() & 0xFF); break;
        case 2: m &= 0xFFFFFF8000000ull; break;
        default: break;
    }
    const int64_t e = (int64_t)(next64() % (uint64_t)(2 * span + 1)) - span;
    return from_bits(((next64() & 1) << 63) | ((uint64_t)(1023 + e) << 52) | m);
}

int main(int argc, char** argv) {
    const int64_t divisors = argc > 1 ? std::atoll(argv[1]) : 1000;
    const int span = argc > 2 ? std::atoi(argv[2]) : 499;
    int64_t tried = 0, bad = 0;
    for (int64_t k = 0; k < divisors; k++) {
        const double b = std::fabs(value(span));
        const ms3gpu::Reciprocal c = ms3gpu::reciprocal_of(b);
        for (int i = 0; i < 1000; i++) {
            const double y = value(span);
            if (!c.in_range || !ms3gpu::quotient_range(y)) continue;
            const double q = ms3gpu::quotient_in_range(y, b, c), ref = y / b;
            tried++;
            bad += std::memcmp(&q, &ref, 8) != 0;
        }
    }
    std::printf("%" PRId64 " %" PRId64 "\n", tried, bad);
    return 0;
}
