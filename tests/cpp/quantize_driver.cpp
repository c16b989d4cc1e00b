// Host run of quantize.cuh against floor(x / 0.0001 + 0.5) * 0.0001 in double, for every
// n-th float below its range and both signs.  Prints values tried and differences.
#define __host__
#define __device__
#include "quantize.cuh"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

int main(int argc, char** argv) {
    const uint64_t step = argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1;
    uint32_t limit;
    const float range = ms3gpu::kQuantizeRange;
    std::memcpy(&limit, &range, 4);
    uint64_t tried = 0, bad = 0;
    for (uint64_t b = 0; b < limit; b += step)
        for (uint32_t sign : {0u, 0x80000000u}) {
            const uint32_t u = (uint32_t)b | sign;
            float x;
            std::memcpy(&x, &u, 4);
            const float want = (float)(std::floor((double)x / 0.0001 + 0.5) * 0.0001);
            const float got = ms3gpu::quantize_1e4_small(x);
            tried++;
            bad += std::memcmp(&want, &got, 4) != 0;
        }
    std::printf("%llu %llu\n", (unsigned long long)tried, (unsigned long long)bad);
    return 0;
}
