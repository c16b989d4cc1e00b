// Host run of div_by.cuh: quotients of zero.  Prints the number of
// divisors tried and of quotients whose bits differ from the ordinary division's.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "div_by.cuh"

int main() {
    int tried = 0, bad = 0;
    for (int e = -499; e < 500; e++)
        for (double m = 1.0; m < 2.0; m += 1.0 / 64 + 1e-9) {
            const double b = std::ldexp(m, e);
            const ms3gpu::Reciprocal c = ms3gpu::reciprocal_of(b);
            const double q = ms3gpu::quotient_in_range(0.0, b, c), ref = 0.0 / b;
            bad += std::memcmp(&q, &ref, 8) != 0;
            tried += c.in_range;
        }
    std::printf("%d %d\n", tried, bad);
    return 0;
}
