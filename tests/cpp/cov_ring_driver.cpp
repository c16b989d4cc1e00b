// The stage ring of the tensor-core covariance on the host: a producer whose copies land
// after random times and out of order, two converter groups of several warps that take the
// stages in turn through converter_may_take, and MMAs that read the planes in order, on
// barriers with an mbarrier's phases and parity test, stepped in random order.  Prints the
// stages converted, how many were taken before their tiles had landed or their slot's
// planes had been read, and how many arrivals met a phase that expected none.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "cov_ring.h"

static long over = 0;

struct Barrier {
    int count, pending, tx = 0;
    long phase = 0;
    explicit Barrier(int c) : count(c), pending(c) {}
    void settle() {
        if (pending == 0 && tx == 0) {
            phase++;
            pending = count;
        }
    }
    void arrive() {
        if (pending == 0) over++;
        else pending--;
        settle();
    }
    void expect() {
        tx++;
        arrive();
    }
    void land() {
        tx--;
        settle();
    }
    bool test(uint32_t parity) const { return (uint32_t)(phase & 1) != parity; }  // the phase of that parity is over
};

int main() {
    constexpr int S = 3, kWarps = 3;  // slots; warps of a group
    long total = 0, early = 0;
    for (unsigned seed = 0; seed < 400; seed++) {
        std::mt19937 rng(seed);
        auto chance = [&](int n) { return (int)(rng() % (unsigned)n) == 0; };
        const long n = 300;
        std::vector<Barrier> full(S, Barrier(1)), empty(S, Barrier(kWarps)), planes(S, Barrier(kWarps)), read(S, Barrier(1));
        std::vector<char> landed(n, 0), consumed(n, 0);
        long issued = 0, mma = 0;
        struct Warp {
            long g;
            bool saw_read = false, saw_tiles = false;  // waits of stage g that have returned
        };
        std::vector<Warp> warps[2];
        for (int g = 0; g < 2; g++) warps[g].assign(kWarps, Warp{g});
        std::vector<long> flying;
        const int slow = 1 + (int)(seed % 40);  // of the copies
        long steps = 0;
        while (mma < n && steps++ < 2000000) {
            switch (rng() % 4) {
                case 0:  // producer
                    if (issued < n && (issued < S || empty[issued % S].test((uint32_t)((issued / S - 1) & 1)))) {
                        full[issued % S].expect();
                        flying.push_back(issued++);
                    }
                    break;
                case 1:  // a copy lands
                    if (!flying.empty() && chance(slow)) {
                        const size_t k = rng() % flying.size();
                        const long g = flying[k];
                        flying.erase(flying.begin() + (long)k);
                        landed[g] = 1;
                        full[g % S].land();
                    }
                    break;
                case 2: {  // a converter warp
                    Warp& w = warps[rng() % 2][rng() % kWarps];
                    const long g = w.g;
                    if (g >= n) break;
                    const int s = (int)(g % S);
                    // a wait that has returned is not made again
                    auto wait = [](bool& saw, const Barrier& b, uint32_t p) { return saw = saw || b.test(p); };
                    if (!ms3gpu::converter_may_take(
                            g, S, (uint32_t)((g / S) & 1), [&](uint32_t p) { return wait(w.saw_read, read[s], p); },
                            [&](uint32_t p) { return wait(w.saw_tiles, full[s], p); }))
                        break;
                    early += !landed[g] || (g >= S && !consumed[g - S]);
                    total++;
                    empty[s].arrive();
                    planes[s].arrive();
                    w = Warp{g + 2};
                    break;
                }
                default:  // MMAs
                    if (planes[mma % S].test((uint32_t)((mma / S) & 1)) && chance(2)) {
                        consumed[mma] = 1;
                        read[mma % S].arrive();
                        mma++;
                    }
            }
        }
    }
    std::printf("%ld %ld %ld\n", total, early, over);
    return 0;
}
