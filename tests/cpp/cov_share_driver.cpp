// Deals the items of many (runs, blocks, grid) shapes with CovShare: every (run, pair)
// once, and no CTA's level (an off-diagonal item counting 4, a diagonal one 3) more than
// one off-diagonal item above the mean.  Prints the shapes tried and those that fail.
#include <cstdio>
#include <set>
#include <tuple>

#include "cov_share.h"

int main() {
    long tried = 0, bad = 0;
    for (int nb : {1, 2, 3, 4, 7, 17, 22})
        for (long runs : {1, 2, 3, 5, 23, 37, 46, 92, 147, 148, 149, 300})
            for (long sms : {1, 2, 3, 147, 148}) {
                const long n = runs * nb * (nb + 1) / 2, G = n < sms ? n : sms;
                std::set<std::tuple<long, int, int>> seen;
                long count = 0, top = 0;
                bool ok = true;
                for (long c = 0; c < G; c++) {
                    const ms3gpu::CovShare s(runs, nb, c, G);
                    long level = 0;
                    for (long i = 0; i < s.items(); i++, count++) {
                        int64_t r;
                        int bi, bj;
                        s.item(i, r, bi, bj);
                        ok = ok && r >= 0 && r < runs && bi >= 0 && bi <= bj && bj < nb;
                        seen.insert({(long)r, bi, bj});
                        level += bi == bj ? 3 : 4;
                    }
                    top = level > top ? level : top;
                }
                ok = ok && count == n && (long)seen.size() == n;
                ok = ok && top * G <= runs * (3 * nb + 2 * nb * (nb - 1)) + 4 * G;
                tried++;
                bad += !ok;
            }
    std::printf("%ld %ld\n", tried, bad);
    return 0;
}
