// Which (run, block pair) items of the tensor-core covariance each CTA takes.
//
// An off-diagonal item takes 0.85 us per 32 timepoints, a diagonal one 0.61.  The
// off-diagonal items of all runs are dealt to the CTAs in turn, run by run; the
// diagonal items then fill the CTAs up to one level: a CTA that got one
// off-diagonal item fewer than the others takes a diagonal item before the rest
// are dealt to all CTAs in turn, those CTAs first.  (With two, which would be
// right at half the cost, 384 channels x 300 k timepoints took 440 us, with one 387.)
// CTAs that run at the same time work on neighbouring runs, whose rows they
// share through L2.
#ifndef MS3_COV_SHARE_H
#define MS3_COV_SHARE_H

#include <cstdint>

#ifdef __CUDACC__
#define MS3_SHARE_HD __host__ __device__
#else
#define MS3_SHARE_HD
#endif

namespace ms3gpu {

struct CovShare {
    int64_t n_off, n_diag;  // items of each kind in the call
    int64_t c, G;           // this CTA, the grid
    int64_t late;           // CTAs c >= late have one off-diagonal item fewer
    int nb;                 // 128-channel blocks

    MS3_SHARE_HD CovShare(int64_t nruns, int nb_, int64_t cta, int64_t grid)
        : n_off(nruns * (nb_ * (nb_ - 1) / 2)), n_diag(nruns * nb_), c(cta), G(grid), late(n_off % grid), nb(nb_) {}

    // items dealt in turn to `width` CTAs, of which this one is number `at`
    MS3_SHARE_HD static int64_t dealt(int64_t n, int64_t at, int64_t width) {
        return n > at ? (n - 1 - at) / width + 1 : 0;
    }
    MS3_SHARE_HD int64_t off_items() const { return dealt(n_off, c, G); }
    MS3_SHARE_HD int64_t first() const {  // diagonal items that fill up the late CTAs
        const int64_t f = n_off > 0 ? G - late : 0;
        return f < n_diag ? f : n_diag;
    }
    MS3_SHARE_HD int64_t first_items() const { return c >= late ? dealt(first(), c - late, G - late) : 0; }
    MS3_SHARE_HD int64_t items() const { return off_items() + first_items() + dealt(n_diag - first(), G - 1 - c, G); }

    // run and blocks of this CTA's item i (0 <= i < items())
    MS3_SHARE_HD void item(int64_t i, int64_t& r, int& bi, int& bj) const {
        const int64_t no = off_items(), nf = first_items();
        if (i < no) {
            const int64_t w = i * G + c;
            const int per = nb * (nb - 1) / 2;
            r = w / per;
            int p = (int)(w % per);
            bi = 0;
            while (p >= nb - 1 - bi) p -= nb - 1 - bi++;
            bj = bi + 1 + p;
            return;
        }
        const int64_t w = i < no + nf ? (i - no) * (G - late) + (c - late) : first() + (i - no - nf) * G + (G - 1 - c);
        r = w / nb;
        bi = bj = (int)(w % nb);
    }
};

}  // namespace ms3gpu

#endif
