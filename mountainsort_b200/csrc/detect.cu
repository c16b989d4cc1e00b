// Event detection of mountainsortalg on the whitened timeseries, the first
// consumer of the filter + whiten output:
//   detect_events (packages/mountainsortalg/detect_events.cpp:69-135) as
//   NeighborhoodSorter::addTimeChunk applies it (neighborhoodsorter.cpp:74-100)
//   to the central channel of every neighborhood over the time chunks of
//   p_mountainsort3.cpp:190-215 / get_time_chunk_infos (:507-533).
//
// Per (channel, time chunk), with the chunk [t1 - pad, t1 + size + pad) read
// with zeros outside the recording (readChunk's zero fill):
//   1. the chunk's mean and sample stdev in double, with the bits of a sum in
//      index order (MLCompute::mean / stdev, common/mlcompute.cpp:67-85);
//   2. the candidates -- samples whose signed (or absolute, for sign 0)
//      deviation from the mean exceeds threshold * stdev -- counted and written
//      in time order, a thread per (channel, segment of samples);
//   3. the reference's greedy strongest-within-detect_interval rule.  Between
//      candidates more than the interval apart it starts afresh, so a thread
//      takes each run of closer ones;
//   4. the kept times inside [t1, t1 + size), channel after channel.
//
// The index-order sums are what a long recording waits for if one thread forms
// them (two dependent FP64 additions per sample: 59 ms for 64 channels x 1.8M,
// one chunk).  With thousands of (channel, chunk) pairs a thread does (serial_stats);
// fewer are formed in parallel with the same bits:
//   sum of x    When every partial sum is a multiple of 2^q and at most
//               2^(53 + q) in magnitude, no addition rounds and any order gives
//               the value.  2^q divides the samples (floats) and the sum so far;
//               |sum so far| + sum |x| bounds the partial sums.
//   sum of x^2  The squares are exact in double.  While the sum stays in one
//               binade [2^E, 2^(E+1)), an addition moves it by a multiple of u =
//               2^(E-52) that depends on the square and, for ties, on whether sum
//               / u is even.  So a segment moves it by one of two amounts, found
//               by adding the segment to 2^E and to 2^E + u; the amounts of
//               consecutive segments compose.
// detect_segments and detect_binades find E for each segment from approximate
// sums, detect_increments the two amounts, and detect_stats, a warp per (channel,
// chunk), puts the segments together 32 at a time, checks every condition against
// the exact sums, and adds up a segment sample by sample where one fails: a binade is
// crossed (about 20 times in a chunk), infinities, NaN, or 2^q is too fine for the sum
// (values rounded to 1e-4: none; unrounded floats: up to a third of the segments).  A
// segment of zeros adds nothing.
// 64 channels x 1.8M timepoints in one chunk, whole call, serially and by segments: 75 and
// 1.1 ms for values rounded to 1e-4, 9 ms for unrounded ones, 26 ms for values over 40
// octaves.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

#include "common.cuh"
#include "detect.h"

namespace ms3gpu {

namespace {

constexpr int kSeg = 512;    // samples per segment at most
constexpr int kShortSeg = 64;  // where there are few of them (segment_length)
constexpr int kBatch = 16;   // samples loaded together

struct ChunkStats {
    double mean, threshold2;
};

struct Dims {
    int64_t M, N, chunk, pad, nchunks, nseg;  // nseg: segments of the longest chunk
    int seg;                                  // samples per segment
};

__device__ __forceinline__ int64_t chunk_size_at(int64_t c, int64_t chunk, int64_t N) {
    const int64_t t1 = c * chunk;
    return (chunk < N - t1) ? chunk : N - t1;
}

// Calls f(n, x) for the samples n in [a, e) of chunk c of channel m in order
// (x = 0 outside the recording), B loads in flight.
template <int B = kBatch, class F>
__device__ __forceinline__ void for_samples(const float* __restrict__ X, const Dims& d, int64_t m, int64_t c, int64_t a,
                                            int64_t e, F f) {
    const int64_t t0 = c * d.chunk - d.pad;
    for (int64_t n0 = a; n0 < e; n0 += B) {
        float x[B];
        const int64_t t = t0 + n0;
        if (t >= 0 && t + B <= d.N && n0 + B <= e) {
            const float* p = X + t * d.M + m;
#pragma unroll
            for (int k = 0; k < B; k++) x[k] = __ldg(p + (int64_t)k * d.M);
#pragma unroll
            for (int k = 0; k < B; k++) f(n0 + k, x[k]);
        } else {
#pragma unroll
            for (int k = 0; k < B; k++)
                x[k] = (n0 + k < e && t + k >= 0 && t + k < d.N) ? X[(t + k) * d.M + m] : 0.f;
#pragma unroll
            for (int k = 0; k < B; k++)
                if (n0 + k < e) f(n0 + k, x[k]);
        }
    }
}

// The (channel, segment) of a thread of the segment kernels: neighbouring threads
// take neighbouring channels; blockIdx.y is the chunk.
struct Work {
    int64_t m, c, s, a, e;
    int64_t slot;  // (m, c, s) in channel-major order
    bool any;
};
__device__ __forceinline__ Work segment_work(const Dims& d) {
    Work w;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    w.s = i / d.M;
    w.m = i - w.s * d.M;
    w.c = blockIdx.y;
    const int64_t len = chunk_size_at(w.c, d.chunk, d.N) + 2 * d.pad;
    w.a = w.s * d.seg;
    w.e = w.a + d.seg < len ? w.a + d.seg : len;
    w.any = w.s < d.nseg;
    w.slot = (w.m * d.nchunks + w.c) * d.nseg + w.s;
    return w;
}

// Per segment: sum of x (in order), of |x| (rounded up) and of x^2 (approximate),
// and the bits of the smallest non-zero |x| (0: none).
__global__ void __launch_bounds__(256) detect_segments(const float* __restrict__ X, Dims d, double* __restrict__ seg_x,
                                                       float* __restrict__ seg_abs, double* __restrict__ seg_sq,
                                                       uint32_t* __restrict__ seg_min) {
    const Work w = segment_work(d);
    if (!w.any) return;
    double sx = 0.0, sa = 0.0, sq = 0.0;
    uint32_t least = 0xFFFFFFFFu;  // of |x| bits minus one: zero wraps to the largest
    for_samples(X, d, w.m, w.c, w.a, w.e, [&](int64_t, float x) {
        const double v = (double)x;
        sx += v;
        sa += fabs(v);
        sq = fma(v, v, sq);
        least = min(least, (__float_as_uint(x) & 0x7FFFFFFFu) - 1u);
    });
    seg_x[w.slot] = sx;
    seg_abs[w.slot] = __double2float_ru(sa * (1.0 + 1e-12));
    seg_sq[w.slot] = sq;
    seg_min[w.slot] = least + 1u;
}

constexpr int kNoBinade = -100000;

__device__ __forceinline__ ChunkStats stats_of(double sum, double sumsqr, int64_t len, double detect_threshold) {
    const double ct = (double)len;
    const double mean = __ddiv_rn(sum, ct);
    const double stdev =
        len >= 2 ? sqrt(__ddiv_rn(__dsub_rn(sumsqr, __ddiv_rn(__dmul_rn(sum, sum), ct)), ct - 1.0)) : 0.0;
    return {mean, __dmul_rn(detect_threshold, stdev)};
}

// The statistics of one (channel, chunk) per thread, sample by sample: where there are
// enough of them to fill the GPU (serial_stats).
__global__ void __launch_bounds__(32) detect_stats_serial(const float* __restrict__ X, Dims d, double detect_threshold,
                                                          ChunkStats* __restrict__ stats) {
    const int64_t i = (int64_t)blockIdx.x * 32 + threadIdx.x;
    if (i >= d.M * d.nchunks) return;
    const int64_t c = i / d.M, m = i - c * d.M;
    const int64_t len = chunk_size_at(c, d.chunk, d.N) + 2 * d.pad;
    double sum = 0.0, sumsqr = 0.0;
    for_samples<32>(X, d, m, c, 0, len, [&](int64_t, float x) {
        const double v = (double)x;
        sum = __dadd_rn(sum, v);
        sumsqr = __dadd_rn(sumsqr, __dmul_rn(v, v));
    });
    stats[i] = stats_of(sum, sumsqr, len, detect_threshold);
}

__device__ __forceinline__ int binade_of(double x) {  // floor(log2 x) for normal x > 0
    const int e = (__double2hiint(x) >> 20) & 0x7FF;
    return (x > 0.0 && e > 60 && e < 2046) ? e - 1023 : kNoBinade;
}

__device__ __forceinline__ double two_to(int k) { return __hiloint2double((k + 1023) << 20, 0); }  // normal range

// Per segment: the binade of the approximate sum of squares before it.  One warp
// per (channel, chunk).
__global__ void __launch_bounds__(128) detect_binades(const double* __restrict__ seg_sq, int64_t MC, int64_t nseg,
                                                      int* __restrict__ seg_e) {
    const int64_t k = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int l = threadIdx.x & 31;
    if (k >= MC) return;
    double before = 0.0;
    for (int64_t s0 = 0; s0 < nseg; s0 += 32) {
        const int64_t s = s0 + l;
        const double own = s < nseg ? seg_sq[k * nseg + s] : 0.0;
        double incl = own;
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, incl, o);
            if (l >= o) incl += up;
        }
        const double first = __shfl_up_sync(0xffffffffu, incl, 1);
        if (s < nseg) seg_e[k * nseg + s] = binade_of(before + (l ? first : 0.0));
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// Per segment: what it adds, in units of u, to a sum of squares in its binade whose
// value / u is even (inc0) or odd (inc1); -1 when the binade is not known or has no
// room.
__global__ void __launch_bounds__(256) detect_increments(const float* __restrict__ X, Dims d,
                                                         const double* __restrict__ seg_sq,
                                                         const int* __restrict__ seg_e, int64_t* __restrict__ seg_inc0,
                                                         int64_t* __restrict__ seg_inc1) {
    const Work w = segment_work(d);
    if (!w.any) return;
    const int E = seg_e[w.slot];
    int64_t k0 = -1, k1 = -1;
    if (E != kNoBinade && seg_sq[w.slot] < 0.999 * two_to(E)) {
        const double c0 = two_to(E), u = two_to(E - 52), c1 = c0 + u;
        double s0 = c0, s1 = c1;
        for_samples(X, d, w.m, w.c, w.a, w.e, [&](int64_t, float x) {
            const double v = (double)x;
            const double sq = __dmul_rn(v, v);
            s0 = __dadd_rn(s0, sq);
            s1 = __dadd_rn(s1, sq);
        });
        // both lie in [2^E, 2^(E+1)): their bits count units of u
        if (s0 < 2.0 * c0 && s1 < 2.0 * c0) {
            k0 = __double_as_longlong(s0) - __double_as_longlong(c0);
            k1 = __double_as_longlong(s1) - __double_as_longlong(c1);
        }
    }
    seg_inc0[w.slot] = k0;
    seg_inc1[w.slot] = k1;
}

// The exponent of the lowest set bit of a double (large for zero; infinities and
// NaN end in sums that fail the bound).
__device__ __forceinline__ int lowest_bit(double x) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7FF);
    const long long f = b & 0xFFFFFFFFFFFFFll;
    if (e == 0) return f == 0 ? 100000 : __ffsll(f) - 1 - 1074;
    return f == 0 ? e - 1023 : e - 1075 + __ffsll(f) - 1;
}

// A lower bound of that exponent for every non-zero float of at least these
// magnitude bits.
__device__ __forceinline__ int float_grid(uint32_t bits) {
    return bits == 0 ? 100000 : max((int)(bits >> 23), 1) - 150;
}

// Whether additions whose partial sums are multiples of 2^q and at most `bound` in
// magnitude are all exact.
__device__ __forceinline__ bool sums_exact(double bound, int q) {
    if (q > 900) return bound < 1e300;
    return q > -1000 && bound <= two_to(q + 53);
}

// The reference's statistics of one (channel, chunk) per warp.
constexpr int kStatWarps = 2;
template <int SEG>  // d.seg
__global__ void __launch_bounds__(32 * kStatWarps) detect_stats(const float* __restrict__ X, Dims d,
                                                               double detect_threshold,
                                                               const double* __restrict__ seg_x,
                                                               const float* __restrict__ seg_abs,
                                                               const uint32_t* __restrict__ seg_min,
                                                               const int* __restrict__ seg_e,
                                                               const int64_t* __restrict__ seg_inc0,
                                                               const int64_t* __restrict__ seg_inc1,
                                                               ChunkStats* __restrict__ stats) {
    __shared__ __align__(16) float staged[kStatWarps][SEG];
    const int l = threadIdx.x & 31;
    const int64_t k = (int64_t)blockIdx.x * kStatWarps + (threadIdx.x >> 5);
    if (k >= d.M * d.nchunks) return;
    float* mine = staged[threadIdx.x >> 5];
    const int64_t m = k / d.nchunks, c = k - m * d.nchunks;
    const int64_t t1 = c * d.chunk;
    const int64_t len = chunk_size_at(c, d.chunk, d.N) + 2 * d.pad;
    const int64_t nseg = (len + SEG - 1) / SEG;
    double sum = 0.0, sumsqr = 0.0;

    auto one_by_one = [&](int64_t s) {
        const int64_t a = s * SEG;
        const int n = (int)(a + SEG < len ? SEG : len - a);
        __syncwarp();
        for (int i = l; i < SEG; i += 32) {
            const int64_t t = t1 - d.pad + a + i;
            mine[i] = (i < n && t >= 0 && t < d.N) ? X[t * d.M + m] : 0.f;
        }
        __syncwarp();
        for (int i = 0; i < n; i += 4) {  // zeros beyond n add nothing
            const float4 x = *reinterpret_cast<const float4*>(mine + i);
            const double v[4] = {(double)x.x, (double)x.y, (double)x.z, (double)x.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                sum = __dadd_rn(sum, v[j]);
                sumsqr = __dadd_rn(sumsqr, __dmul_rn(v[j], v[j]));
            }
        }
    };
    // sumsqr plus i0 or i1 units, when it stays in the binade E
    auto move_sumsqr = [&](int E, int64_t i0, int64_t i1) -> bool {
        if (i0 < 0 || i1 < 0 || binade_of(sumsqr) != E) return false;
        const long long b = __double_as_longlong(sumsqr), moved = b + ((b & 1) ? i1 : i0);
        if ((moved >> 52) != (b >> 52)) return false;
        sumsqr = __longlong_as_double(moved);
        return true;
    };

    for (int64_t s0 = 0; s0 < nseg; s0 += 32) {
        const int64_t s = s0 + l, at = k * d.nseg + s;
        const bool have = s < nseg;
        const double x = have ? seg_x[at] : 0.0;
        const double ab = have ? (double)seg_abs[at] : 0.0;
        const int E = have ? seg_e[at] : kNoBinade;
        const uint32_t least = have ? seg_min[at] : 0u;
        const int q = float_grid(least);
        // a segment of zeros adds nothing to either sum, whatever they are
        const bool adds = least != 0u;
        const unsigned adding = __ballot_sync(0xffffffffu, adds);
        if (!adding) continue;
        const int64_t i0 = adds ? seg_inc0[at] : 0, i1 = adds ? seg_inc1[at] : 0;
        // the 32 segments at once
        double xs = x, as = ab;
        int qs = q;
        int64_t c0 = i0, c1 = i1;
        const int E0 = __shfl_sync(0xffffffffu, E, __ffs(adding) - 1);
        const bool one_binade = __all_sync(0xffffffffu, !adds || (E == E0 && i0 >= 0 && i1 >= 0));
        for (int o = 1; o < 32; o <<= 1) {
            xs += __shfl_xor_sync(0xffffffffu, xs, o);
            as += __shfl_xor_sync(0xffffffffu, as, o);
            qs = min(qs, __shfl_xor_sync(0xffffffffu, qs, o));
            const int64_t n0 = __shfl_down_sync(0xffffffffu, c0, o), n1 = __shfl_down_sync(0xffffffffu, c1, o);
            if (l + o < 32) {
                c0 += (c0 & 1) ? n1 : n0;
                c1 += (c1 & 1) ? n0 : n1;
            }
        }
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        c1 = __shfl_sync(0xffffffffu, c1, 0);
        const double sum_before = sum, sq_before = sumsqr;
        const bool sum_ok = sums_exact((fabs(sum) + as) * (1.0 + 1e-12), min(qs, lowest_bit(sum)));
        if (sum_ok && one_binade && move_sumsqr(E0, c0, c1)) {
            sum += xs;
            continue;
        }
        // one after another
        sum = sum_before;
        sumsqr = sq_before;
        for (int i = 0; i < 32; i++) {
            if (!((adding >> i) & 1)) continue;
            const double xi = __shfl_sync(0xffffffffu, x, i), ai = __shfl_sync(0xffffffffu, ab, i);
            const int qi = __shfl_sync(0xffffffffu, q, i), Ei = __shfl_sync(0xffffffffu, E, i);
            const int64_t j0 = __shfl_sync(0xffffffffu, i0, i), j1 = __shfl_sync(0xffffffffu, i1, i);
            if (sums_exact((fabs(sum) + ai) * (1.0 + 1e-12), min(qi, lowest_bit(sum))) && move_sumsqr(Ei, j0, j1))
                sum += xi;
            else
                one_by_one(s0 + i);
        }
    }
    if (l == 0) stats[c * d.M + m] = stats_of(sum, sumsqr, len, detect_threshold);
}

__device__ __forceinline__ double deviation(float x, double mean, int sign) {
    double val = (double)x - mean;
    if (sign < 0)
        val = -val;
    else if (sign == 0)
        val = fabs(val);
    return val;
}

// Candidates of a segment: counted (WRITE == false) or written in time order from
// base[slot] (their index n inside the padded chunk, their deviation and their
// (channel, chunk)).
template <bool WRITE>
__global__ void __launch_bounds__(256) detect_candidates(const float* __restrict__ X, Dims d,
                                                         const ChunkStats* __restrict__ stats, int sign,
                                                         int64_t* __restrict__ counts,
                                                         const int64_t* __restrict__ base,
                                                         int64_t* __restrict__ cand_n, double* __restrict__ cand_v,
                                                         int32_t* __restrict__ cand_k) {
    const Work w = segment_work(d);
    if (!w.any) return;
    const ChunkStats st = stats[w.c * d.M + w.m];
    int64_t k = 0;
    if (WRITE) {
        k = base[w.slot];
        if (k == base[w.slot + 1]) return;
    }
    for_samples(X, d, w.m, w.c, w.a, w.e, [&](int64_t n, float x) {
        const double val = deviation(x, st.mean, sign);
        if (val > st.threshold2) {
            if (WRITE) {
                cand_n[k] = n;
                cand_v[k] = val;
                cand_k[k] = (int32_t)(w.m * d.nchunks + w.c);
            }
            k++;
        }
    });
    if (!WRITE) counts[w.slot] = k;
}

// The greedy rule of detect_events (detect_events.cpp:87-125) over the candidates
// of one (channel, chunk) in time order.  At a candidate more than `interval`
// after the one before it, the rule forgets what came before: the thread of such a
// candidate (or of a chunk's first) applies it up to the next one.  use[i] = kept
// and inside [pad, pad + size).
__global__ void __launch_bounds__(128) detect_greedy(Dims d, int64_t ncand, double interval,
                                                     const int64_t* __restrict__ tc, const double* __restrict__ vc,
                                                     const int32_t* __restrict__ kc, uint8_t* __restrict__ use) {
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (first >= ncand) return;
    const int32_t k = kc[first];
    auto starts = [&](int64_t i) {
        return i == 0 || kc[i - 1] != k || (double)tc[i - 1] < (double)tc[i] - interval;
    };
    if (!starts(first)) return;
    int64_t best = first, end = first + 1;
    use[first] = 1;
    for (int64_t i = end; i < ncand && kc[i] == k && !starts(i); i++) {
        end = i + 1;
        if ((double)tc[best] < (double)tc[i] - interval) {
            // candidate i - 1 lies within the interval (no start at i): the
            // strongest of those that do
            best = i - 1;
            for (int64_t j = best; j - 1 >= first && (double)tc[j - 1] >= (double)tc[i] - interval; j--)
                if (vc[j - 1] > vc[best]) best = j - 1;
        }
        if (vc[i] > vc[best]) {
            use[i] = 1;
            use[best] = 0;
            best = i;
        } else {
            use[i] = 0;
        }
    }
    const int64_t size = chunk_size_at(k % d.nchunks, d.chunk, d.N);
    for (int64_t i = first; i < end; i++) {
        const int64_t t = tc[i] - d.pad;
        if (t < 0 || t >= size) use[i] = 0;
    }
}

__global__ void detect_write(Dims d, int64_t ncand, const int64_t* __restrict__ tc, const int32_t* __restrict__ kc,
                             const uint8_t* __restrict__ use, const int64_t* __restrict__ at,
                             int64_t* __restrict__ times) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ncand && use[i]) times[at[i]] = tc[i] - d.pad + (int64_t)(kc[i] % d.nchunks) * d.chunk;
}

// counts[m] = events of channel m, from the positions at its first and last candidate
__global__ void detect_channel_counts(Dims d, const int64_t* __restrict__ base, const int64_t* __restrict__ at,
                                      int64_t* __restrict__ counts) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m < d.M) counts[m] = at[base[(m + 1) * d.nchunks * d.nseg]] - at[base[m * d.nchunks * d.nseg]];
}

// ------------------------------------------------------------ prefix sums

constexpr int kScanItems = 4096;  // per block of 256

__device__ __forceinline__ int64_t block_sum_256(int64_t v, int64_t* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    int64_t t = 0;
    for (int i = 0; i < 8; i++) t += red[i];
    __syncthreads();
    return t;
}

// exclusive prefix of the block's 256 values; *total = their sum
__device__ __forceinline__ int64_t block_prefix_256(int64_t v, int64_t* red, int64_t* total) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (l >= o) incl += up;
    }
    if (l == 31) red[w] = incl;
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int i = 0; i < 8; i++) {
        if (i < w) before += red[i];
        all += red[i];
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

template <class T>
__global__ void __launch_bounds__(256) scan_block_sums(const T* __restrict__ in, int64_t n, int64_t* __restrict__ sums) {
    __shared__ int64_t red[8];
    const int64_t b = (int64_t)blockIdx.x * kScanItems;
    int64_t v = 0;
    for (int i = threadIdx.x; i < kScanItems; i += 256)
        if (b + i < n) v += (int64_t)in[b + i];
    v = block_sum_256(v, red);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

__global__ void __launch_bounds__(256) scan_of_sums(int64_t* __restrict__ sums, int64_t n) {
    __shared__ int64_t red[8];
    int64_t before = 0;
    for (int64_t b = 0; b < n; b += 256) {
        const int64_t i = b + threadIdx.x;
        int64_t total;
        const int64_t p = block_prefix_256(i < n ? sums[i] : 0, red, &total);
        if (i < n) sums[i] = before + p;
        before += total;
    }
}

// out[i] = sum of in[0 .. i) for i <= n
template <class T>
__global__ void __launch_bounds__(256) scan_write(const T* __restrict__ in, int64_t n, const int64_t* __restrict__ sums,
                                                  int64_t* __restrict__ out) {
    __shared__ int64_t red[8];
    int64_t before = sums ? sums[blockIdx.x] : 0;
    for (int64_t b = (int64_t)blockIdx.x * kScanItems, e = b + kScanItems; b < e && b < n; b += 256) {
        const int64_t i = b + threadIdx.x;
        int64_t total;
        const int64_t v = i < n ? (int64_t)in[i] : 0;
        const int64_t p = block_prefix_256(v, red, &total);
        if (i < n) out[i] = before + p;
        if (i == n - 1) out[n] = before + p + v;
        before += total;
    }
}

int64_t scan_blocks(int64_t n) { return ceil_div(n, kScanItems); }

// n >= 1; sums: scan_blocks(n) values
template <class T>
void prefix_sums(const T* in, int64_t n, int64_t* out, int64_t* sums, cudaStream_t stream) {
    const int64_t blocks = scan_blocks(n);
    if (blocks > 1) {
        scan_block_sums<<<(unsigned)blocks, 256, 0, stream>>>(in, n, sums);
        MS3_LAUNCH_CHECK();
        scan_of_sums<<<1, 256, 0, stream>>>(sums, blocks);
        MS3_LAUNCH_CHECK();
    }
    scan_write<<<(unsigned)blocks, 256, 0, stream>>>(in, n, blocks > 1 ? sums : nullptr, out);
    MS3_LAUNCH_CHECK();
}

// Arrays of one allocation: short recordings waited for the allocations and frees of one
// each (1 channel x 100 timepoints: 292 us a call, with one allocation 259).
class Arrays {
public:
    template <class T>
    void add(T** p, int64_t n) {
        parts_.push_back({reinterpret_cast<void**>(p), bytes_});
        bytes_ += (sizeof(T) * (size_t)n + 255) / 256 * 256;
    }
    void alloc(cudaStream_t stream) {
        buf_.alloc(bytes_, stream);
        for (const auto& p : parts_) *p.first = buf_.as<char>() + p.second;
    }

private:
    std::vector<std::pair<void**, size_t>> parts_;
    size_t bytes_ = 0;
    DevBuf buf_;
};

// Whether a thread per (channel, chunk) forms the statistics.  From 4096 pairs on they
// hide one another's additions, and the segments' passes over X and the segments that go
// sample by sample cost more.  Whole calls, us, serial and by segments:
//   pairs (chunk)                 rounded to 1e-4   unrounded   values over 40 octaves
//    3840 (64 ch,  30 k)           1277    984      1263   1415      2459   3294
//    5376 (384 ch, 30 k)           1545   1444      1554   1798      3163   4667
//    6144 (1536 ch, 163 k)         7065   5810      7063   8066     20018  27686
//    7680 (128 ch, 30 k)           1475   1608      1467   2030      3746   5735
//   30720 (1536 ch, 30 k)          3690   6476      3670   6915     16579  26455
// and 1536 (384 ch, 651 k): 19639 and 4236, 19643 and 11706, 29235 and 26311.
bool serial_stats(int64_t pairs) { return pairs >= 4096; }

// A thread takes a segment, 16 loads at a time: with few threads a pass over segments of
// 512 waits for 32 such batches one after another.  Short chunks (at most eight times 32
// segments of 64, which detect_stats puts together one after another) with few of them
// take 64 (1 channel x 100 timepoints: 259 and 141 us a call; 16 x 8000: 287 and 184).
int segment_length(int64_t len, int64_t pairs) {
    return len <= 8 * 32 * kShortSeg && pairs * ceil_div(len, kSeg) < 16384 ? kShortSeg : kSeg;
}

}  // namespace

int64_t detect_chunk_size(int64_t M, int64_t N, int64_t num_simultaneous) {
    // get_time_chunk_infos (p_mountainsort3.cpp:507-517) with min_num_chunks 1
    int64_t chunk_size = (int64_t)1e9 / (M * num_simultaneous * 4);
    if (chunk_size > N) chunk_size = N;
    if (chunk_size < 20000) chunk_size = 20000;
    return chunk_size;
}

void detect_events_device(const float* X, int64_t M, int64_t N, double detect_threshold, double detect_interval,
                          int sign, int64_t chunk, int64_t pad, std::vector<int64_t>& counts,
                          std::vector<int64_t>& times, cudaStream_t stream) {
    counts.assign((size_t)std::max<int64_t>(M, 0), 0);
    times.clear();
    if (M <= 0 || N <= 0) return;
    const int64_t nchunks = ceil_div(N, chunk);
    if (nchunks > 65535) throw_unsupported("too many time chunks");
    const int64_t len = std::min(chunk, N) + 2 * pad;
    const int seg = segment_length(len, M * nchunks);
    Dims d{M, N, chunk, pad, nchunks, ceil_div(len, seg), seg};
    const int64_t MC = M * nchunks, slots = MC * d.nseg;
    if (MC > 0x7fffffff) throw_unsupported("too many (channel, chunk) pairs");
    const int64_t work_blocks = ceil_div(M * d.nseg, 256);
    if (work_blocks > 0x7fffffff) throw_unsupported("too many segments");
    const dim3 gs((unsigned)work_blocks, (unsigned)nchunks);

    ChunkStats* stats;
    int64_t *base, *cnt, *sums;  // candidates, channel-major, then chunk, then segment (time order)
    Arrays first;
    first.add(&stats, MC);
    first.add(&base, slots + 1);
    first.add(&cnt, slots);
    first.add(&sums, scan_blocks(slots));
    first.alloc(stream);
    if (serial_stats(MC)) {
        detect_stats_serial<<<(unsigned)ceil_div(MC, 32), 32, 0, stream>>>(X, d, detect_threshold, stats);
        MS3_LAUNCH_CHECK();
    } else {
        double *sx, *sq;
        float* sa;
        uint32_t* sm;
        int* se;
        int64_t *i0, *i1;
        Arrays segs;
        segs.add(&sx, slots);
        segs.add(&sa, slots);
        segs.add(&sq, slots);
        segs.add(&sm, slots);
        segs.add(&se, slots);
        segs.add(&i0, slots);
        segs.add(&i1, slots);
        segs.alloc(stream);
        detect_segments<<<gs, 256, 0, stream>>>(X, d, sx, sa, sq, sm);
        MS3_LAUNCH_CHECK();
        detect_binades<<<(unsigned)ceil_div(MC, 4), 128, 0, stream>>>(sq, MC, d.nseg, se);
        MS3_LAUNCH_CHECK();
        detect_increments<<<gs, 256, 0, stream>>>(X, d, sq, se, i0, i1);
        MS3_LAUNCH_CHECK();
        const auto stats_kernel = seg == kSeg ? detect_stats<kSeg> : detect_stats<kShortSeg>;
        stats_kernel<<<(unsigned)ceil_div(MC, kStatWarps), 32 * kStatWarps, 0, stream>>>(X, d, detect_threshold, sx, sa, sm,
                                                                                       se, i0, i1, stats);
        MS3_LAUNCH_CHECK();
    }
    detect_candidates<false><<<gs, 256, 0, stream>>>(X, d, stats, sign, cnt, nullptr, nullptr, nullptr, nullptr);
    MS3_LAUNCH_CHECK();
    prefix_sums(cnt, slots, base, sums, stream);
    int64_t ncand = 0;
    MS3_CUDA(cudaMemcpyAsync(&ncand, base + slots, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    MS3_CUDA(cudaStreamSynchronize(stream));
    if (ncand > ((int64_t)1 << 31)) throw_unsupported("too many threshold crossings (lower the sensitivity)");
    if (ncand == 0) return;
    int64_t *cn, *at, *dcounts, *dtimes, *cand_sums;
    double* cv;
    int32_t* ck;
    uint8_t* use;
    Arrays cand;
    cand.add(&cn, ncand);
    cand.add(&cv, ncand);
    cand.add(&ck, ncand);
    cand.add(&use, ncand);
    cand.add(&at, ncand + 1);
    cand.add(&dcounts, M);
    cand.add(&dtimes, ncand);
    cand.add(&cand_sums, scan_blocks(ncand));
    cand.alloc(stream);
    detect_candidates<true><<<gs, 256, 0, stream>>>(X, d, stats, sign, nullptr, base, cn, cv, ck);
    MS3_LAUNCH_CHECK();
    const unsigned gg = (unsigned)ceil_div(ncand, 128);
    detect_greedy<<<gg, 128, 0, stream>>>(d, ncand, detect_interval, cn, cv, ck, use);
    MS3_LAUNCH_CHECK();
    prefix_sums(use, ncand, at, cand_sums, stream);
    detect_channel_counts<<<(unsigned)ceil_div(M, 128), 128, 0, stream>>>(d, base, at, dcounts);
    MS3_LAUNCH_CHECK();
    detect_write<<<gg, 128, 0, stream>>>(d, ncand, cn, ck, use, at, dtimes);
    MS3_LAUNCH_CHECK();
    MS3_CUDA(cudaMemcpyAsync(counts.data(), dcounts, sizeof(int64_t) * counts.size(), cudaMemcpyDeviceToHost, stream));
    MS3_CUDA(cudaStreamSynchronize(stream));
    int64_t total = 0;
    for (int64_t n : counts) total += n;
    times.resize((size_t)total);
    if (total == 0) return;
    MS3_CUDA(cudaMemcpyAsync(times.data(), dtimes, sizeof(int64_t) * (size_t)total, cudaMemcpyDeviceToHost, stream));
    MS3_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace ms3gpu
