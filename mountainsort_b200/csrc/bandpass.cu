// ms3.bandpass_filter on the GPU.
//
// Reference: packages/ms3/p_bandpass_filter.cpp:115-229.  The recording is
// cut into chunks of `chunk` timepoints (chunk from the reference's formula,
// :147-155); chunk c is filtered inside the window
//     [c*chunk - 60000, c*chunk + chunk + 60000)           (L = chunk + 120000)
// zero-padded outside [0, N) (mda/diskreadmda32.cpp:615-661), by an L-point
// DFT, multiplication with kernel[k]/L (define_kernel, :421-447, DC bin exactly
// 0 when freq_min != 0) and the inverse DFT; the middle `chunk` samples are
// kept (:198).  Keeping this geometry exactly is what makes the output match
// the reference: the DC kill subtracts H(0)*mean(window) per window and the
// circular wrap of the long filter tail depends on L.
//
// GPU formulation ("four-step" FFT, L = L1 * L2, window index n = L2*n1 + n2,
// frequency k = k1 + L1*k2):
//   F1  bp_cols_forward : for each n2, the L1-point DFT over n1 of the window
//                         column -> A[k1][n2]
//   F2  bp_rows_filter  : for each k1, twiddle w_L^{n2 k1}, L2-point DFT over
//                         n2 -> k2, multiply by kernel[k1 + L1 k2]/L, inverse
//                         L2-point DFT, twiddle w_L^{-n2 k1}   (in place)
//   F3  bp_cols_inverse : for each n2, the inverse L1-point DFT over k1 -> n1,
//                         keep the samples inside [60000, 60000 + chunk),
//                         subsample / quantize, store.
// Two real channels (2p, 2p+1) travel as one complex signal x_2p + i x_2p+1:
// the band kernel is real and even (kernel[k] == kernel[L-k] for even L), so
// the real and imaginary parts of the inverse transform are the two filtered
// channels.  A unit of work is (window, group of G channel pairs); its
// spectrum lives in a scratch slab of L*G complex values between F1 and F3.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "bandpass.h"
#include "common.cuh"
#include "fft_block.cuh"
#include "fft_reg.cuh"
#include "host_dft.h"
#include "ms3gpu.h"
#include "tc_sm100.cuh"

namespace ms3gpu {

namespace {

constexpr int64_t kOverlap = 60000;
constexpr int kThreads = 256;
constexpr size_t kSmemBudget = 200 * 1024;

struct Geom {
    int64_t M, N;        // input shape
    int64_t P;           // complex signals: channel pairs (or channels when unpaired)
    int paired;          // 1: two channels per complex signal
    int m_even;          // M even (pairs load as aligned float2)
    int log2G;           // signals per unit = 1 << log2G
    int ngroups;
    int64_t c_begin;     // first window of this call
    int64_t nwin;        // windows in this call
    int64_t L, L1, L2;   // FFT length and its factors
    int64_t Lw;          // window length chunk + 120000 (< L when the window is zero-padded to a longer FFT)
    int64_t chunk;
    int sub;
    int64_t N2;          // output timepoints
    int out_i16;
    double qscale;       // 1 / quantization_unit
    int half_lines;      // int16 input or output: neighbouring groups share 128-byte lines
    int in_i16;          // raw is int16 (converted to float on load, like the reference's reader)
};

// ---------------------------------------------------------------- kernels

// v * kernel[k] / L for the kernel value held as hi + lo floats: the product
// rounds once to float like the reference's float *= double
// (p_bandpass_filter.cpp:87-95) instead of after a rounding of the kernel
// value itself, which would be the same relative error in every window and
// channel at that frequency.
__device__ __forceinline__ float2 kern_mul(float2 v, float2 k) {
    return make_float2(__fmaf_rn(v.x, k.x, __fmul_rn(v.x, k.y)), __fmaf_rn(v.y, k.x, __fmul_rn(v.y, k.y)));
}

__device__ __forceinline__ float2 load_signal(const void* __restrict__ raw, const Geom& g, int64_t t, int64_t s) {
    if (t < 0 || t >= g.N || s >= g.P) return make_float2(0.f, 0.f);
    const int64_t m0 = g.paired ? 2 * s : s;
    if (g.in_i16) {
        // int16 -> float as mdaReadData converts (mda/mdaio.cpp:205-230)
        const int16_t* row = static_cast<const int16_t*>(raw) + t * g.M;
        if (!g.paired) return make_float2((float)row[s], 0.f);
        if (g.m_even) {
            const short2 v = *reinterpret_cast<const short2*>(row + m0);
            return make_float2((float)v.x, (float)v.y);
        }
        return make_float2((float)row[m0], (m0 + 1 < g.M) ? (float)row[m0 + 1] : 0.f);
    }
    const float* row = static_cast<const float*>(raw) + t * g.M;
    if (!g.paired) return make_float2(row[s], 0.f);
    if (g.m_even) return *reinterpret_cast<const float2*>(row + m0);
    return make_float2(row[m0], (m0 + 1 < g.M) ? row[m0 + 1] : 0.f);
}

// Units are ordered group-major: consecutive units are consecutive windows of
// the same channel group, so the half of a window shared with the previous
// window is read again while it is still in L2.  For int16 input or output a group's
// row is half a 128-byte line: two neighbouring groups alternate, so that the second
// finds its half of each line in L2 (384 int16 channels x 600k: F1 901 us, with whole lines fetched 845).
// Not for subsampled int16 stores (64 channels, every second timepoint: 2201 us a call
// as it was, 2227 alternating), and for int16 input alone only where a group's piece of a
// row is half a line, M a multiple of 32 (700 channels: 3420 and 3475).
struct UnitIdx {
    int64_t c;
    int grp;
};
__device__ __forceinline__ UnitIdx unit_index(const Geom& g, int64_t unit64) {
    // 32 bits (the divisions are in every block): windows x groups of a call that fits in memory
    const uint32_t unit = (uint32_t)unit64, nwin = (uint32_t)g.nwin;
    UnitIdx u;
    const uint32_t both = g.half_lines ? (uint32_t)(g.ngroups / 2) * 2 * nwin : 0;  // units of group pairs
    uint32_t c;
    if (unit < both) {
        const uint32_t pair = unit / (2 * nwin), r = unit - pair * 2 * nwin;
        u.grp = (int)(pair * 2 + (r & 1));
        c = r >> 1;
    } else {
        u.grp = (int)(unit / nwin);  // `both` is a multiple of nwin
        c = unit % nwin;
    }
    u.c = g.c_begin + c;
    return u;
}

__device__ __forceinline__ void load_plan(SubFft& dst, const SubFft& src) {
    int* d = reinterpret_cast<int*>(&dst);
    const int* s = reinterpret_cast<const int*>(&src);
    for (int i = threadIdx.x; i < (int)(sizeof(SubFft) / sizeof(int)); i += blockDim.x) d[i] = s[i];
}

// F1: forward L1-point transforms of the window columns.
__global__ void __launch_bounds__(kThreads) bp_cols_forward(const void* __restrict__ raw,
                                                            float2* __restrict__ scratch, Geom g,
                                                            SubFft P1, const float2* __restrict__ tw1,
                                                            int64_t unit0) {
    extern __shared__ float4 smem_f4[];
    float2* smem = reinterpret_cast<float2*>(smem_f4);
    __shared__ SubFft plan;
    const int G = 1 << g.log2G;
    const int n1len = (int)g.L1;
    float2* bufA = smem;
    float2* bufB = bufA + (size_t)n1len * G;
    float2* twS = bufB + (size_t)n1len * G;
    load_plan(plan, P1);
    for (int i = threadIdx.x; i < P1.twlen; i += blockDim.x) twS[i] = tw1[i];

    const int n2 = blockIdx.x;
    const UnitIdx ui = unit_index(g, unit0 + blockIdx.y);
    const int64_t c = ui.c;
    const int grp = ui.grp;
    const int64_t t0 = c * g.chunk - kOverlap + n2;
    for (int idx = threadIdx.x; idx < n1len * G; idx += blockDim.x) {
        const int n1 = idx >> g.log2G;
        const int gi = idx & (G - 1);
        const int64_t n = (int64_t)n1 * g.L2 + n2;  // window index
        bufA[idx] = n < g.Lw ? load_signal(raw, g, t0 + (int64_t)n1 * g.L2, (int64_t)grp * G + gi)
                             : make_float2(0.f, 0.f);
    }
    __syncthreads();
    float2* res = fft_smem<false>(bufA, bufB, twS, plan, g.log2G);
    float2* slab = scratch + (size_t)blockIdx.y * (size_t)(g.L * G);
    for (int idx = threadIdx.x; idx < n1len * G; idx += blockDim.x) {
        const int k1 = idx >> g.log2G;
        const int gi = idx & (G - 1);
        slab[(((size_t)k1 * g.L2 + n2) << g.log2G) + gi] = res[idx];
    }
}

// F2: per k1 row: twiddle, L2-point forward DFT, band kernel, inverse DFT,
// inverse twiddle.
__global__ void __launch_bounds__(kThreads) bp_rows_filter(float2* __restrict__ scratch, Geom g, SubFft P2,
                                                           const float2* __restrict__ tw2,
                                                           const float2* __restrict__ twL,
                                                           const float2* __restrict__ kern) {
    extern __shared__ float4 smem_f4[];
    float2* smem = reinterpret_cast<float2*>(smem_f4);
    __shared__ SubFft plan;
    const int G = 1 << g.log2G;
    const int n2len = (int)g.L2;
    float2* bufA = smem;
    float2* bufB = bufA + (size_t)n2len * G;
    float2* twS = bufB + (size_t)n2len * G;
    load_plan(plan, P2);
    for (int i = threadIdx.x; i < P2.twlen; i += blockDim.x) twS[i] = tw2[i];

    const int k1 = blockIdx.x;
    float2* row = scratch + (size_t)blockIdx.y * (size_t)(g.L * G) + (((size_t)k1 * g.L2) << g.log2G);
    const float2* twrow = twL + (size_t)k1 * g.L2;
    const float2* krow = kern + (size_t)k1 * g.L2;
    for (int idx = threadIdx.x; idx < n2len * G; idx += blockDim.x) {
        const int n2 = idx >> g.log2G;
        bufA[idx] = cmul(row[idx], twrow[n2]);
    }
    __syncthreads();
    float2* res = fft_smem<false>(bufA, bufB, twS, plan, g.log2G);
    float2* other = (res == bufA) ? bufB : bufA;
    for (int idx = threadIdx.x; idx < n2len * G; idx += blockDim.x) {
        res[idx] = kern_mul(res[idx], krow[idx >> g.log2G]);
    }
    __syncthreads();
    float2* res2 = fft_smem<true>(res, other, twS, plan, g.log2G);
    for (int idx = threadIdx.x; idx < n2len * G; idx += blockDim.x) {
        const int n2 = idx >> g.log2G;
        float2 w = twrow[n2];
        w.y = -w.y;
        row[idx] = cmul(res2[idx], w);
    }
}

// F3: inverse L1-point transforms of the columns, trim, subsample, quantize,
// store.
__global__ void __launch_bounds__(kThreads) bp_cols_inverse(const float2* __restrict__ scratch,
                                                            void* __restrict__ out, Geom g, SubFft P1,
                                                            const float2* __restrict__ tw1,
                                                            int64_t unit0) {
    extern __shared__ float4 smem_f4[];
    float2* smem = reinterpret_cast<float2*>(smem_f4);
    __shared__ SubFft plan;
    const int G = 1 << g.log2G;
    const int n1len = (int)g.L1;
    float2* bufA = smem;
    float2* bufB = bufA + (size_t)n1len * G;
    float2* twS = bufB + (size_t)n1len * G;
    load_plan(plan, P1);
    for (int i = threadIdx.x; i < P1.twlen; i += blockDim.x) twS[i] = tw1[i];

    const int n2 = blockIdx.x;
    const UnitIdx ui = unit_index(g, unit0 + blockIdx.y);
    const int64_t c = ui.c;
    const int grp = ui.grp;
    const float2* slab = scratch + (size_t)blockIdx.y * (size_t)(g.L * G);
    for (int idx = threadIdx.x; idx < n1len * G; idx += blockDim.x) {
        const int k1 = idx >> g.log2G;
        const int gi = idx & (G - 1);
        bufA[idx] = slab[(((size_t)k1 * g.L2 + n2) << g.log2G) + gi];
    }
    __syncthreads();
    float2* res = fft_smem<true>(bufA, bufB, twS, plan, g.log2G);
    const int64_t nsub = g.chunk / g.sub;
    const int64_t ot0 = (c * g.chunk) / g.sub;
    for (int idx = threadIdx.x; idx < n1len * G; idx += blockDim.x) {
        const int n1 = idx >> g.log2G;
        const int gi = idx & (G - 1);
        const int64_t s = (int64_t)grp * G + gi;
        if (s >= g.P) continue;
        const int64_t j = (int64_t)n1 * g.L2 + n2 - kOverlap;
        if (j < 0 || j >= g.chunk) continue;
        if (j % g.sub) continue;
        const int64_t jj = j / g.sub;
        if (jj >= nsub) continue;
        const int64_t ot = ot0 + jj;
        if (ot >= g.N2) continue;
        const float2 v = res[idx];
        const int64_t m0 = g.paired ? 2 * s : s;
        const bool has2 = g.paired && (m0 + 1 < g.M);
        const size_t o = (size_t)(ot * g.M + m0);
        if (g.out_i16) {
            int16_t* o16 = static_cast<int16_t*>(out);
            o16[o] = x86_float_to_int16((float)((double)v.x * g.qscale));
            if (has2) o16[o + 1] = x86_float_to_int16((float)((double)v.y * g.qscale));
        } else {
            float* of = static_cast<float*>(out);
            if (has2 && g.m_even) {
                *reinterpret_cast<float2*>(of + o) = v;
            } else {
                of[o] = v.x;
                if (has2) of[o + 1] = v.y;
            }
        }
    }
}


// Stores one filtered complex sample (two channels) at window index n of a
// window whose first kept sample lands at output timepoint ot_base =
// (c * chunk) / sub, applying the trim to [60000, 60000 + chunk), the
// subsampling and the int16 quantization of the reference
// (p_bandpass_filter.cpp:196-212).  chunk < 2^31 (at most 2^30 / 24), so the
// window arithmetic is 32-bit and needs no division when sub == 1.
__device__ __forceinline__ void store_filtered(void* __restrict__ out, const Geom& g, int64_t ot_base, int64_t s,
                                               int n, float2 v) {
    if (s >= g.P) return;
    const int j = n - (int)kOverlap;
    if ((unsigned)j >= (unsigned)g.chunk) return;
    int64_t ot = ot_base + j;
    if (g.sub != 1) {
        const int sub = g.sub;
        if (j % sub) return;
        const int jj = j / sub;
        if (jj >= (int)g.chunk / sub) return;
        ot = ot_base + jj;
    }
    if (ot >= g.N2) return;
    const int64_t m0 = g.paired ? 2 * s : s;
    const bool has2 = g.paired && (m0 + 1 < g.M);
    const size_t o = (size_t)(ot * g.M + m0);
    if (!MS3_IN_BOUNDS((int64_t)o + (has2 ? 1 : 0), g.N2 * g.M, 101)) return;
    if (g.out_i16) {
        int16_t* o16 = static_cast<int16_t*>(out);
        o16[o] = x86_float_to_int16((float)((double)v.x * g.qscale));
        if (has2) o16[o + 1] = x86_float_to_int16((float)((double)v.y * g.qscale));
    } else {
        float* of = static_cast<float*>(out);
        if (has2 && g.m_even) {
            *reinterpret_cast<float2*>(of + o) = v;
        } else {
            of[o] = v.x;
            if (has2) of[o + 1] = v.y;
        }
    }
}

// ------------------------------------------------- register-pass kernels
// Each sub-transform of length n = RA * RB runs as two Stockham passes whose
// butterflies live entirely in registers (RegDft), with one shared-memory
// exchange between them:
//   pass 1 (radix RA, p = 1):  item i < RB reads x[i + q RB], writes y[i RA + q]
//   pass 2 (radix RB, p = RA): item i < RA reads y[i + q RA] * w_n^{q i},
//                              writes z[i + q RA]   (natural order)
// Global loads feed pass 1 directly and pass 2 stores directly.

// A read-only load that brings its whole 128-byte line into L2.
__device__ __forceinline__ uint32_t load_line(const uint32_t* p) {
    uint32_t v;
    asm("ld.global.nc.L2::128B.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Two int16 as floats, the same values as the conversion: with its sign bit flipped, a
// value's 16 bits under the exponent of 2^23 are the float 2^23 + 32768 + value.  The
// conversion instructions run at a quarter of the rate of these (byte permutes, adds):
// 384 int16 channels x 600k, F1 912 us with them, 901 without (float input 670).
__device__ __forceinline__ float2 floats_of(uint32_t pair) {
    const uint32_t u = pair ^ 0x80008000u;
    const float lo = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7410));
    const float hi = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7432));
    return make_float2(__fadd_rn(lo, -8421376.0f), __fadd_rn(hi, -8421376.0f));
}

// F1, forward columns of length L1 = RA * RB.
// LG >= 0 and KL2 > 0 fix log2 G and L2 at compile time (the canonical
// window with 16 signals per unit), so the index arithmetic folds into
// constant offsets; LG = -1 reads them from g.
// FORM says what the host found, so that the other forms are not in the kernel: float
// pairs, int16 pairs, an odd channel count; 0 takes any.  (One kernel with all of them
// and a predicate on every load: 64 channels x 3.1 M 2062 us a call, 700 int16 channels
// kept every third timepoint 3546; before there were other forms 2018 and 3447.)
enum { kAnyForm = 0, kFloatPairs = 1, kInt16Pairs = 2, kOddCount = 3 };
template <int RA, int RB, int LG, int KL2, int FORM>
__global__ void __launch_bounds__(256, 3) bpr_cols_forward(const void* __restrict__ raw, float2* __restrict__ scratch,
                                                        Geom g, const float2* __restrict__ roots, int64_t unit0) {
    constexpr int n = RA * RB;
    const int lg = LG >= 0 ? LG : g.log2G;
    const int64_t L2 = KL2 > 0 ? KL2 : g.L2;
    extern __shared__ float4 smem_f4[];
    float2* buf = reinterpret_cast<float2*>(smem_f4);
    float2* rt = buf + ((size_t)n << lg);
    for (int i = threadIdx.x; i < n; i += blockDim.x) rt[i] = roots[i];
    const int G = 1 << lg;
    const int n2 = blockIdx.x;
    const UnitIdx ui = unit_index(g, unit0 + blockIdx.y);
    const int64_t t0 = ui.c * g.chunk - kOverlap + n2;
    const int64_t s0 = (int64_t)ui.grp * G;
    // a window inside the recording: strided loads without index checks.  An odd channel
    // count loads a pair's two channels one by one, and the last group's signals beyond P
    // are left out by a predicate (63 int16 channels: 340 us a launch of 14 units by the
    // checked loads, now 214).
    const bool whole = s0 + G <= g.P;
    const bool inside = g.paired && t0 >= 0 && t0 + (int64_t)(n - 1) * L2 < g.N;
    for (int it = threadIdx.x; it < (RB << lg); it += blockDim.x) {
        const int gi = it & (G - 1), i = it >> lg;
        float2 u[RA];
        if (inside) {
            const int64_t s = s0 + gi;
            const int64_t at = (t0 + (int64_t)i * L2) * g.M + 2 * s;  // the pair's first channel
            const int64_t step = (int64_t)RB * L2 * g.M;              // RB window rows
            const bool ok = s < g.P;
            if (FORM == kAnyForm ? g.m_even != 0 : FORM != kOddCount) {
                if (FORM == kAnyForm ? g.in_i16 != 0 : FORM == kInt16Pairs) {
                    const uint32_t* p = reinterpret_cast<const uint32_t*>(static_cast<const int16_t*>(raw) + at);
                    if (whole) {
#pragma unroll
                        for (int q = 0; q < RA; q++) u[q] = floats_of(load_line(p + q * (step / 2)));
                    } else {
#pragma unroll
                        for (int q = 0; q < RA; q++) u[q] = floats_of(ok ? load_line(p + q * (step / 2)) : 0u);
                    }
                } else {
                    const float2* p = reinterpret_cast<const float2*>(static_cast<const float*>(raw) + at);
                    if (whole) {
#pragma unroll
                        for (int q = 0; q < RA; q++) u[q] = __ldg(p + q * (step / 2));
                    } else {
#pragma unroll
                        for (int q = 0; q < RA; q++) u[q] = ok ? __ldg(p + q * (step / 2)) : make_float2(0.f, 0.f);
                    }
                }
            } else {
                const bool two = 2 * s + 1 < g.M;
                if (g.in_i16) {
                    const int16_t* p = static_cast<const int16_t*>(raw) + at;
#pragma unroll
                    for (int q = 0; q < RA; q++)
                        u[q] = floats_of((ok ? (uint32_t)(uint16_t)__ldg(p + q * step) : 0u) |
                                         (two ? (uint32_t)(uint16_t)__ldg(p + q * step + 1) << 16 : 0u));
                } else {
                    const float* p = static_cast<const float*>(raw) + at;
#pragma unroll
                    for (int q = 0; q < RA; q++)
                        u[q] = make_float2(ok ? __ldg(p + q * step) : 0.f, two ? __ldg(p + q * step + 1) : 0.f);
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < RA; q++) u[q] = load_signal(raw, g, t0 + (int64_t)(i + q * RB) * L2, s0 + gi);
        }
        RegDft<RA, false>::run(u);
#pragma unroll
        for (int q = 0; q < RA; q++) buf[((i * RA + q) << lg) + gi] = u[q];
    }
    __syncthreads();
    float2* slab = scratch + (size_t)blockIdx.y * (size_t)(g.L * G);
    for (int it = threadIdx.x; it < (RA << lg); it += blockDim.x) {
        const int gi = it & (G - 1), i = it >> lg;
        float2 u[RB];
#pragma unroll
        for (int q = 0; q < RB; q++) {
            const float2 v = buf[((i + q * RA) << lg) + gi];
            u[q] = (q == 0) ? v : cmul(v, rt[q * i]);
        }
        RegDft<RB, false>::run(u);
        float2* o = slab + (((size_t)i * L2 + n2) << lg) + gi;
        const size_t step = ((size_t)RA * L2) << lg;
        const int64_t e0 = (int64_t)((((size_t)i * L2 + n2) << lg) + gi);
#pragma unroll
        for (int q = 0; q < RB; q++)
            if (MS3_IN_BOUNDS(e0 + (int64_t)(q * step), g.L << lg, 103)) o[q * step] = u[q];
    }
}

// F2, one k1 row: twiddle, forward L2 = SA * SB, band kernel, inverse, twiddle.
// The forward pass 2 and the inverse pass 1 (radix SB, p = 1) share the same
// item -> thread mapping, so the spectrum never leaves registers between them.
// Launched with exactly SA * G threads (one middle-phase item per thread).
template <int SA, int SB>
__global__ void __launch_bounds__(320) bpr_rows_filter(float2* __restrict__ scratch, Geom g,
                                                       const float2* __restrict__ roots,
                                                       const float2* __restrict__ twL,
                                                       const float2* __restrict__ kern) {
    constexpr int n = SA * SB;
    extern __shared__ float4 smem_f4[];
    float2* buf = reinterpret_cast<float2*>(smem_f4);
    float2* rt = buf + ((size_t)n << g.log2G);
    for (int i = threadIdx.x; i < n; i += blockDim.x) rt[i] = roots[i];
    const int G = 1 << g.log2G;
    const int k1 = blockIdx.x;
    float2* row = scratch + (size_t)blockIdx.y * (size_t)(g.L * G) + (((size_t)k1 * g.L2) << g.log2G);
    const float2* twrow = twL + (size_t)k1 * g.L2;
    const float2* krow = kern + (size_t)k1 * g.L2;
    // forward pass 1 (radix SA over items i < SB)
    for (int it = threadIdx.x; it < (SB << g.log2G); it += blockDim.x) {
        const int gi = it & (G - 1), i = it >> g.log2G;
        float2 u[SA];
#pragma unroll
        for (int q = 0; q < SA; q++) {
            const int n2 = i + q * SB;
            u[q] = cmul(row[(n2 << g.log2G) + gi], __ldg(&twrow[n2]));
        }
        RegDft<SA, false>::run(u);
#pragma unroll
        for (int q = 0; q < SA; q++) buf[((i * SA + q) << g.log2G) + gi] = u[q];
    }
    __syncthreads();
    // forward pass 2 (radix SB, item i < SA), kernel, inverse pass 1 (radix SB)
    const int it = threadIdx.x;
    const bool active = it < (SA << g.log2G);
    const int gi = it & (G - 1), i = it >> g.log2G;
    float2 u[SB];
    if (active) {
#pragma unroll
        for (int q = 0; q < SB; q++) {
            const float2 v = buf[((i + q * SA) << g.log2G) + gi];
            u[q] = (q == 0) ? v : cmul(v, rt[q * i]);
        }
        RegDft<SB, false>::run(u);
#pragma unroll
        for (int q = 0; q < SB; q++) u[q] = kern_mul(u[q], __ldg(&krow[i + q * SA]));
        RegDft<SB, true>::run(u);
    }
    __syncthreads();
    if (active) {
#pragma unroll
        for (int q = 0; q < SB; q++) buf[((i * SB + q) << g.log2G) + gi] = u[q];
    }
    __syncthreads();
    // inverse pass 2 (radix SA, p = SB, items i < SB)
    for (int it2 = threadIdx.x; it2 < (SB << g.log2G); it2 += blockDim.x) {
        const int gj = it2 & (G - 1), j = it2 >> g.log2G;
        float2 v[SA];
#pragma unroll
        for (int q = 0; q < SA; q++) {
            const float2 x = buf[((j + q * SB) << g.log2G) + gj];
            if (q == 0) {
                v[q] = x;
            } else {
                float2 w = rt[q * j];
                w.y = -w.y;
                v[q] = cmul(x, w);
            }
        }
        RegDft<SA, true>::run(v);
#pragma unroll
        for (int q = 0; q < SA; q++) {
            const int n2 = j + q * SB;
            float2 w = __ldg(&twrow[n2]);
            w.y = -w.y;
            row[(n2 << g.log2G) + gj] = cmul(v[q], w);
        }
    }
}

// F2, pipelined: the same arithmetic as bpr_rows_filter (bit-identical
// results) in a persistent CTA per SM that walks rows nrows - 1 - r,
// r = blockIdx.x + j * gridDim.x.  A copy warp brings each row (L2 x 16
// complex values, 64000 bytes), its twiddle row and its kernel row by 1-D
// bulk copies into a ring of kF2Ring shared-memory slots, one row ahead of
// the compute warps, and refills a slot as soon as the 13 compute warps have
// released it.  The three
// register passes ping-pong between the slot and one transfer buffer (slot ->
// transfer -> slot), so a row needs only two barriers of the compute warps
// (named barrier 1): one after each exchange.  A failed wait sets the error
// flag; the warps keep the same barrier sequence (skipping their stores), so
// the kernel still ends.
constexpr int kF2Ring = 2;
constexpr int kF2Compute = 416;              // 400 items in the outer passes, 320 in the middle one
constexpr int kF2Threads = kF2Compute + 32;  // and the copy warp

__device__ int g_bp_timeout;  // set when a pipeline wait gave up (checked by the host)

template <int SA, int SB>
struct F2Pipe {
    static constexpr int n = SA * SB;
    static constexpr int G = 16;
    static constexpr int kRowBytes = n * G * 8;
    static constexpr int kTwBytes = n * 8;
    static constexpr int kKernBytes = n * 8;  // (hi, lo) per bin
    static constexpr int kSlotBytes = kRowBytes + kTwBytes + kKernBytes;
    static constexpr size_t kSmemBytes =
        (size_t)kF2Ring * kSlotBytes + kRowBytes /*transfer*/ + n * 8 /*roots*/ + 2 * kF2Ring * 8 /*barriers*/;
    static_assert(kRowBytes % 16 == 0 && kTwBytes % 16 == 0 && kKernBytes % 16 == 0, "bulk copies need 16-byte sizes");
    static_assert(SB * G <= kF2Compute && SA * G <= kF2Compute, "one item per thread");
};

// Named barrier 1 over the compute warps of the row pass.
__device__ __forceinline__ void f2_compute_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kF2Compute) : "memory"); }

template <int SA, int SB>
__global__ void __launch_bounds__(kF2Threads, 1)
    bpr_rows_filter_pipe(float2* __restrict__ scratch, Geom g, const float2* __restrict__ roots,
                         const float2* __restrict__ twL, const float2* __restrict__ kern, int64_t nrows) {
    using P = F2Pipe<SA, SB>;
    constexpr int n = P::n, G = P::G;
    extern __shared__ float4 smem_f4[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(smem_f4);
    float2* xfer = reinterpret_cast<float2*>(smem + (size_t)kF2Ring * P::kSlotBytes);
    float2* rt = xfer + n * G;
    uint64_t* full = reinterpret_cast<uint64_t*>(rt + n);
    uint64_t* empty = full + kF2Ring;
    int* err = &g_bp_timeout;
    const int64_t L1 = g.L1;
    const int64_t mine = (blockIdx.x < nrows) ? (nrows - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    auto slot_ptr = [&](int64_t j) { return smem + (size_t)(j % kF2Ring) * P::kSlotBytes; };
    // rows in reverse order of the batch: the forward-column pass wrote the
    // last units most recently, so the first rows read here are still in L2
    // (and the inverse-column pass, which walks the units forward, finds the
    // first units this pass wrote last)
    auto row_of = [&](int64_t j) {
        const int64_t r = nrows - 1 - (blockIdx.x + j * gridDim.x);
        return MS3_IN_BOUNDS(r, nrows, 104) ? r : int64_t(0);
    };
    auto row_ptr = [&](int64_t j) {
        const int64_t r = row_of(j);
        return scratch + (size_t)(r / L1) * (size_t)(g.L * G) + (size_t)(r % L1) * (n * G);
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < kF2Ring; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], kF2Compute / 32);
        }
        tc::fence_mbar_init();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) rt[i] = roots[i];
    __syncthreads();

    if (threadIdx.x >= kF2Compute) {
        // the copy warp: row j into slot j % kF2Ring once its previous row is released
        if (threadIdx.x == kF2Compute) {
            int64_t issued = 0;
            for (int64_t j = 0; j < mine; j++) {
                if (j >= kF2Ring &&
                    !tc::mbar_wait(&empty[j % kF2Ring], (uint32_t)(((j / kF2Ring) - 1) & 1), err))
                    break;
                const int64_t k1 = row_of(j) % L1;
                uint8_t* slot = slot_ptr(j);
                uint64_t* bar = &full[j % kF2Ring];
                tc::mbar_expect_tx(bar, P::kSlotBytes);
                tc::bulk_load_1d(slot, row_ptr(j), P::kRowBytes, bar);
                tc::bulk_load_1d(slot + P::kRowBytes, twL + k1 * n, P::kTwBytes, bar);
                tc::bulk_load_1d(slot + P::kRowBytes + P::kTwBytes, kern + k1 * n, P::kKernBytes, bar);
                issued = j + 1;
            }
            // no copy may still be landing in shared memory when the CTA exits
            for (int64_t j = (issued > kF2Ring ? issued - kF2Ring : 0); j < issued; j++)
                tc::mbar_wait(&full[j % kF2Ring], (uint32_t)((j / kF2Ring) & 1), err);
        }
        return;
    }

    const int t = threadIdx.x;
    const bool outer = t < SB * G, middle = t < SA * G;
    bool ok = true;
    for (int64_t j = 0; j < mine; j++) {
        // Re-derived every row through an opaque move: otherwise the compiler
        // keeps the 40-odd loop-invariant root offsets q * i in registers
        // across the row loop.
        int i;
        asm volatile("shr.b32 %0, %1, 4;" : "=r"(i) : "r"(t));
        const int gi = t & (G - 1);
        if (ok) ok = tc::mbar_wait(&full[j % kF2Ring], (uint32_t)((j / kF2Ring) & 1), err);
        uint8_t* slot = slot_ptr(j);
        float2* buf = reinterpret_cast<float2*>(slot);
        const float2* tw = reinterpret_cast<const float2*>(slot + P::kRowBytes);
        const float2* kr = reinterpret_cast<const float2*>(slot + P::kRowBytes + P::kTwBytes);
        // forward pass 1 (radix SA over items i < SB): slot -> transfer buffer
        if (outer) {
            float2 u[SA];
#pragma unroll
            for (int q = 0; q < SA; q++) {
                const int n2 = i + q * SB;
                u[q] = cmul(buf[n2 * G + gi], tw[n2]);
            }
            RegDft<SA, false>::run(u);
#pragma unroll
            for (int q = 0; q < SA; q++) xfer[(i * SA + q) * G + gi] = u[q];
        }
        f2_compute_bar();
        // forward pass 2 (radix SB, items i < SA), kernel, inverse pass 1: transfer -> slot
        if (middle) {
            float2 v[SB];
#pragma unroll
            for (int q = 0; q < SB; q++) {
                const float2 x = xfer[(i + q * SA) * G + gi];
                v[q] = (q == 0) ? x : cmul(x, rt[q * i]);
            }
            RegDft<SB, false>::run(v);
#pragma unroll
            for (int q = 0; q < SB; q++) v[q] = kern_mul(v[q], kr[i + q * SA]);
            RegDft<SB, true>::run(v);
#pragma unroll
            for (int q = 0; q < SB; q++) buf[(i * SB + q) * G + gi] = v[q];
        }
        f2_compute_bar();
        // inverse pass 2 (radix SA, items i < SB), twiddle, store
        if (outer) {
            float2 u[SA];
#pragma unroll
            for (int q = 0; q < SA; q++) {
                const float2 x = buf[(i + q * SB) * G + gi];
                if (q == 0) {
                    u[q] = x;
                } else {
                    float2 w = rt[q * i];
                    w.y = -w.y;
                    u[q] = cmul(x, w);
                }
            }
            RegDft<SA, true>::run(u);
            if (ok) {
                float2* row = row_ptr(j);
#pragma unroll
                for (int q = 0; q < SA; q++) {
                    const int n2 = i + q * SB;
                    float2 w = tw[n2];
                    w.y = -w.y;
                    row[n2 * G + gi] = cmul(u[q], w);
                }
            }
        }
        // the slot's generic-proxy accesses are ordered before the next bulk copy into it
        tc::fence_proxy_async_smem();
        __syncwarp();
        if ((t & 31) == 0) tc::mbar_arrive(&empty[j % kF2Ring]);
    }
}

// F3, inverse columns of length L1 = RA * RB (inverse order: radix RB, then
// radix RA), trim / subsample / quantize, store.
// LG, KL2 as for bpr_cols_forward.
// FORM, as the host found: float pairs with direct stores, subsampled (no direct
// stores), or 0 for any.
enum { kDirectFloatPairs = 1, kSubsampled = 2 };
template <int RA, int RB, int LG, int KL2, int FORM>
__global__ void __launch_bounds__(256, 3) bpr_cols_inverse(const float2* __restrict__ scratch, void* __restrict__ out,
                                                        Geom g, const float2* __restrict__ roots, int64_t unit0,
                                                        int direct_ok) {
    constexpr int n = RA * RB;
    const int lg = LG >= 0 ? LG : g.log2G;
    const int64_t L2v = KL2 > 0 ? KL2 : g.L2;
    extern __shared__ float4 smem_f4[];
    float2* buf = reinterpret_cast<float2*>(smem_f4);
    float2* rt = buf + ((size_t)n << lg);
    for (int i = threadIdx.x; i < n; i += blockDim.x) rt[i] = roots[i];
    const int G = 1 << lg;
    const int n2 = blockIdx.x;
    const UnitIdx ui = unit_index(g, unit0 + blockIdx.y);
    const int64_t s0 = (int64_t)ui.grp * G;
    const int64_t ot_base = (ui.c * g.chunk) / g.sub;
    const int L2 = (int)L2v;
    // no subsampling, the whole chunk inside the output: the kept window rows n1 in
    // [60000 / L2, (60000 + chunk) / L2] are exactly q in [kQ0, kQ1) for every item i < RB
    // (checked on the host for this geometry), so plain strided stores of those q only
    constexpr int kQ0 = 4, kQ1 = 12;
    const bool direct = FORM != kSubsampled && direct_ok && g.sub == 1 && g.paired && (ui.c + 1) * g.chunk <= g.N2;
    const bool whole = s0 + G <= g.P;
    const bool pairs_fit =
        FORM == kDirectFloatPairs || (g.m_even && (reinterpret_cast<uintptr_t>(out) & (g.out_i16 ? 3 : 7)) == 0);
    const float2* slab = scratch + (size_t)blockIdx.y * (size_t)(g.L * G);
    for (int it = threadIdx.x; it < (RA << lg); it += blockDim.x) {
        const int gi = it & (G - 1), i = it >> lg;
        float2 u[RB];
        const float2* p = slab + (((size_t)i * L2v + n2) << lg) + gi;
        const size_t step = ((size_t)RA * L2v) << lg;
        const int64_t e0 = (int64_t)((((size_t)i * L2v + n2) << lg) + gi);
#pragma unroll
        for (int q = 0; q < RB; q++)
            u[q] = MS3_IN_BOUNDS(e0 + (int64_t)(q * step), g.L << lg, 105) ? p[q * step] : make_float2(0.f, 0.f);
        RegDft<RB, true>::run(u);
#pragma unroll
        for (int q = 0; q < RB; q++) buf[((i * RB + q) << lg) + gi] = u[q];
    }
    __syncthreads();
    for (int it = threadIdx.x; it < (RB << lg); it += blockDim.x) {
        const int gi = it & (G - 1), i = it >> lg;
        float2 u[RA];
#pragma unroll
        for (int q = 0; q < RA; q++) {
            const float2 x = buf[((i + q * RB) << lg) + gi];
            if (q == 0) {
                u[q] = x;
            } else {
                float2 w = rt[q * i];
                w.y = -w.y;
                u[q] = cmul(x, w);
            }
        }
        RegDft<RA, true>::run(u);
        if (direct) {
            const int64_t s = s0 + gi;
            const bool two = FORM == kDirectFloatPairs || 2 * s + 1 < g.M;
            const int64_t step = (int64_t)RB * L2 * g.M;
            const int64_t at = (ot_base + (int64_t)i * L2 + n2 - kOverlap + (int64_t)kQ0 * RB * L2) * g.M + 2 * s;
            if (whole || s < g.P) {
#pragma unroll
                for (int q = kQ0; q < kQ1; q++) {
                    const int64_t o = at + (q - kQ0) * step;
                    if (!MS3_IN_BOUNDS(o + (two ? 1 : 0), g.N2 * g.M, 102)) continue;
                    if (FORM != kDirectFloatPairs && g.out_i16) {
                        int16_t* o16 = static_cast<int16_t*>(out) + o;
                        const int16_t a = x86_float_to_int16((float)((double)u[q].x * g.qscale));
                        const int16_t b = x86_float_to_int16((float)((double)u[q].y * g.qscale));
                        if (pairs_fit) {
                            *reinterpret_cast<short2*>(o16) = make_short2(a, b);
                        } else {
                            o16[0] = a;
                            if (two) o16[1] = b;
                        }
                    } else {
                        float* of = static_cast<float*>(out) + o;
                        if (pairs_fit) {
                            *reinterpret_cast<float2*>(of) = u[q];
                        } else {
                            of[0] = u[q].x;
                            if (two) of[1] = u[q].y;
                        }
                    }
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < RA; q++) {
                const int n1 = i + q * RB;
                store_filtered(out, g, ot_base, s0 + gi, n1 * L2 + n2, u[q]);
            }
        }
    }
}

// Two-pass factorisations compiled for the reference's canonical window
// (chunk 120000, L = 240000 = 480 x 500, used whenever M * T >= 187).
constexpr int kFastRA = 16, kFastRB = 30;  // L1 = 480
constexpr int kFastSA = 20, kFastSB = 25;  // L2 = 500
constexpr int kFastL2 = kFastSA * kFastSB;

// ---------------------------------------------------------------- plans

int max_prime_factor(int64_t n) {
    int64_t m = 1;
    for (int64_t p = 2; p * p <= n; p++)
        while (n % p == 0) { m = std::max(m, p); n /= p; }
    if (n > 1) m = std::max(m, n);
    return (int)m;
}

SubFft make_subfft(int n, std::vector<float2>& tw) {
    SubFft P{};
    P.n = n;
    std::vector<int> rad;
    int m = n;
    while (m % 8 == 0) { rad.push_back(8); m /= 8; }
    while (m % 4 == 0) { rad.push_back(4); m /= 4; }
    while (m % 2 == 0) { rad.push_back(2); m /= 2; }
    while (m % 5 == 0) { rad.push_back(5); m /= 5; }
    while (m % 3 == 0) { rad.push_back(3); m /= 3; }
    for (int f = 7; f <= m; f += 2)
        while (m % f == 0) { rad.push_back(f); m /= f; }
    if ((int)rad.size() > kMaxPasses) throw_unsupported("FFT factor has too many passes");
    P.npass = (int)rad.size();
    int64_t p = 1;
    tw.clear();
    for (int s = 0; s < P.npass; s++) {
        const int r = rad[s];
        P.radix[s] = r;
        P.p[s] = (int)p;
        P.twoff[s] = (int)tw.size();
        for (int64_t k = 0; k < p; k++)
            for (int q = 0; q < r; q++) {
                const int64_t num = (q * k) % (p * r);
                const double a = -2.0 * M_PI * (double)num / (double)(p * r);
                tw.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
            }
        p *= r;
    }
    if (n == 1) P.npass = 0;
    P.twlen = (int)tw.size();
    return P;
}

size_t smem_bytes_for(const SubFft& P, int G) {
    return ((size_t)2 * P.n * G + (size_t)P.twlen + (size_t)extra_entries(P)) * sizeof(float2);
}

// Device-resident tables for one (L, filter) combination.
struct BandpassPlan {
    int device = -1;
    int64_t L = 0, L1 = 0, L2 = 0;  // FFT length = L1 * L2
    int64_t Lw = 0;                 // window length (L == Lw unless the window is zero-padded)
    int paired = 1;
    SubFft P1{}, P2{};
    float2* tw1 = nullptr;  // P1 twiddles
    float2* tw2 = nullptr;  // P2 twiddles
    float2* twL = nullptr;  // [k1][n2] exp(-2 pi i n2 k1 / L)
    float2* kern = nullptr;  // [k1][k2] kernel[k1 + L1 k2] / L as (hi, lo) floats
    float2* root1 = nullptr;  // exp(-2 pi i e / L1), e < L1
    float2* root2 = nullptr;  // exp(-2 pi i e / L2), e < L2
    bool fast = false;        // L1 x L2 = 480 x 500: register-pass kernels
    ~BandpassPlan() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (device >= 0) cudaSetDevice(device);
        cudaFree(tw1);
        cudaFree(tw2);
        cudaFree(twL);
        cudaFree(kern);
        cudaFree(root1);
        cudaFree(root2);
        if (cur >= 0) cudaSetDevice(cur);
    }
};

// Choose L = L1 * L2 with both factors built from primes <= kMaxGenericRadix,
// minimising the larger factor.
bool factor_window(int64_t L, int64_t& L1, int64_t& L2) {
    int64_t best = -1;
    for (int64_t a = 1; a * a <= L; a++) {
        if (L % a) continue;
        const int64_t b = L / a;
        if (max_prime_factor(a) > kMaxGenericRadix || max_prime_factor(b) > kMaxGenericRadix) continue;
        if (best < 0 || b < best) { best = b; L1 = a; L2 = b; }
    }
    if (best < 0) return false;
    // the longer transform goes to the contiguous (row) pass
    if (L1 > L2) std::swap(L1, L2);
    return true;
}

// The band kernel of a window of length n (define_kernel,
// p_bandpass_filter.cpp:421-447), in FP64.
std::vector<double> band_kernel(int64_t n, double fs, double fmin, double fmax, double fwid) {
    std::vector<double> K((size_t)n);
    const double T = n / fs;
    const double df = 1 / T;
    for (int64_t i = 0; i < n; i++) {
        const double fgrid = (i <= (n + 1) / 2) ? df * i : df * (i - n);
        const double absf = std::fabs(fgrid);
        double val = 1.0;
        if (fmin != 0) {
            if (i == 0)
                val = 0.0;
            else
                val *= (1 + std::erf(3.0 * (absf - fmin) / fmin)) / 2;
        }
        if (fmax != 0) val *= (1 - std::erf((absf - fmax) / fwid)) / 2;
        K[(size_t)i] = std::sqrt(val);
    }
    return K;
}

// Lw: the reference's window length (chunk + 120000).  When Lw factors into
// primes up to 64 the FFT has length Lw and the kernel is kernel / Lw, as in
// the reference.  Otherwise (a prime factor above 64, e.g. Lw = 466033 or
// 1398101 = 23 * 89 * 683) the window's circular convolution is done with an
// FFT of a 5-smooth length L >= 2 Lw - 1: the reference computes, per window,
//     y = Re(IDFT(kernel .* DFT(x))) / Lw = x (*) h  (circular, length Lw),
//     h[j] = Re(sum_k kernel[k] exp(2 pi i j k / Lw)) / Lw   (real, even),
// and with the window zero-padded to L and the taps laid out as g[j] = h[j],
// g[L - j] = h[j] (0 < j < Lw), the length-L circular convolution x (*) g
// equals y on [0, Lw) because L >= 2 Lw - 1 leaves no wrap-around.  g is
// symmetric, so DFT_L(g) is real and even and the L-point plan applies it as
// it applies the band kernel (channel pairs included).  h and DFT_L(g) are
// formed in FP64 on the host.
std::shared_ptr<BandpassPlan> build_plan(int64_t Lw, double fs, double fmin, double fmax, double fwid) {
    constexpr int64_t kMaxRow = 8192;  // longest row transform of a zero-padded plan (shared memory)
    auto plan = std::make_shared<BandpassPlan>();
    MS3_CUDA(cudaGetDevice(&plan->device));
    plan->Lw = Lw;
    const std::vector<double> Kw = band_kernel(Lw, fs, fmin, fmax, fwid);
    std::vector<double> KF;  // the kernel applied to the L-point spectrum, including the 1/L
    int64_t L = Lw;
    if (factor_window(Lw, plan->L1, plan->L2) && plan->L2 <= 16384) {
        KF.resize((size_t)Lw);
        for (int64_t i = 0; i < Lw; i++) KF[(size_t)i] = Kw[(size_t)i] * (1.0 / Lw);
    } else {
        L = hostdft::next_smooth5(2 * Lw - 1);
        while (!(factor_window(L, plan->L1, plan->L2) && plan->L2 <= kMaxRow)) L = hostdft::next_smooth5(L + 1);
        std::vector<hostdft::cd> kc((size_t)Lw);
        for (int64_t i = 0; i < Lw; i++) kc[(size_t)i] = Kw[(size_t)i];
        const std::vector<hostdft::cd> hc = hostdft::dft(kc, +1);
        std::vector<hostdft::cd> g((size_t)L, hostdft::cd(0));
        for (int64_t j = 0; j < Lw; j++) {
            const double h = hc[(size_t)j].real() / (double)Lw;
            g[(size_t)j] = h;
            if (j > 0) g[(size_t)(L - j)] = h;
        }
        const std::vector<hostdft::cd> G = hostdft::dft(g, -1);
        KF.resize((size_t)L);
        for (int64_t i = 0; i < L; i++) KF[(size_t)i] = G[(size_t)i].real() / (double)L;
        for (int64_t i = 1; i < L; i++) KF[(size_t)i] = KF[(size_t)(L - i)] = 0.5 * (KF[(size_t)i] + KF[(size_t)(L - i)]);
    }
    plan->L = L;
    const int64_t L1 = plan->L1, L2 = plan->L2;
    std::vector<float2> tw1, tw2;
    plan->P1 = make_subfft((int)L1, tw1);
    plan->P2 = make_subfft((int)L2, tw2);

    // Two channels can share one complex transform only if the kernel is even.
    plan->paired = 1;
    for (int64_t i = 1; i < L; i++)
        if (KF[(size_t)i] != KF[(size_t)(L - i)]) { plan->paired = 0; break; }
    if (const char* up = std::getenv("MS3GPU_BP_UNPAIRED"))  // one channel per complex signal (testing)
        if (up[0] == '1') plan->paired = 0;

    std::vector<float2> kern((size_t)L);
    std::vector<float2> twL((size_t)L);
    for (int64_t k1 = 0; k1 < L1; k1++)
        for (int64_t j = 0; j < L2; j++) {
            const double kd = KF[(size_t)(k1 + L1 * j)];
            const float hi = (float)kd;
            kern[(size_t)(k1 * L2 + j)] = make_float2(hi, (float)(kd - (double)hi));
            const double a = -2.0 * M_PI * (double)(j * k1) / (double)L;
            twL[(size_t)(k1 * L2 + j)] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
    MS3_CUDA(cudaMalloc(&plan->tw1, std::max<size_t>(1, tw1.size()) * sizeof(float2)));
    MS3_CUDA(cudaMalloc(&plan->tw2, std::max<size_t>(1, tw2.size()) * sizeof(float2)));
    MS3_CUDA(cudaMalloc(&plan->twL, (size_t)L * sizeof(float2)));
    MS3_CUDA(cudaMalloc(&plan->kern, (size_t)L * sizeof(float2)));
    if (!tw1.empty()) MS3_CUDA(cudaMemcpy(plan->tw1, tw1.data(), tw1.size() * sizeof(float2), cudaMemcpyHostToDevice));
    if (!tw2.empty()) MS3_CUDA(cudaMemcpy(plan->tw2, tw2.data(), tw2.size() * sizeof(float2), cudaMemcpyHostToDevice));
    MS3_CUDA(cudaMemcpy(plan->twL, twL.data(), (size_t)L * sizeof(float2), cudaMemcpyHostToDevice));
    MS3_CUDA(cudaMemcpy(plan->kern, kern.data(), (size_t)L * sizeof(float2), cudaMemcpyHostToDevice));
    auto roots = [](int64_t n) {
        std::vector<float2> r((size_t)n);
        for (int64_t e = 0; e < n; e++) {
            const double a = -2.0 * M_PI * (double)e / (double)n;
            r[(size_t)e] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
        return r;
    };
    const std::vector<float2> r1 = roots(L1), r2 = roots(L2);
    MS3_CUDA(cudaMalloc(&plan->root1, (size_t)L1 * sizeof(float2)));
    MS3_CUDA(cudaMalloc(&plan->root2, (size_t)L2 * sizeof(float2)));
    MS3_CUDA(cudaMemcpy(plan->root1, r1.data(), (size_t)L1 * sizeof(float2), cudaMemcpyHostToDevice));
    MS3_CUDA(cudaMemcpy(plan->root2, r2.data(), (size_t)L2 * sizeof(float2), cudaMemcpyHostToDevice));
    plan->fast = plan->paired && L1 == kFastRA * kFastRB && L2 == kFastSA * kFastSB;
    const char* nofast = std::getenv("MS3GPU_BP_GENERIC");
    if (nofast && nofast[0] == '1') plan->fast = false;
    return plan;
}

std::mutex g_plan_mu;
std::map<std::tuple<int, int64_t, double, double, double, double>, std::shared_ptr<BandpassPlan>> g_plans;

std::shared_ptr<BandpassPlan> get_plan(int64_t L, double fs, double fmin, double fmax, double fwid) {
    int dev = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    auto key = std::make_tuple(dev, L, fs, fmin, fmax, fwid);
    std::lock_guard<std::mutex> lk(g_plan_mu);
    auto it = g_plans.find(key);
    if (it != g_plans.end()) return it->second;
    if (g_plans.size() >= 16) g_plans.clear();
    auto p = build_plan(L, fs, fmin, fmax, fwid);
    g_plans[key] = p;
    return p;
}

size_t env_size(const char* name, size_t dflt) {
    const char* v = std::getenv(name);
    if (!v || !*v) return dflt;
    return (size_t)std::strtoull(v, nullptr, 10);
}

}  // namespace

int64_t bandpass_chunk_size(int64_t M, int64_t num_threads) {
    // p_bandpass_filter.cpp:147-155
    const int overhead = 6;
    const int64_t overlap_size = kOverlap;
    const int64_t min_chunk_size = overlap_size * 2;
    const double target_ram_bytes = 1.0 * (1024 * 1024 * 1024);
    const double target_chunk_size =
        target_ram_bytes / (overhead * sizeof(float) * M * num_threads) - 2 * overlap_size;
    int64_t chunk_size = (int64_t)(target_chunk_size);
    if (chunk_size < min_chunk_size) chunk_size = min_chunk_size;
    return chunk_size;
}

void bandpass_output_rows(int64_t N, int64_t chunk, int sub, int64_t c_begin, int64_t c_end, int64_t& o0,
                          int64_t& o1) {
    o0 = std::min(N / sub, (c_begin * chunk) / sub);
    o1 = std::min(N / sub, (c_end * chunk) / sub);
}

void bandpass_device(const void* raw, int64_t M, int64_t N, void* out, const BandpassParams& bp,
                     cudaStream_t stream, int64_t c_begin, int64_t c_end, bool in_i16, int64_t raw_row0,
                     int64_t out_row0) {
    const int sub = bp.subsample_factor ? bp.subsample_factor : 1;
    if (sub < 1) throw_invalid("subsample_factor must be >= 1");
    const int64_t N2 = N / sub;
    const bool out_i16 = bp.quantization_unit != 0;
    if (raw_row0 < 0 || out_row0 < 0) throw_invalid("negative slab origin");
    if (bp.freq_max == 0) {
        // p_bandpass_filter.cpp:117-119: the input file is copied unchanged.
        if (raw_row0 != 0 || out_row0 != 0) throw_invalid("the copy (freq_max 0) takes whole recordings");
        if (M * N > 0)
            MS3_CUDA(cudaMemcpyAsync(out, raw, (in_i16 ? 2 : 4) * (size_t)(M * N), cudaMemcpyDeviceToDevice,
                                     stream));
        return;
    }
    if (M <= 0 || N2 <= 0) return;
    if (bp.num_threads < 1) throw_invalid("num_threads must be >= 1");
    const int64_t chunk = bandpass_chunk_size(M, bp.num_threads);
    const int64_t Lw = chunk + 2 * kOverlap;
    auto plan = get_plan(Lw, bp.samplerate, bp.freq_min, bp.freq_max, bp.freq_wid);
    const int64_t L = plan->L;  // FFT length (Lw, or a zero-padded length)

    Geom g{};
    g.M = M;
    g.N = N;
    g.paired = plan->paired;
    g.P = g.paired ? (M + 1) / 2 : M;
    // pair loads (float2, or short2 for int16 input) and float2 stores need
    // even M and aligned caller buffers
    g.in_i16 = in_i16 ? 1 : 0;
    g.m_even = (M % 2 == 0) && ((uintptr_t)raw % (in_i16 ? 4 : 8) == 0) &&
               (out_i16 || ((uintptr_t)out % 8 == 0));
    g.L = L;
    g.Lw = Lw;
    g.L1 = plan->L1;
    g.L2 = plan->L2;
    g.chunk = chunk;
    g.sub = sub;
    g.N2 = N2;
    g.out_i16 = out_i16 ? 1 : 0;
    g.half_lines = (out_i16 && sub == 1) || (in_i16 && M % 32 == 0);
    g.qscale = out_i16 ? 1.0 / bp.quantization_unit : 1.0;
    // signals per unit: up to 16, limited by the shared-memory budget
    // signals per unit: 16 by default (MS3GPU_BP_LOG2G lowers it, for tuning)
    int log2G = (int)std::min<size_t>(4, env_size("MS3GPU_BP_LOG2G", 4));
    while (log2G > 0 && ((int64_t(1) << (log2G - 1)) >= g.P)) log2G--;
    while (log2G > 0 && (smem_bytes_for(plan->P1, 1 << log2G) > kSmemBudget ||
                         smem_bytes_for(plan->P2, 1 << log2G) > kSmemBudget))
        log2G--;
    const size_t sm1 = smem_bytes_for(plan->P1, 1 << log2G);
    const size_t sm2 = smem_bytes_for(plan->P2, 1 << log2G);
    if (sm1 > kSmemBudget || sm2 > kSmemBudget)
        throw_unsupported("FFT factors of L=" + std::to_string(L) + " exceed shared memory");
    g.log2G = log2G;
    const int G = 1 << log2G;
    g.ngroups = (int)ceil_div(g.P, G);
    const int64_t nchunks = ceil_div(N, chunk);
    if (c_end < 0 || c_end > nchunks) c_end = nchunks;
    if (c_begin < 0) c_begin = 0;
    if (c_begin >= c_end) return;
    g.c_begin = c_begin;
    g.nwin = c_end - c_begin;
    const int64_t units = g.nwin * g.ngroups;
    const size_t unit_bytes = (size_t)L * G * sizeof(float2);
    const size_t budget = env_size("MS3GPU_BP_SCRATCH_MB", 4096) << 20;
    int64_t per_batch = std::max<int64_t>(1, (int64_t)(budget / unit_bytes));
    per_batch = std::min<int64_t>(per_batch, std::min<int64_t>(units, 65535));

    static bool attrs_set[64] = {false};
    {
        int dev = 0;
        MS3_CUDA(cudaGetDevice(&dev));
        if (dev < 64 && !attrs_set[dev]) {
            const int lim = (int)kSmemBudget;
            MS3_CUDA(cudaFuncSetAttribute(bp_cols_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bp_rows_filter, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bp_cols_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_forward<kFastRA, kFastRB, -1, 0, kAnyForm>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kFloatPairs>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kInt16Pairs>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kOddCount>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_rows_filter<kFastSA, kFastSB>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_inverse<kFastRA, kFastRB, -1, 0, kAnyForm>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kAnyForm>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kDirectFloatPairs>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kSubsampled>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
            MS3_CUDA(cudaFuncSetAttribute(bpr_rows_filter_pipe<kFastSA, kFastSB>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)F2Pipe<kFastSA, kFastSB>::kSmemBytes));
            attrs_set[dev] = true;
        }
    }
    // Gaps between subsampled chunks stay zero, as in the preallocated file.
    const size_t in_esz = in_i16 ? 2 : 4, out_esz = out_i16 ? 2 : 4;
    if (sub > 1 && chunk % sub != 0) {
        int64_t o0 = 0, o1 = 0;
        bandpass_output_rows(N, chunk, sub, c_begin, c_end, o0, o1);
        if (o0 < out_row0) throw_invalid("output slab starts after the windows' first row");
        if (o1 > o0)
            MS3_CUDA(cudaMemsetAsync(static_cast<char*>(out) + (size_t)((o0 - out_row0) * M) * out_esz, 0,
                                     out_esz * (size_t)((o1 - o0) * M), stream));
    }
    // The kernels index rows of the whole recording: a slab's pointers are
    // moved back to where row 0 would be (only rows inside the slab are read
    // or written).  Shifts are whole rows, so alignment is unchanged.
    raw = reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(raw) - (uintptr_t)(raw_row0 * M) * in_esz);
    out = reinterpret_cast<void*>(reinterpret_cast<uintptr_t>(out) - (uintptr_t)(out_row0 * M) * out_esz);
    int nsm = 0;
    {
        int dev = 0;
        MS3_CUDA(cudaGetDevice(&dev));
        MS3_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    }
    // fewer units per launch batch when the device has no room for the full scratch
    DevBuf scratch;
    for (;;) {
        try {
            scratch.alloc((size_t)per_batch * unit_bytes, stream);
            break;
        } catch (const Error& e) {
            if (e.code != MS3GPU_ERR_NOMEM || per_batch == 1) throw;
            per_batch = (per_batch + 1) / 2;
        }
    }
    const size_t fsm1 = ((size_t)plan->L1 * G + plan->L1) * sizeof(float2);
    const size_t fsm2 = ((size_t)plan->L2 * G + plan->L2) * sizeof(float2);
    // the register-pass inverse stores kept rows q in [4, 12) of each 16-point
    // column transform directly when the trim falls on those row boundaries
    const int direct_ok = (plan->fast && kOverlap == 4 * kFastRB * plan->L2 &&
                           chunk == 8 * kFastRB * plan->L2) ? 1 : 0;
    // the forms of the 16-signal kernels' loads and stores
    const auto forward4 = !g.m_even ? bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kOddCount>
                          : in_i16  ? bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kInt16Pairs>
                                    : bpr_cols_forward<kFastRA, kFastRB, 4, kFastL2, kFloatPairs>;
    const bool float_pairs = g.m_even && !out_i16 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    const auto inverse4 = sub > 1 ? bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kSubsampled>
                          : float_pairs ? bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kDirectFloatPairs>
                                        : bpr_cols_inverse<kFastRA, kFastRB, 4, kFastL2, kAnyForm>;
    for (int64_t u0 = 0; u0 < units; u0 += per_batch) {
        const int64_t nb = std::min<int64_t>(per_batch, units - u0);
        dim3 g1((unsigned)plan->L2, (unsigned)nb);
        dim3 g2((unsigned)plan->L1, (unsigned)nb);
        float2* sc = scratch.as<float2>();
        if (plan->fast) {
            if (g.log2G == 4)
                forward4<<<g1, 256, fsm1, stream>>>(raw, sc, g, plan->root1, u0);
            else
                bpr_cols_forward<kFastRA, kFastRB, -1, 0, kAnyForm><<<g1, 256, fsm1, stream>>>(raw, sc, g, plan->root1, u0);
            MS3_LAUNCH_CHECK();
            if (G == F2Pipe<kFastSA, kFastSB>::G && reinterpret_cast<uintptr_t>(sc) % 16 == 0) {
                const int64_t nrows = nb * plan->L1;
                bpr_rows_filter_pipe<kFastSA, kFastSB>
                    <<<(unsigned)std::min<int64_t>(nrows, nsm), kF2Threads, F2Pipe<kFastSA, kFastSB>::kSmemBytes,
                       stream>>>(sc, g, plan->root2, plan->twL, plan->kern, nrows);
            } else {
                bpr_rows_filter<kFastSA, kFastSB><<<g2, kFastSA * G, fsm2, stream>>>(sc, g, plan->root2, plan->twL,
                                                                                     plan->kern);
            }
            MS3_LAUNCH_CHECK();
            if (g.log2G == 4)
                inverse4<<<g1, 256, fsm1, stream>>>(sc, out, g, plan->root1, u0, direct_ok);
            else
                bpr_cols_inverse<kFastRA, kFastRB, -1, 0, kAnyForm>
                    <<<g1, 256, fsm1, stream>>>(sc, out, g, plan->root1, u0, direct_ok);
            MS3_LAUNCH_CHECK();
        } else {
            bp_cols_forward<<<g1, kThreads, sm1, stream>>>(raw, sc, g, plan->P1, plan->tw1, u0);
            MS3_LAUNCH_CHECK();
            bp_rows_filter<<<g2, kThreads, sm2, stream>>>(sc, g, plan->P2, plan->tw2, plan->twL, plan->kern);
            MS3_LAUNCH_CHECK();
            bp_cols_inverse<<<g1, kThreads, sm1, stream>>>(sc, out, g, plan->P1, plan->tw1, u0);
            MS3_LAUNCH_CHECK();
        }
    }
}

void bandpass_read_timeout(int* flag, cudaStream_t stream) {
    MS3_CUDA(cudaMemcpyFromSymbolAsync(flag, g_bp_timeout, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
}

void bandpass_check_timeout(cudaStream_t stream) {
    int h = 0;
    bandpass_read_timeout(&h, stream);
    MS3_CUDA(cudaStreamSynchronize(stream));
    bandpass_raise_timeout(h, stream);
}

void bandpass_raise_timeout(int flag, cudaStream_t stream) {
    if (flag) {
        const int zero = 0;
        MS3_CUDA(cudaMemcpyToSymbolAsync(g_bp_timeout, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
        MS3_CUDA(cudaStreamSynchronize(stream));
        throw Error(MS3GPU_ERR_CUDA, "bandpass: pipeline wait timed out");
    }
}

int bounds_site_bandpass(cudaStream_t s) {
#ifdef MS3GPU_BOUNDS_CHECK
    return take_bounds_site(s);
#else
    (void)s;
    return 0;
#endif
}

}  // namespace ms3gpu
