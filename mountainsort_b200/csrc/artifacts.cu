// ms3.mask_out_artifacts on the GPU (packages/ms3/p_mask_out_artifacts.cpp:24-104),
// the next step on the filtered or whitened timeseries in some pipelines.
//
//   norms(m, i) = sqrt(sum_{a < I} x(m, i*I + a)^2)      i < N / I (floor), double,
//                 summed in timepoint order as the reference's loop does
//   per channel: mean and sample stdev of its norms (MLCompute::mean / stdev,
//                common/mlcompute.cpp:67-85, sums in interval order)
//   an interval whose norm exceeds mean + threshold * stdev on any channel
//   masks itself and its two neighbours (the reference's write to use_it[-1]
//   for interval 0 lands outside the array and is dropped here)
//   out = x on the kept intervals, 0 on masked intervals and on the tail
//         beyond the last whole interval (never written by the reference).
//
// Four kernels: norms (one thread per channel and interval), per-channel limits,
// interval flags (a few by the limits kernel), and a masked copy.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "artifacts.h"
#include "common.cuh"

namespace ms3gpu {

namespace {

// norms[i * M + m]: a thread per channel and interval, neighbouring threads taking
// neighbouring channels.  The sum is in timepoint order (8 cycles an addition), so what
// counts is loads in flight: sixteen per thread, and no thread idle when M is not a
// multiple of the block (64 channels x 3M, intervals of 2000: 683 us with 128-thread
// rows and loads as the loop came to them, now 197 us).
// AHEAD: the next sixteen load during the additions, for few sums (below 512 per SM):
// 64 channels x 1.6 M 396 us a call without, 312 with; x 3 M, whose sums are enough
// to hide the loads, 549 and 568.
constexpr int kBatch = 16;
template <bool AHEAD>
__global__ void __launch_bounds__(128) artifact_norms(const float* __restrict__ X, int64_t M, int64_t I, int64_t nint,
                                                      double* __restrict__ norms) {
    const int64_t n = M * nint, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        const int64_t i = k / M, m = k - i * M;
        const float* p = X + i * I * M + m;
        double s = 0.0;
        int64_t a = 0;
        float b[kBatch];
        if (AHEAD && I >= kBatch) {
#pragma unroll
            for (int j = 0; j < kBatch; j++) b[j] = __ldg(p + j * M);
        }
        for (; a + kBatch <= I; a += kBatch) {
            float c[kBatch];
            if (AHEAD ? a + 2 * kBatch <= I : true) {
                const float* from = p + (AHEAD ? a + kBatch : a) * M;
#pragma unroll
                for (int j = 0; j < kBatch; j++) c[j] = __ldg(from + j * M);
            }
#pragma unroll
            for (int j = 0; j < kBatch; j++) {
                const double v = (double)(AHEAD ? b[j] : c[j]);
                s = __dadd_rn(s, __dmul_rn(v, v));
            }
            if (AHEAD) {
#pragma unroll
                for (int j = 0; j < kBatch; j++) b[j] = c[j];
            }
        }
        for (; a < I; a++) {
            const double v = (double)p[a * M];
            s = __dadd_rn(s, __dmul_rn(v, v));
        }
        norms[k] = sqrt(s);
    }
}

// limits[m] = mean + threshold * stdev of channel m's norms, summed in interval order:
// the block brings in 32 channels x kTile intervals at a time, its first warp adds them
// (one channel per lane), the next tile on its way meanwhile.  With a few intervals the
// block flags its own channels' (exceed) instead of storing the limits: a kernel and an
// allocation less (2 channels x 999 timepoints: 64.2 us a call, now 60.5).
constexpr int kTile = 64;
constexpr int64_t kFewIntervals = 256;
__global__ void __launch_bounds__(256) artifact_limits(const double* __restrict__ norms, int64_t M, int64_t nint,
                                                       double threshold, double* __restrict__ limits,
                                                       int* __restrict__ exceed) {
    __shared__ double tile[2][kTile][32];
    __shared__ double found[32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t m = (int64_t)blockIdx.x * 32 + l;
    auto bring = [&](int64_t i0, int b) {
        for (int r = w; r < kTile; r += 8)
            tile[b][r][l] = (i0 + r < nint && m < M) ? norms[(i0 + r) * M + m] : 0.0;
    };
    double sum = 0.0, sumsqr = 0.0;
    bring(0, 0);
    __syncthreads();
    int b = 0;
    for (int64_t i0 = 0; i0 < nint; i0 += kTile, b ^= 1) {
        if (i0 + kTile < nint && w > 0) {  // warps 1..7 bring the next tile
            for (int r = w - 1; r < kTile; r += 7) {
                const int64_t i = i0 + kTile + r;
                tile[b ^ 1][r][l] = (i < nint && m < M) ? norms[i * M + m] : 0.0;
            }
        }
        if (w == 0) {
            const int n = (int)(nint - i0 < kTile ? nint - i0 : kTile);
#pragma unroll 8
            for (int r = 0; r < n; r++) {
                const double v = tile[b][r][l];
                sum = __dadd_rn(sum, v);
                sumsqr = __dadd_rn(sumsqr, __dmul_rn(v, v));
            }
        }
        __syncthreads();
    }
    if (w == 0) {
        const double mean0 = nint ? __ddiv_rn(sum, (double)nint) : 0.0;
        double sigma0 = 0.0;
        if (nint >= 2) {
            const double ct = (double)nint;
            sigma0 = sqrt(__ddiv_rn(__dsub_rn(sumsqr, __ddiv_rn(__dmul_rn(sum, sum), ct)), ct - 1.0));
        }
        const double limit = __dadd_rn(mean0, __dmul_rn(sigma0, threshold));
        if (!exceed && m < M) limits[m] = limit;
        found[l] = limit;
    }
    if (!exceed) return;
    __syncthreads();
    if (m < M) {
#pragma unroll 4
        for (int64_t i = w; i < nint; i += 8)
            if (norms[i * M + m] > found[l]) exceed[i] = 1;
    }
}

// exceed[i] is set for an interval whose norm is beyond its channel's limit.
__global__ void __launch_bounds__(256) artifact_flags(const double* __restrict__ norms, int64_t M, int64_t nint,
                                                      const double* __restrict__ limits, int* __restrict__ exceed) {
    const int64_t n = M * nint, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        const int64_t i = k / M;
        if (norms[k] > limits[k - i * M]) exceed[i] = 1;
    }
}

// out(m, t) = x(m, t) where interval t / I is kept, else 0; X and out hold the N
// timepoints from t0.  An interval is one stretch of memory, kept or not as a whole:
// blocks take stretches of kStretch values of it, copy them 16 bytes at a time where
// both sides allow, and do not read what they clear.  (A 64-bit division per value bound
// the flat copy: 668 us for 64 channels x 3M, now 248 us.)
constexpr int64_t kStretch = 16384;
__global__ void __launch_bounds__(256) artifact_write(const float* X, int64_t M, int64_t N, int64_t I, int64_t nint,
                                                      const int* __restrict__ exceed, float* out, int64_t t0,
                                                      int64_t stretches, int64_t total) {
    for (int64_t s = blockIdx.x; s < total; s += gridDim.x) {
        const int64_t i = t0 / I + s / stretches;  // interval
        const int64_t first = i * I > t0 ? i * I : t0, last = (i + 1) * I < t0 + N ? (i + 1) * I : t0 + N;
        const int64_t end = (last - t0) * M;
        const int64_t a = (first - t0) * M + (s % stretches) * kStretch;
        const int64_t e = a + kStretch < end ? a + kStretch : end;
        bool keep = i < nint;
        if (keep) keep = !exceed[i] && !exceed[i + 1] && !(i >= 1 && exceed[i - 1]);
        // up to three values to a 16-byte boundary of the output, then fours
        const int64_t h = min(e, a + (int64_t)(((16 - (reinterpret_cast<uintptr_t>(out + a) & 15)) & 15) / 4));
        const bool fours = a < e && (!keep || ((reinterpret_cast<uintptr_t>(X + h) & 15) == 0));
        const int64_t v = fours ? (e - h) / 4 : 0;
        if (a < e) {
            for (int64_t k = a + threadIdx.x; k < h; k += blockDim.x) out[k] = keep ? X[k] : 0.f;
            float4* o4 = reinterpret_cast<float4*>(out + h);
            const float4* x4 = reinterpret_cast<const float4*>(X + h);
            if (keep) {
#pragma unroll 4
                for (int64_t k = threadIdx.x; k < v; k += blockDim.x) o4[k] = x4[k];
            } else {
                for (int64_t k = threadIdx.x; k < v; k += blockDim.x) o4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            for (int64_t k = h + 4 * v + threadIdx.x; k < e; k += blockDim.x) out[k] = keep ? X[k] : 0.f;
        }
    }
}

// The same value by value: short intervals, where a block per stretch would have little
// to do (whole calls, 4 channels x 3M by stretches and value by value: 849 and 794 us at
// 400 values an interval, 453 and 462 at 800; 64 channels x 500k, 2048 values: 614 and 690).
__global__ void __launch_bounds__(256) artifact_write_flat(const float* X, int64_t M, int64_t N, int64_t I, int64_t nint,
                                                           const int* __restrict__ exceed, float* out, int64_t t0) {
    const int64_t total = M * N;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = (t0 + k / M) / I;
        bool keep = i < nint;
        if (keep) keep = !exceed[i] && !exceed[i + 1] && !(i >= 1 && exceed[i - 1]);
        out[k] = keep ? X[k] : 0.f;
    }
}
constexpr int64_t kShortInterval = 600;  // values

int sm_count() {
    int dev = 0, n = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    MS3_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    return n;
}

}  // namespace

int64_t mask_out_artifacts_device(const float* X, int64_t M, int64_t N, double threshold, int64_t interval_size,
                                  float* out, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const int64_t I = interval_size;
    const int64_t nint = N / I;
    DevBuf norms(sizeof(double) * (size_t)std::max<int64_t>(1, nint * M), stream);
    DevBuf exceed(sizeof(int) * (size_t)(nint + 2), stream);
    if (nint > 0) artifact_norms_device(X, M, I, nint, norms.as<double>(), stream);
    artifact_flags_device(norms.as<double>(), M, nint, threshold, exceed.as<int>(), stream);
    artifact_write_device(X, M, N, 0, I, nint, exceed.as<int>(), out, stream);
    return artifact_kept(exceed.as<int>(), nint, I, stream);
}

void artifact_norms_device(const float* X, int64_t M, int64_t I, int64_t nint, double* norms, cudaStream_t stream) {
    if (M <= 0 || nint <= 0) return;
    const int threads = M * nint < (int64_t)sm_count() * 128 ? 32 : 128;  // few sums: on more SMs
    const int64_t blocks = std::min<int64_t>(ceil_div(M * nint, threads), (int64_t)sm_count() * 64);
    if (M * nint < (int64_t)sm_count() * 512)
        artifact_norms<true><<<(unsigned)blocks, threads, 0, stream>>>(X, M, I, nint, norms);
    else
        artifact_norms<false><<<(unsigned)blocks, threads, 0, stream>>>(X, M, I, nint, norms);
    MS3_LAUNCH_CHECK();
}

void artifact_flags_device(const double* norms, int64_t M, int64_t nint, double threshold, int* exceed,
                           cudaStream_t stream) {
    MS3_CUDA(cudaMemsetAsync(exceed, 0, sizeof(int) * (size_t)(nint + 2), stream));
    if (M <= 0 || nint <= 0) return;
    if (nint <= kFewIntervals) {
        artifact_limits<<<(unsigned)ceil_div(M, 32), 256, 0, stream>>>(norms, M, nint, threshold, nullptr, exceed);
        MS3_LAUNCH_CHECK();
        return;
    }
    DevBuf limits(sizeof(double) * (size_t)M, stream);
    artifact_limits<<<(unsigned)ceil_div(M, 32), 256, 0, stream>>>(norms, M, nint, threshold, limits.as<double>(),
                                                                  nullptr);
    MS3_LAUNCH_CHECK();
    const int64_t blocks = std::min<int64_t>(ceil_div(M * nint, 256), (int64_t)sm_count() * 16);
    artifact_flags<<<(unsigned)blocks, 256, 0, stream>>>(norms, M, nint, limits.as<double>(), exceed);
    MS3_LAUNCH_CHECK();
}

void artifact_write_device(const float* X, int64_t M, int64_t rows, int64_t t0, int64_t I, int64_t nint,
                           const int* exceed, float* out, cudaStream_t stream) {
    if (M <= 0 || rows <= 0) return;
    if (I < kShortInterval && I * M < kShortInterval) {
        const int64_t flat = std::min<int64_t>(ceil_div(M * rows, 256), (int64_t)sm_count() * 32);
        artifact_write_flat<<<(unsigned)flat, 256, 0, stream>>>(X, M, rows, I, nint, exceed, out, t0);
        MS3_LAUNCH_CHECK();
        return;
    }
    const int64_t stretches = ceil_div(std::min(I, rows) * M, kStretch);  // of one interval
    const int64_t total = ((t0 + rows - 1) / I - t0 / I + 1) * stretches;
    const int64_t blocks = std::min<int64_t>(total, (int64_t)sm_count() * 8);
    artifact_write<<<(unsigned)blocks, 256, 0, stream>>>(X, M, rows, I, nint, exceed, out, t0, stretches, total);
    MS3_LAUNCH_CHECK();
}

int64_t artifact_kept(const int* exceed, int64_t nint, int64_t I, cudaStream_t stream) {
    // timepoints kept, for the reference's "Using x% of all timepoints" line
    std::vector<int> h((size_t)(nint + 2));
    MS3_CUDA(cudaMemcpyAsync(h.data(), exceed, sizeof(int) * (size_t)(nint + 2), cudaMemcpyDeviceToHost, stream));
    MS3_CUDA(cudaStreamSynchronize(stream));
    int64_t kept = 0;
    for (int64_t i = 0; i < nint; i++)
        if (!h[(size_t)i] && !h[(size_t)i + 1] && !(i >= 1 && h[(size_t)i - 1])) kept += I;
    return kept;
}

}  // namespace ms3gpu
