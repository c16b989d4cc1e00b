// ms3.whiten on the GPU.
//
// Reference: packages/ms3/p_whiten.cpp:45-206 and packages/ms3/pca.cpp.
//   pass 1   XXt = sum_t x_t x_t^T / (N-1)            (p_whiten.cpp:64-118)
//   matrix   W = whitening_matrix_from_XXt(XXt)        (pca.cpp:635-651)
//   pass 2   y_t = W^T x_t, rounded to multiples of 1e-4, optional int16
//                                                     (p_whiten.cpp:153-206)
//
// Kernels:
//   cov_partial / cov_reduce   channel covariance: 64x64 channel tiles of the
//       upper triangle x time slices.  Products are summed in FP32 over 32
//       timepoints (round-to-nearest FMA, unbiased) and those sums in FP64,
//       so the result agrees with the reference's double sum of float
//       products to ~1e-10 relative.  Partial tiles are reduced in a fixed
//       order: repeat runs are bit-identical.
//   cov_partial_small   the same for up to 32 channels, by 4 x 4 blocks on and above
//       the diagonal.
//   pca_reg       the reference's power iteration, FP64, the working matrix in
//       the registers of one CTA or one cluster of 16 (up to 512 channels)
//   pca_cluster   the same for more channels, one thread-block
//       cluster: the working matrix XXtw is split by rows across the CTAs'
//       shared memory (global memory beyond what fits); each matvec result
//       is broadcast to every CTA through distributed shared memory, one
//       cluster barrier per matvec.  Deflation (I-cc')X(I-cc') is applied as
//       the equivalent symmetric rank-2 update.
//   w_assemble    W = (C D) C^T in the reference's exact summation order.
//   apply_gemm    y = W^T x with W rounded to float, FP32 FMA accumulation,
//       1e-4 rounding in FP64 in the epilogue (bit-exact rounding rule).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>

#include "common.cuh"
#include "div_by.cuh"
#include "ms3gpu.h"
#include "tc_sm100.cuh"
#include "whiten.h"

namespace cg = cooperative_groups;

namespace ms3gpu {

namespace {

// ------------------------------------------------------------ covariance

constexpr int kCT = 64;   // channel tile
constexpr int kTT = 32;  // timepoints summed in FP32 before the FP64 add (slice granularity)
constexpr int kTG = 32;   // timepoints per shared-memory stage of cov_partial

__global__ void __launch_bounds__(256) cov_partial(const float* __restrict__ X, int64_t M, int64_t ld, int64_t r0,
                                                   int64_t N,
                                                   int nb, int64_t tslice, double* __restrict__ partials) {
    __shared__ __align__(16) float As[kTG][kCT];
    __shared__ __align__(16) float Bs[kTG][kCT];
    const int pair = blockIdx.x;
    const int npairs = gridDim.x;
    int bi = 0, rem = pair;
    while (rem >= nb - bi) { rem -= nb - bi; bi++; }
    const int bj = bi + rem;
    const int64_t t_begin = r0 + (int64_t)blockIdx.y * tslice;
    const int64_t t_end = min(N, t_begin + tslice);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double accd[4][4];
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            accd[i][j] = 0.0;
            acc[i][j] = 0.f;
        }

    for (int64_t t0 = t_begin; t0 < t_end; t0 += kTG) {
        for (int e = threadIdx.x; e < kTG * kCT; e += blockDim.x) {
            const int tt = e / kCT, c = e % kCT;
            const int64_t t = t0 + tt;
            const int64_t ma = (int64_t)bi * kCT + c, mb = (int64_t)bj * kCT + c;
            const bool tv = t < t_end;
            As[tt][c] = (tv && ma < M) ? X[t * ld + ma] : 0.f;
            Bs[tt][c] = (tv && mb < M) ? X[t * ld + mb] : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int tt = 0; tt < kTG; tt++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[tt][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[tt][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        // flush the FP32 run every kTT timepoints of the slice
        if (((t0 - t_begin + kTG) % kTT) == 0 || t0 + kTG >= t_end) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    accd[i][j] += (double)acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        __syncthreads();
    }
    double* dst = partials + ((size_t)blockIdx.y * npairs + pair) * (kCT * kCT);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) dst[(ty * 4 + i) * kCT + tx * 4 + j] = accd[i][j];
}

// cov_partial8: the same partial tiles as cov_partial with 8 x 8 register
// micro-tiles (64 threads per 64 x 64 tile), a 3-deep cp.async ring of
// 16-timepoint stages, and packed FP32 FMAs (fma.rn.f32x2: two independent
// round-to-nearest FMAs per instruction, the same values as two fmaf calls),
// which halve the issue slots of the inner product.  FP32 runs of kTT
// timepoints are flushed to FP64, as in cov_partial, so both kernels produce
// the same FP32 partial sums.  Needs M % 4 == 0, ld % 4 == 0 and a 16-byte aligned X.
constexpr int kTS = 16;     // timepoints per stage
constexpr int kStages8 = 3;

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
    const int n = valid ? 16 : 0;  // src-size 0: zero fill
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// (a, a) as a packed FP32 pair
__device__ __forceinline__ uint64_t dup_f32x2(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
// d = a * b + d on both halves of packed FP32 pairs
__device__ __forceinline__ void fma_f32x2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__global__ void __launch_bounds__(64) cov_partial8(const float* __restrict__ X, int64_t M, int64_t ld, int64_t r0,
                                                   int64_t N,
                                                   int nb, int64_t tslice, double* __restrict__ partials) {
    __shared__ __align__(16) float As[kStages8][kTS][kCT];
    __shared__ __align__(16) float Bs[kStages8][kTS][kCT];
    const int pair = blockIdx.x;
    const int npairs = gridDim.x;
    int bi = 0, rem = pair;
    while (rem >= nb - bi) { rem -= nb - bi; bi++; }
    const int bj = bi + rem;
    const bool diag = (bi == bj);
    const int64_t t_begin = r0 + (int64_t)blockIdx.y * tslice;
    const int64_t t_end = min(N, t_begin + tslice);
    const int nst = (int)((t_end - t_begin + kTS - 1) / kTS);
    const int tid = threadIdx.x;
    const int tx = tid & 7, ty = tid >> 3;

    // each thread copies 4 float4 of A (and of B): stage rows tt = tid/16 + 4k, 16-byte column tid%16
    auto issue = [&](int st, int buf) {
        const int64_t tb = t_begin + (int64_t)st * kTS;
        const int c4 = (tid & 15) * 4;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int tt = (tid >> 4) + 4 * k;
            const int64_t t = tb + tt;
            const int64_t ca = (int64_t)bi * kCT + c4, cb = (int64_t)bj * kCT + c4;
            const bool tv = t < t_end;
            cp_async16(&As[buf][tt][c4], X + (tv && ca < M ? t * ld + ca : 0), tv && ca < M);
            if (!diag) cp_async16(&Bs[buf][tt][c4], X + (tv && cb < M ? t * ld + cb : 0), tv && cb < M);
        }
    };

    uint64_t acc[8][4];  // packed pairs: columns (2j, 2j + 1) of row i
    double accd[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll
        for (int j = 0; j < 8; j++) accd[i][j] = 0.0;
    }
#pragma unroll
    for (int p = 0; p < kStages8 - 1; p++) {
        if (p < nst) issue(p, p);
        cp_async_commit();
    }
    for (int st = 0; st < nst; st++) {
        const int buf = st % kStages8;
        if (st + kStages8 - 1 < nst) issue(st + kStages8 - 1, (st + kStages8 - 1) % kStages8);
        cp_async_commit();
        cp_async_wait<kStages8 - 1>();
        __syncthreads();
        const float(*A)[kCT] = As[buf];
        const float(*B)[kCT] = diag ? As[buf] : Bs[buf];
#pragma unroll
        for (int tt = 0; tt < kTS; tt++) {
            const float4 a0 = *reinterpret_cast<const float4*>(&A[tt][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&A[tt][32 + ty * 4]);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&B[tt][tx * 4]);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&B[tt][32 + tx * 4]);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint64_t ai = dup_f32x2(av[i]);
#pragma unroll
                for (int j = 0; j < 4; j++) fma_f32x2(acc[i][j], ai, bv[j]);
            }
        }
        __syncthreads();
        if ((((st + 1) * kTS) % kTT) == 0 || st + 1 == nst) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    accd[i][2 * j] += (double)__uint_as_float((uint32_t)acc[i][j]);
                    accd[i][2 * j + 1] += (double)__uint_as_float((uint32_t)(acc[i][j] >> 32));
                    acc[i][j] = 0ull;
                }
        }
    }
    double* dst = partials + ((size_t)blockIdx.y * npairs + pair) * (kCT * kCT);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = (i < 4) ? ty * 4 + i : 32 + ty * 4 + (i - 4);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int c = (j < 4) ? tx * 4 + j : 32 + tx * 4 + (j - 4);
            dst[r * kCT + c] = accd[i][j];
        }
    }
}

// cov_partial_small: the same partial sums for up to 32 channels, whose 64 x 64 tile is
// three quarters empty and the rest symmetric: one thread per 4 x 4 block on or above the
// diagonal of the M x M corner (36 at 32 channels), stages of kTT timepoints, only those
// elements written.  32 channels x 1.8M: 333 us with cov_partial8, now 115; 16 x 900k: 176 and 35.
constexpr int kSmallC = 32;
template <int THREADS>
__global__ void __launch_bounds__(THREADS) cov_partial_small(const float* __restrict__ X, int M, int64_t ld,
                                                             int64_t r0, int64_t N, int64_t tslice,
                                                             double* __restrict__ partials) {
    __shared__ __align__(16) float As[kStages8][kTT][kSmallC];
    const int tid = threadIdx.x;
    const int nq = M / 4;  // channel quads
    const int64_t t_begin = r0 + (int64_t)blockIdx.x * tslice;
    const int64_t t_end = min(N, t_begin + tslice);
    const int nst = (int)((t_end - t_begin + kTT - 1) / kTT);
    int bi = 0, rem = tid;
    while (bi < nq && rem >= nq - bi) { rem -= nq - bi; bi++; }
    const bool active = bi < nq;
    const int bj = bi + rem;
    auto issue = [&](int st, int buf) {
        const int q = tid & 7;
        if (q < nq) {
#pragma unroll
            for (int tt = tid >> 3; tt < kTT; tt += THREADS / 8) {
                const int64_t t = t_begin + (int64_t)st * kTT + tt;
                const bool in = t < t_end;
                cp_async16(&As[buf][tt][4 * q], X + (in ? t * ld + 4 * q : 0), in);
            }
        }
    };
    uint64_t acc[4][2];  // packed pairs: columns (2j, 2j + 1) of row i
    double accd[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) accd[i][j] = 0.0;
#pragma unroll
    for (int p = 0; p < kStages8 - 1; p++) {
        if (p < nst) issue(p, p);
        cp_async_commit();
    }
    for (int st = 0; st < nst; st++) {
        const int buf = st % kStages8;
        if (st + kStages8 - 1 < nst) issue(st + kStages8 - 1, (st + kStages8 - 1) % kStages8);
        cp_async_commit();
        cp_async_wait<kStages8 - 1>();
        __syncthreads();
        if (active) {
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll
            for (int tt = 0; tt < kTT; tt++) {
                const float4 a = *reinterpret_cast<const float4*>(&As[buf][tt][4 * bi]);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&As[buf][tt][4 * bj]);
                const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint64_t ai = dup_f32x2(av[i]);
                    fma_f32x2(acc[i][0], ai, b.x);
                    fma_f32x2(acc[i][1], ai, b.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    accd[i][2 * j] += (double)__uint_as_float((uint32_t)acc[i][j]);
                    accd[i][2 * j + 1] += (double)__uint_as_float((uint32_t)(acc[i][j] >> 32));
                }
        }
        __syncthreads();
    }
    if (!active) return;
    double* dst = partials + (size_t)blockIdx.x * (kCT * kCT);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) dst[(4 * bi + i) * kCT + 4 * bj + j] = accd[i][j];
}

// XXt from the slices' partial tiles, added in slice order: a block takes 32 elements
// of a tile row; its warps keep kRedStages groups of kRedTile slices on their way to
// shared memory, the first warp adds them.  (A thread per element waited for its own
// loads: 174 us for 1172 slices of 32 channels, now 16 us.)  Elements below the
// diagonal mirror.
constexpr int kRedTile = 32, kRedStages = 4;
__global__ void __launch_bounds__(256) cov_reduce(const double* __restrict__ partials, int S, int npairs, int nb,
                                                  int64_t M, int64_t N, double* __restrict__ XXt) {
    __shared__ __align__(16) double tile[kRedStages][kRedTile][32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t idx = (int64_t)blockIdx.x * 32 + l;
    const int pair = (int)(idx / (kCT * kCT));
    const int e = (int)(idx % (kCT * kCT));
    const int r = e / kCT, c = e % kCT;
    int bi = 0, rem = pair;
    while (rem >= nb - bi) { rem -= nb - bi; bi++; }
    const int bj = bi + rem;
    const int64_t i = (int64_t)bi * kCT + r, j = (int64_t)bj * kCT + c;
    const bool wanted = i < M && j < M && i <= j;
    if (!__syncthreads_or(wanted)) return;
    const double* src = partials + (size_t)pair * (kCT * kCT) + e;
    const size_t step = (size_t)npairs * (kCT * kCT);
    auto issue = [&](int g) {  // slices g kRedTile ..: four per warp
#pragma unroll
        for (int h = 0; h < kRedTile / 8; h++) {
            const int k = g * kRedTile + w + 8 * h;
            if (wanted && k < S) {
                const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(&tile[g % kRedStages][w + 8 * h][l]));
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src + k * step) : "memory");
            }
        }
        cp_async_commit();
    };
    const int groups = (S + kRedTile - 1) / kRedTile;
#pragma unroll
    for (int g = 0; g < kRedStages - 1; g++) issue(g);
    double s = 0.0;
    for (int g = 0; g < groups; g++) {
        cp_async_wait<kRedStages - 2>();
        __syncthreads();  // the group is here, and the one before has been added
        issue(g + kRedStages - 1);
        if (w == 0) {
            const int n = min(kRedTile, S - g * kRedTile);
            const double(*t)[32] = tile[g % kRedStages];
#pragma unroll 8
            for (int k = 0; k < n; k++) s += t[k][l];
        }
    }
    if (w || !wanted) return;
    if (N > 1) s /= (double)(N - 1);
    XXt[i + M * j] = s;
    XXt[j + M * i] = s;
}

// ------------------------------------------------------------ power iteration

constexpr int kPcaThreads = 512;

// Sum over the block of per-thread values; every thread returns the total.
// Fixed reduction tree: identical results in every CTA of the cluster.
__device__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    const int nw = blockDim.x >> 5;
    for (int i = 0; i < nw; i++) t += red[i];
    return t;
}

// Sum over n < M of f(n), formed by one warp: lane l adds f(l), f(l + 32),
// ... in order, then a 32-lane XOR tree.  Addition is commutative, so every
// lane ends with the same bits; both power-iteration kernels form their norms
// and dot products this way, which keeps their results identical.  The
// dependent chain is M/32 adds plus five shuffles (the previous per-chunk
// trees cost five shuffles per 32 elements).
template <class F>
__device__ __forceinline__ double warp_ordered_sum(int M, F f) {
    const int l = threadIdx.x & 31;
    double t = 0.0;
    for (int n = l; n < M; n += 32) t += f(n);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// y = X v for this CTA's rows, written into `dst` of every CTA in the cluster,
// followed by a cluster barrier.
__device__ void cluster_matvec(cg::cluster_group& cluster, const double* __restrict__ X, int RS, int r0,
                               int nr, int M, const double* __restrict__ v, double* dst) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    const int CS = (int)cluster.num_blocks();
    for (int r = w; r < nr; r += nw) {
        const double* row = X + (size_t)r * RS;
        double s = 0.0;
        for (int n = l; n < M; n += 32) s += row[n] * v[n];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        for (int d = l; d < CS; d += 32) {
            double* remote = cluster.map_shared_rank(dst, d);
            remote[r0 + r] = s;
        }
    }
    cluster.sync();
}

// pca_from_XXt (pca.cpp:172-195) for all M components.
// Xg: optional global copy of the rows (when they do not fit shared memory).
__global__ void __launch_bounds__(kPcaThreads) pca_cluster(const double* __restrict__ XXt, int M, int R,
                                                            int num_iter, int rows_in_smem, double* Xg,
                                                            double* __restrict__ comps,
                                                            double* __restrict__ sigma) {
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    extern __shared__ double sm[];
    const int RS = M + 1;  // padded row stride
    double* vb[2];
    vb[0] = sm;
    vb[1] = vb[0] + M;
    double* vinit = vb[1] + M;
    double* red = vinit + M;
    double* X = rows_in_smem ? (red + 32) : (Xg + (size_t)rank * R * RS);
    const int r0 = rank * R;
    const int nr = max(0, min(R, M - r0));

    for (int idx = threadIdx.x; idx < nr * M; idx += blockDim.x) {
        const int r = idx % nr, n = idx / nr;
        X[(size_t)r * RS + n] = XXt[(size_t)(r0 + r) + (size_t)M * n];
    }
    // start vector sin(i+1), normalised (pca.cpp:546-549, 457-466)
    for (int n = threadIdx.x; n < M; n += blockDim.x) vinit[n] = sin((double)(n + 1));
    __syncthreads();
    {
        double part = 0.0;
        for (int n = threadIdx.x; n < M; n += blockDim.x) part += vinit[n] * vinit[n];
        const double nrm = sqrt(block_sum(part, red));
        __syncthreads();
        if (nrm != 0.0)
            for (int n = threadIdx.x; n < M; n += blockDim.x) vinit[n] = vinit[n] / nrm;
    }
    cluster.sync();

    for (int k = 0; k < M; k++) {
        int cur = 0;
        for (int n = threadIdx.x; n < M; n += blockDim.x) vb[0][n] = vinit[n];
        __syncthreads();
        double sig = 0.0;
        for (int it = 0; it < num_iter; it++) {
            const int nxt = cur ^ 1;
            cluster_matvec(cluster, X, RS, r0, nr, M, vb[cur], vb[nxt]);
            const double* y = vb[nxt];
            sig = sqrt(warp_ordered_sum(M, [&](int n) { return y[n] * y[n]; }));
            __syncthreads();
            if (sig != 0.0)
                for (int n = threadIdx.x; n < M; n += blockDim.x) vb[nxt][n] = vb[nxt][n] / sig;
            __syncthreads();
            cur = nxt;
        }
        const double* v = vb[cur];
        if (rank == 0) {
            for (int n = threadIdx.x; n < M; n += blockDim.x) comps[(size_t)n + (size_t)M * k] = v[n];
            if (threadIdx.x == 0) sigma[k] = sig;
        }
        // deflation: X <- X - v u' - u v' + (v'u) v v',  u = X v
        double* u = vb[cur ^ 1];
        cluster_matvec(cluster, X, RS, r0, nr, M, v, u);
        const double alpha = warp_ordered_sum(M, [&](int n) { return v[n] * u[n]; });
        for (int idx = threadIdx.x; idx < nr * M; idx += blockDim.x) {
            const int r = idx / M, n = idx % M;
            const int m = r0 + r;
            const double s = __dadd_rn(__dmul_rn(v[m], u[n]), __dmul_rn(u[m], v[n]));
            const double x = __dsub_rn(X[(size_t)r * RS + n], s);
            X[(size_t)r * RS + n] = __dadd_rn(x, __dmul_rn(alpha, __dmul_rn(v[m], v[n])));
        }
        cluster.sync();
    }
}

// The same power iteration with the working matrix in registers: lane l of a
// warp holds its RPW rows at columns l + 32 j (j < CPL) and the current vector
// at the same columns.  Every sum is formed in the order pca_cluster forms it
// (per-lane column sums, then the XOR shuffle tree), and the quotient y / sigma
// is the correctly rounded one (div_by.cuh), so components, sigma and W have
// the same bits.
//
// What bounds it: the M * 11 matvec steps depend on one another, so a step's
// latency is the time (at 384 channels one step is 147,456 FP64 FMAs, 0.15 us of
// the FP64 pipes of 16 SMs, while DFMA takes 9 cycles, a shuffle level about 30,
// sqrt 85 and an 8-byte exchange between two SMs 311).  A step is: read the
// exchanged vector (CPL values per lane), norm (FMA chain, shuffle tree, sqrt),
// v = y / sigma in registers (one reciprocal, four FMAs per value), the row
// sums, the trees of all the warp's rows merged (each level halves the rows a
// lane holds, so RPW rows cost about as many shuffles as one), and the
// exchange.  Every warp forms norm and quotient itself, which costs less than
// handing them round.
//
// CS = 1 (M <= 128): one CTA; rows meet in shared memory, one block barrier a
// step.  344 us at 32 channels and 1468 us at 128 with the 8-CTA cluster that this
// replaces; now 139 us and 1097 us.
// CS = 16 (M > 128): sixteen CTAs of NW warps; row m belongs to CTA m % CS, so
// every CTA owns rows.  A CTA gathers its rows in shared memory (the step's one
// block barrier) and each warp stores them to its share of the sixteen CTAs with
// st.async, a CTA's rows contiguous in one warp store, counted in bytes on the
// receiver's mbarrier.  The exchange is bound by those stores: 16 x 24 rows take
// 596 cycles that way and 880 as 8- or 16-byte stores scattered over the CTAs
// (1130-1160 as bulk copies).  Since a CTA sends step s + 1 after all its warps
// have read step s, having received all M rows of step s + 1 means every CTA is
// done with step s: buffer s & 1 is free for step s + 2, and no mbarrier gets two
// phases ahead of one of its readers.  Waits spin first (an exchange takes well
// under a microsecond, less than a suspended wait takes to wake) and are bounded
// (error flag g_pca_timeout).  Eight CTAs of 16 warps and 3 rows, with division
// and vector handed round through shared memory, took 8230 us at 384 channels and
// 3023 us at 200; this takes 4107 us and 1624 us.
__device__ int g_pca_timeout;  // set when an exchange wait gave up (checked by the host)

__device__ __noinline__ double plain_quotient(double y, double b) { return y / b; }

// Whether v[j] / b may use quotient_in_range for every element with 32 j < left
// (the others are zero and stay so), as far as v decides it; called by all lanes
// of a warp.  +0 may: a silent channel's entry is zero in every vector (384 channels, one
// silent: 9520 us with ordinary divisions, now 4190).
template <int N>
__device__ __forceinline__ bool quotients_in_range(const double (&v)[N], int left) {
    bool fast = true;
#pragma unroll
    for (int j = 0; j < N; j++)
        fast &= quotient_range(v[j]) || (__double2hiint(v[j]) | __double2loint(v[j])) == 0 || 32 * j >= left;
    return __all_sync(0xffffffffu, fast);
}

// v[j] = v[j] / b.  Up to two elements the ordinary division is the shorter
// chain (one: 112 cycles against 196).
template <int N>
__device__ __forceinline__ void divide_by(double (&v)[N], double b, int left, bool in_range) {
    if (N > 2) {
        const Reciprocal c = reciprocal_of(b);
        if (in_range && c.in_range) {
#pragma unroll
            for (int j = 0; j < N; j++) v[j] = quotient_in_range(v[j], b, c);
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < N; j++)
        if (32 * j < left) v[j] = N > 2 ? plain_quotient(v[j], b) : v[j] / b;
}

// element J0 + i (i < K) of lane `lane`'s v
template <int J0, int K, int N>
__device__ __forceinline__ double shfl_element(const double (&v)[N], int i, int lane) {
    double x = v[J0];
#pragma unroll
    for (int k = 1; k < K; k++)
        if (i == k) x = v[J0 + k];
    return __shfl_sync(0xffffffffu, x, lane);
}

// out[r] = element m of the vector held as v[j] on lane l (element l + 32 j),
// for the row slots m = r G + base, base < G
template <int G, int R, int RPW, int N>
__device__ __forceinline__ void row_elements_from(const double (&v)[N], int base, double (&out)[RPW]) {
    if constexpr (R < RPW) {
        const int m = R * G + base;
        out[R] = shfl_element<R * G / 32, (G >= 32 ? G / 32 : 1)>(v, G >= 32 ? base >> 5 : 0, m & 31);
        row_elements_from<G, R + 1>(v, base, out);
    }
}
template <int G, int RPW, int N>
__device__ __forceinline__ void row_elements(const double (&v)[N], int base, double (&out)[RPW]) {
    row_elements_from<G, 0>(v, base, out);
}

__host__ __device__ constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// GIVE_UP (testing): the second warp of each cluster's first CTA takes its wait of step
// give_up_step as run out.
template <int CS, int NW, int CPL, bool GIVE_UP = false>
__global__ void __launch_bounds__(NW * 32, 1) pca_reg(const double* __restrict__ XXt_all, int M, int num_iter,
                                                      double* __restrict__ comps_all,
                                                      double* __restrict__ sigma_all, int give_up_step) {
    constexpr int G = CS * NW;             // rows per row slot of the whole cluster
    constexpr int RPW = 32 * CPL / G;      // row slots of a warp
    static_assert(RPW * G == 32 * CPL, "the rows fill the column range");
    constexpr int RP2 = pow2_at_least(RPW);
    static_assert(RP2 <= 32, "rows of a warp's merged tree");
    constexpr int S = 32 / RP2;            // lanes that end up with the same row's sum
    constexpr int kMaxM = 32 * CPL;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = CS > 1 ? (int)cluster.block_rank() : 0;
    const int64_t mat = blockIdx.x / CS;   // one cluster per matrix
    const double* XXt = XXt_all + mat * M * M;
    double* comps = comps_all + mat * M * M;
    double* sigma = sigma_all + mat * M;
    int* err = &g_pca_timeout;
    // matvec results; entries beyond M stay zero.  CS > 1: row m at (m % CS) * RS
    // + m / CS, so that a CTA's rows are contiguous; RS odd keeps the strided
    // reads free of bank conflicts.
    constexpr int R = NW * RPW;  // rows of a CTA
    constexpr int RS = R | 1;
    static_assert(CS == 1 || R <= 32, "a CTA's rows in one warp store");
    constexpr int kYLen = CS > 1 ? CS * RS : kMaxM;
    __shared__ double ybuf[2][kYLen];
    __shared__ double stage[2][CS > 1 ? R : 1];  // CS > 1: this CTA's rows on their way out
    __shared__ double vinit[kMaxM];
    __shared__ __align__(8) uint64_t ybar[2];  // CS > 1: bytes of ybuf[b] received in the current step
    __shared__ int gave_up[2];                 // CS > 1: a warp gave up in the step before (by step parity)
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int base = w * CS + rank;  // row of slot 0
    const uint32_t step_bytes = (uint32_t)M * 8u;

    double A[RPW][CPL];
#pragma unroll
    for (int r = 0; r < RPW; r++)
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const int m = r * G + base, n = l + 32 * j;
            A[r][j] = (m < M && n < M) ? XXt[(size_t)m + (size_t)M * n] : 0.0;
        }
    for (int n = threadIdx.x; n < 2 * kYLen; n += NW * 32) (&ybuf[0][0])[n] = 0.0;
    if (CS > 1 && threadIdx.x == 0) {
        gave_up[0] = gave_up[1] = 0;
        tc::mbar_init(&ybar[0], 1);
        tc::mbar_init(&ybar[1], 1);
        tc::fence_mbar_init();
    }
    double v[CPL];
    // start vector sin(i+1), normalised (pca.cpp:546-549, 457-466); squares
    // summed per 32 elements (tree), then chunk after chunk
    {
        double nrm2 = 0.0;
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const int n = l + 32 * j;
            v[j] = n < M ? sin((double)(n + 1)) : 0.0;
            double p = __dmul_rn(v[j], v[j]);
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            nrm2 += p;
        }
        const double nrm = sqrt(nrm2);
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            if (nrm != 0.0 && l + 32 * j < M) v[j] = v[j] / nrm;
            if (w == 0) vinit[l + 32 * j] = v[j];
        }
    }
    if (CS > 1 && threadIdx.x == 0) {
        tc::mbar_expect_tx(&ybar[0], step_bytes);  // steps 0 and 1
        tc::mbar_expect_tx(&ybar[1], step_bytes);
    }
    // every CTA's barriers are initialised and armed before any store reaches them
    if (CS > 1)
        cluster.sync();
    else
        __syncthreads();

    // the row whose sum this lane holds after the merged tree: bit 4 of the lane
    // selects the upper half of the slots, bit 3 the upper half of those, ...
    int slot = 0;
#pragma unroll
    for (int o = 16, h = RP2 / 2; h > 0; o >>= 1, h >>= 1) slot += (l & o) ? h : 0;
    const bool holds = slot < RPW && slot * G + base < M && l % S == 0;
    // CS > 1: warp w stores the CTA's rows to the CTAs w + NW i, lane q row q CS + rank
    constexpr int kSends = CS > 1 ? CS / NW : 1;
    uint32_t rbuf[kSends], rbar[kSends];
    const bool sends = l < R && l * CS + rank < M;
    if (CS > 1) {
#pragma unroll
        for (int i = 0; i < kSends; i++) {
            const uint32_t d = (uint32_t)(w + NW * i);
            rbuf[i] = tc::mapa_shared(tc::smem_u32(&ybuf[0][0]), d) + (uint32_t)(rank * RS + l) * 8u;
            rbar[i] = tc::mapa_shared(tc::smem_u32(&ybar[0]), d);
        }
    }
    // where this lane finds element l + 32 j of a vector in ybuf
    const int y0 = CS > 1 ? (l % CS) * RS + l / CS : l;
    constexpr int kYStep = CS > 1 ? 32 / CS : 32;

    // ybuf[step & 1] = A v in every CTA; returns once it is complete.  A warp whose wait
    // gives up leaves the loop, says so in gave_up and takes part in one more block barrier,
    // the next step's; after that barrier the CTA's other warps see it and leave too, so
    // that none stands in the cluster barrier while another waits for it in a block barrier.
    // Two words by step parity: a warp that gives up in step s writes the word of s + 1; the
    // next to write that word has passed the barrier of s + 2, which every warp reaches
    // after its read in s + 1.  (A vote in the block barrier, __syncthreads_and, cost 180 ns
    // a step, and so did a return of its own for a warp that sees the word: 4136 and 4903 us
    // at 384 channels.)
    auto matvec = [&](int step) -> bool {
        const int b = step & 1;
        double s[RP2];
#pragma unroll
        for (int r = 0; r < RP2; r++) s[r] = 0.0;
#pragma unroll
        for (int j = 0; j < CPL; j++)
#pragma unroll
            for (int r = 0; r < RPW; r++) s[r] = __fma_rn(A[r][j], v[j], s[r]);
        int o = 16;
#pragma unroll
        for (int h = RP2 / 2; h > 0; h >>= 1, o >>= 1) {
            const bool up = (l & o) != 0;
#pragma unroll
            for (int i = 0; i < h; i++) {
                const double keep = up ? s[i + h] : s[i], give = up ? s[i] : s[i + h];
                s[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
#pragma unroll
        for (int q = S / 2; q > 0; q >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], q);
        if (CS == 1) {
            if (holds) ybuf[b][slot * G + base] = s[0];
            __syncthreads();
            return true;
        }
        if (holds) stage[b][slot * NW + w] = s[0];
        __syncthreads();
        const int leave = *const_cast<volatile int*>(&gave_up[b]);
        if (sends) {
            const uint64_t x = (uint64_t)__double_as_longlong(stage[b][l]);
#pragma unroll
            for (int i = 0; i < kSends; i++)
                tc::st_async_b64(rbuf[i] + (uint32_t)(b * kYLen * 8), x, rbar[i] + (uint32_t)(b * 8));
        }
        bool ok = __all_sync(0xffffffffu, !leave && tc::mbar_wait_cluster_spin(&ybar[b], (uint32_t)((step >> 1) & 1), err));
        if (GIVE_UP && step == give_up_step && rank == 0 && w == 1) ok = false;  // as if it had run out
        // re-arm for step + 2: its stores arrive only after this CTA has sent step + 1
        if (ok && threadIdx.x == 0) tc::mbar_expect_tx(&ybar[b], step_bytes);
        return ok;
    };

    int step = 0;  // matvec count, at most 512 * 11 (the same sequence in every warp)
    bool ok = true;
    for (int k = 0; k < M && ok; k++) {
#pragma unroll
        for (int j = 0; j < CPL; j++) v[j] = vinit[l + 32 * j];
        double sig = 0.0;
        for (int it = 0; it < num_iter && ok; it++) {
            ok = matvec(step);
            if (!ok) break;
            const double* y = ybuf[step & 1];
            step++;
            double t = 0.0;
#pragma unroll
            for (int j = 0; j < CPL; j++) {
                v[j] = y[y0 + kYStep * j];
                t = __fma_rn(v[j], v[j], t);
            }
            const bool in_range = CPL > 2 && quotients_in_range<CPL>(v, M - l);
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            sig = sqrt(t);
            if (sig != 0.0) divide_by<CPL>(v, sig, M - l, in_range);
        }
        if (!ok) break;
        if (rank == 0 && w == 0) {
#pragma unroll
            for (int j = 0; j < CPL; j++)
                if (l + 32 * j < M) comps[(size_t)(l + 32 * j) + (size_t)M * k] = v[j];
            if (l == 0) sigma[k] = sig;
        }
        // deflation: X <- X - v u' - u v' + (v'u) v v',  u = X v
        ok = matvec(step);
        if (!ok) break;
        const double* u = ybuf[step & 1];
        step++;
        double uj[CPL];
        double alpha = 0.0;
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            uj[j] = u[y0 + kYStep * j];
            alpha = __fma_rn(v[j], uj[j], alpha);
        }
        for (int o = 16; o > 0; o >>= 1) alpha += __shfl_xor_sync(0xffffffffu, alpha, o);
        double vm_of[RPW];
        row_elements<G, RPW>(v, base, vm_of);
#pragma unroll
        for (int r = 0; r < RPW; r++) {
            const double vm = vm_of[r], um = u[CS > 1 ? rank * RS + r * NW + w : r * G + base];
#pragma unroll
            for (int j = 0; j < CPL; j++) {
                if (l + 32 * j < M) {
                    const double sdef = __dadd_rn(__dmul_rn(vm, uj[j]), __dmul_rn(um, v[j]));
                    const double x = __dsub_rn(A[r][j], sdef);
                    A[r][j] = __dadd_rn(x, __dmul_rn(alpha, __dmul_rn(vm, v[j])));
                }
            }
        }
    }
    // No CTA leaves while a peer may still store into its shared memory.  A CTA that has
    // received every step has nothing more on its way; one that gave up lets the stores
    // land that its peers issued before they came here.
    if (CS > 1) {
        // a warp that saw the word has passed the barrier that the others wait for here
        const bool saw = !ok && *const_cast<volatile int*>(&gave_up[step & 1]);
        if (!saw) {
            if (!ok && l == 0) {
                gave_up[(step & 1) ^ 1] = 1;
                atomicExch(err, 1);
            }
            __syncthreads();
        }
        cluster.sync();
        if (gave_up[0] || gave_up[1]) {
            const unsigned long long t0 = tc::globaltimer_ns();
            while (tc::globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
        }
    }
}

// W = (C D) C^T, D = diag(1/sqrt(sigma)) (0 where sigma == 0), in the
// reference's order: tmp(m,l) = C(m,l) d_l (mult_AB with a diagonal,
// pca.cpp:220-243), W(m,n) = sum_l tmp(m,l) C(n,l) (mult_ABtrans, :319-342).
// A 32 x 32 tile of W per block, the l range staged through shared memory 32 at a
// time (tmp formed there once per tile), 2 x 2 sums per thread.  The sums are
// serial in l: one thread per element reading C from L2 spent its time on the
// loads (115 us at 384 channels; now 34 us).  blockIdx.z: the matrix of a batch.
constexpr int kWT = 32;
__global__ void __launch_bounds__(256) w_assemble(const double* __restrict__ C_all,
                                                  const double* __restrict__ sigma_all, int M,
                                                  double* __restrict__ W_all) {
    __shared__ double tmp[kWT][kWT], cn[kWT][kWT];  // [l][m], [l][n]
    __shared__ double dl[2][kWT];                   // d of the l tile in flight
    const double* C = C_all + (size_t)blockIdx.z * M * M;
    const double* sigma = sigma_all + (size_t)blockIdx.z * M;
    double* W = W_all + (size_t)blockIdx.z * M * M;
    const int m0 = blockIdx.x * kWT, n0 = blockIdx.y * kWT;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;  // staging: element x of rows y + 8 i
    const int mi = threadIdx.x & 15, ni = threadIdx.x >> 4;  // sums: m0 + mi + 16 a, n0 + ni + 16 b
    double a[4], c[4];
    auto fetch = [&](int l0) {
        if (y == 0) {
            const double s = l0 + x < M ? sigma[l0 + x] : 0.0;
            dl[(l0 / kWT) & 1][x] = (s != 0.0) ? 1.0 / sqrt(s) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int l = l0 + y + 8 * i;
            a[i] = (l < M && m0 + x < M) ? C[(size_t)(m0 + x) + (size_t)M * l] : 0.0;
            c[i] = (l < M && n0 + x < M) ? C[(size_t)(n0 + x) + (size_t)M * l] : 0.0;
        }
    };
    double acc[2][2] = {};
    fetch(0);
    for (int l0 = 0; l0 < M; l0 += kWT) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            tmp[y + 8 * i][x] = __dmul_rn(a[i], dl[(l0 / kWT) & 1][y + 8 * i]);
            cn[y + 8 * i][x] = c[i];
        }
        __syncthreads();
        if (l0 + kWT < M) fetch(l0 + kWT);
        const int nl = min(kWT, M - l0);
#pragma unroll 8
        for (int l = 0; l < nl; l++) {
            const double t0 = tmp[l][mi], t1 = tmp[l][mi + 16], c0 = cn[l][ni], c1 = cn[l][ni + 16];
            acc[0][0] = __dadd_rn(acc[0][0], __dmul_rn(t0, c0));
            acc[0][1] = __dadd_rn(acc[0][1], __dmul_rn(t0, c1));
            acc[1][0] = __dadd_rn(acc[1][0], __dmul_rn(t1, c0));
            acc[1][1] = __dadd_rn(acc[1][1], __dmul_rn(t1, c1));
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int m = m0 + mi + 16 * i, n = n0 + ni + 16 * j;
            if (m < M && n < M) W[(size_t)m + (size_t)M * n] = acc[i][j];
        }
}

// ------------------------------------------------------------ apply

// Wt[m1][m2] = (float) W[m1*M + m2]  (the element the reference multiplies
// x[m2] with when it accumulates out[m1], p_whiten.cpp:174-183)
__global__ void w_to_float(const double* __restrict__ W, int64_t MM, float* __restrict__ Wt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < MM) Wt[i] = (float)W[i];
}

// quantize(x, 1e-4) = floor(x/1e-4 + 0.5) * 1e-4 in double (p_whiten.cpp:31-41).
// For a float x, x * 1e4 is exact in double (at most 34 significant bits)
// and the quotient x / 0.0001 lies within 0.43 ulp of it (the double 0.0001
// is 1e-4 (1 + 4.8e-17)), so the two are the same double; the division is
// kept as a guard for values within 1e-6 of a rounding boundary.
__device__ __forceinline__ float quantize_1e4(float x) {
    const double xd = (double)x;
    double t = __dadd_rn(__dmul_rn(xd, 10000.0), 0.5);
    double f = floor(t);
    if (t - f < 1e-6 || f + 1.0 - t < 1e-6) {
        t = __dadd_rn(__ddiv_rn(xd, 0.0001), 0.5);
        f = floor(t);
    }
    return (float)__dmul_rn(f, 0.0001);
}

constexpr int kBM = 64, kBN = 64, kBK = 16;

__global__ void __launch_bounds__(256) apply_gemm(const float* __restrict__ X, const float* __restrict__ Wt,
                                                  int64_t M, int64_t N, int64_t ld, double qunit, int round_1e4,
                                                  void* __restrict__ out) {
    __shared__ __align__(16) float Xs[kBK][kBM + 4];
    __shared__ __align__(16) float Ws[kBK][kBN + 4];
    // column blocks of one time tile are adjacent in launch order, so the
    // time tile of X is read from DRAM once and from L2 by the others
    const int64_t ncb = (M + kBN - 1) / kBN;
    const int64_t t0 = ((int64_t)blockIdx.x / ncb) * kBM;
    const int64_t n0 = ((int64_t)blockIdx.x % ncb) * kBN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int64_t k0 = 0; k0 < M; k0 += kBK) {
        for (int e = threadIdx.x; e < kBM * kBK; e += blockDim.x) {
            const int r = e / kBK, kk = e % kBK;
            const int64_t t = t0 + r, k = k0 + kk;
            Xs[kk][r] = (t < N && k < M) ? X[t * ld + k] : 0.f;
            const int64_t n = n0 + r;
            Ws[kk][r] = (n < M && k < M) ? Wt[n * M + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kBK; kk++) {
            const float4 a = *reinterpret_cast<const float4*>(&Xs[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int64_t t = t0 + ty * 4 + i;
        if (t >= N) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int64_t n = n0 + tx * 4 + j;
            if (n >= M) continue;
            const float y = round_1e4 ? quantize_1e4(acc[i][j]) : acc[i][j];
            if (qunit > 0) {
                // scale_for_quantization (p_whiten.cpp:445-451): (int)(y/q + 0.5)
                // stored in a float, then written as int16 by the .mda writer.
                const int32_t iv = x86_double_to_int32(__dadd_rn(__ddiv_rn((double)y, qunit), 0.5));
                static_cast<int16_t*>(out)[t * ld + n] = x86_float_to_int16((float)iv);
            } else {
                static_cast<float*>(out)[t * ld + n] = y;
            }
        }
    }
}

// out[t][j] = X[t][ch[j]] for a channel subset (0-based indices, checked by
// the caller): ms3.compute_whitening_matrix's extract_channels_from_chunk
// (p_whiten.cpp:421-433) applied to a whole device array.  A block takes groups
// of rows small enough for 32-bit index arithmetic: a 64-bit division per element
// bound the flat form (300k rows, 1532 of 1536 channels: 1169 us to gather and 1193
// to scatter; now 690 and 767).
constexpr int kGroupElems = 4096;
__global__ void __launch_bounds__(256) gather_channels(const float* __restrict__ X, int64_t M, int64_t N,
                                                       const int32_t* __restrict__ ch, int M2, int rows,
                                                       float* __restrict__ out) {
    for (int64_t t0 = (int64_t)blockIdx.x * rows; t0 < N; t0 += (int64_t)gridDim.x * rows) {
        const unsigned n = (unsigned)min((int64_t)rows, N - t0) * (unsigned)M2;
        const float* Xg = X + t0 * M;
        float* og = out + t0 * M2;
#pragma unroll 4
        for (unsigned e = threadIdx.x; e < n; e += 256) {
            const unsigned t = e / (unsigned)M2, j = e - t * (unsigned)M2;
            if (MS3_IN_BOUNDS(ch[j], M, 201)) og[e] = Xg[(int64_t)t * M + ch[j]];
        }
    }
}

// out[t][ch[j]] = Y[t][j]: a whitened channel block back into its columns
// (element size 4 for float32 output, 2 for int16).
template <class T>
__global__ void __launch_bounds__(256) scatter_channels(const T* __restrict__ Y, int M2, int64_t N,
                                                        const int32_t* __restrict__ ch, int64_t M, int rows,
                                                        T* __restrict__ out) {
    for (int64_t t0 = (int64_t)blockIdx.x * rows; t0 < N; t0 += (int64_t)gridDim.x * rows) {
        const unsigned n = (unsigned)min((int64_t)rows, N - t0) * (unsigned)M2;
        const T* Yg = Y + t0 * M2;
        T* og = out + t0 * M;
#pragma unroll 4
        for (unsigned e = threadIdx.x; e < n; e += 256) {
            const unsigned t = e / (unsigned)M2, j = e - t * (unsigned)M2;
            if (MS3_IN_BOUNDS(ch[j], M, 202)) og[(int64_t)t * M + ch[j]] = Yg[e];
        }
    }
}

int num_sms() {
    int dev = 0, n = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    MS3_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    return n;
}

}  // namespace

// MS3GPU_COV_KERNEL=fma keeps the FP32-FMA kernel for every shape; =tc uses
// the tensor-core kernel whenever M % 4 == 0 (testing).  By default the
// tensor cores take M >= 128 with M % 4 == 0.
static int cov_kernel_choice() {
    static const int v = [] {
        const char* s = std::getenv("MS3GPU_COV_KERNEL");
        if (s && std::string(s) == "fma") return 1;
        if (s && std::string(s) == "tc") return 2;
        return 0;
    }();
    return v;
}

CovPlan cov_plan(const float* X, int64_t M, int64_t ld) {
    CovPlan p;
    if (ld == 0) ld = M;
    p.M = M;
    p.nb = (int)ceil_div(M, kCT);
    p.npairs = p.nb * (p.nb + 1) / 2;
    p.vec = (M % 4 == 0) && (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(X) & 15) == 0);
    const int choice = cov_kernel_choice();
    p.tc = M > 0 && M % 4 == 0 && choice != 1 && (choice == 2 || M >= 128);
    return p;
}

int64_t cov_tslice(const CovPlan& p, int64_t rows) {
    if (p.tc) return cov_i8_run_length(p.M, rows);
    if (rows <= 0) return kTT;
    const int64_t target = std::max<int64_t>(1, (int64_t)(p.vec ? 8 : 4) * num_sms() / p.npairs);
    const int64_t S = std::min<int64_t>(target, ceil_div(rows, kTT));
    return ceil_div(ceil_div(rows, S), kTT) * kTT;
}

int64_t cov_slices(const CovPlan& p, int64_t rows) {
    if (rows <= 0) return 0;
    return ceil_div(rows, cov_tslice(p, rows));
}

size_t cov_partials_bytes(const CovPlan& p, int64_t slices) {
    if (p.tc) return cov_i8_partials_bytes(p.M, slices);
    return (size_t)slices * p.npairs * kCT * kCT * sizeof(double);
}

void cov_partials(const float* X, int64_t M, int64_t r0, int64_t r1, const CovPlan& p, double* partials,
                  int64_t S, cudaStream_t stream, int64_t ld) {
    const int64_t rows = r1 - r0;
    if (rows <= 0 || S <= 0) return;
    if (p.tc) {  // runs of the plan's length: the slicing the streamed forms use too
        const int64_t R = cov_tslice(p, rows);
        if (ceil_div(rows, R) != S) throw_invalid("covariance: slice count does not match the plan");
        cov_partials_sliced(X, M, r0, r1, p, partials, R, stream, ld);
        return;
    }
    cov_partials_sliced(X, M, r0, r1, p, partials, ceil_div(ceil_div(rows, S), kTT) * kTT, stream, ld);
}

void cov_partials_sliced(const float* X, int64_t M, int64_t r0, int64_t r1, const CovPlan& p, double* partials,
                         int64_t tslice, cudaStream_t stream, int64_t ld) {
    const int64_t rows = r1 - r0;
    if (rows <= 0) return;
    if (ld == 0) ld = M;
    if (tslice <= 0 || tslice % kTT != 0) throw_invalid("covariance slice length must be a multiple of 32");
    if (p.tc) {
        if (ld % 4 == 0 && (reinterpret_cast<uintptr_t>(X + r0 * ld) & 15) == 0) {
            cov_i8_partials(X, M, ld, r0, r1, tslice, partials, stream);
        } else {  // the tensor map needs 16-byte aligned rows: work on an aligned copy
            DevBuf copy(sizeof(float) * (size_t)(rows * M), stream);
            MS3_CUDA(cudaMemcpy2DAsync(copy.get(), sizeof(float) * (size_t)M, X + r0 * ld, sizeof(float) * (size_t)ld,
                                       sizeof(float) * (size_t)M, (size_t)rows, cudaMemcpyDeviceToDevice, stream));
            cov_i8_partials(copy.as<float>(), M, M, 0, rows, tslice, partials, stream);
        }
        return;
    }
    const int64_t S = ceil_div(rows, tslice);
    if (p.vec && M <= kSmallC) {
        if (M <= 28)  // 28 blocks of 4 x 4 at most: one warp
            cov_partial_small<32><<<(unsigned)S, 32, 0, stream>>>(X, (int)M, ld, r0, r1, tslice, partials);
        else
            cov_partial_small<64><<<(unsigned)S, 64, 0, stream>>>(X, (int)M, ld, r0, r1, tslice, partials);
    } else if (p.vec)
        cov_partial8<<<dim3(p.npairs, (unsigned)S), 64, 0, stream>>>(X, M, ld, r0, r1, p.nb, tslice, partials);
    else
        cov_partial<<<dim3(p.npairs, (unsigned)S), 256, 0, stream>>>(X, M, ld, r0, r1, p.nb, tslice, partials);
    MS3_LAUNCH_CHECK();
}

void cov_finish(const double* partials, int64_t S, const CovPlan& p, int64_t M, int64_t N, double* XXt,
                cudaStream_t stream) {
    if (p.tc) {
        cov_i8_finish(partials, S, M, N, XXt, stream);
        return;
    }
    if (S == 0) {
        MS3_CUDA(cudaMemsetAsync(XXt, 0, sizeof(double) * (size_t)(M * M), stream));
        return;
    }
    const int64_t total = (int64_t)p.npairs * kCT * kCT;
    cov_reduce<<<(unsigned)(total / 32), 256, 0, stream>>>(partials, (int)S, p.npairs, p.nb, M, N, XXt);
    MS3_LAUNCH_CHECK();
}

void covariance_sum_device(const float* X, int64_t M, int64_t N, double* XXt_sum, cudaStream_t stream) {
    if (M <= 0) return;
    const CovPlan p = cov_plan(X, M);
    const int64_t S = cov_slices(p, N);
    DevBuf partials(cov_partials_bytes(p, S), stream);
    cov_partials(X, M, 0, N, p, partials.as<double>(), S, stream);
    cov_finish(partials.as<double>(), S, p, M, /*N=*/1, XXt_sum, stream);  // N <= 1: no division
}

void covariance_device(const float* X, int64_t M, int64_t N, double* XXt, cudaStream_t stream, int64_t ld) {
    if (M <= 0) return;
    const CovPlan p = cov_plan(X, M, ld);
    const int64_t S = cov_slices(p, N);
    DevBuf partials(cov_partials_bytes(p, S), stream);
    cov_partials(X, M, 0, N, p, partials.as<double>(), S, stream, ld);
    cov_finish(partials.as<double>(), S, p, M, N, XXt, stream);
}

// ------------------------------------------------ covariance without allocation
//
// Scratch for the partial covariance tiles of ms3gpu_whiten_covariance_noalloc:
// a fixed array in the library's device image, present on every GPU that
// loads the library until the process exits.  Host code cannot use the
// symbol's name as a device address; its address is looked up once per
// device with cudaGetSymbolAddress and passed to the kernels.
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;  // 16 MiB
static __device__ __align__(256) unsigned char g_noalloc_cov_scratch[kNoAllocScratchBytes];

namespace {
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {};

// Device address of the scratch array on the current device (looked up on
// the first call for that device).
double* noalloc_scratch() {
    int dev = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw_unsupported("device index above 63");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        MS3_CUDA(cudaGetSymbolAddress(&p, g_noalloc_cov_scratch));
        g_noalloc_ptr[dev] = static_cast<double*>(p);
    }
    return g_noalloc_ptr[dev];
}
}  // namespace

int64_t covariance_noalloc_max_channels() {
    // the scratch must hold one time slice of 64 x 64 FP64 tiles of the upper triangle
    const size_t tile = (size_t)kCT * kCT * sizeof(double);
    int64_t nb = 1;
    while ((size_t)(nb + 1) * (nb + 2) / 2 * tile <= kNoAllocScratchBytes) nb++;
    return nb * kCT;
}

void covariance_device_noalloc(const float* X, int64_t M, int64_t N, double* XXt, cudaStream_t stream) {
    if (M <= 0) return;
    if (M > covariance_noalloc_max_channels())
        throw_invalid("ms3gpu_whiten_covariance_noalloc handles at most " +
                      std::to_string(covariance_noalloc_max_channels()) + " channels (16 MiB scratch); got " +
                      std::to_string(M));
    double* scratch = noalloc_scratch();
    const int nb = (int)ceil_div(M, kCT);
    const int npairs = nb * (nb + 1) / 2;
    if (N == 0) {
        MS3_CUDA(cudaMemsetAsync(XXt, 0, sizeof(double) * (size_t)(M * M), stream));
        return;
    }
    const int64_t s_max = (int64_t)(kNoAllocScratchBytes / ((size_t)npairs * kCT * kCT * sizeof(double)));
    const int64_t target = std::max<int64_t>(1, (int64_t)4 * num_sms() / npairs);
    int64_t S = std::min<int64_t>(std::min(target, s_max), ceil_div(N, kTT));
    const int64_t tslice = ceil_div(ceil_div(N, S), kTT) * kTT;
    S = ceil_div(N, tslice);
    // Every partial tile the reduction reads is written by cov_partial in this
    // call, so nothing left in the array by an earlier call is ever used.
    cov_partial<<<dim3(npairs, (unsigned)S), 256, 0, stream>>>(X, M, M, 0, N, nb, tslice, scratch);
    MS3_LAUNCH_CHECK();
    const int64_t total = (int64_t)npairs * kCT * kCT;
    cov_reduce<<<(unsigned)(total / 32), 256, 0, stream>>>(scratch, (int)S, npairs, nb, M, N, XXt);
    MS3_LAUNCH_CHECK();
}

// pca_cluster launch: rows in shared memory across 8 or 16 CTAs, else in global memory.
void pca_launch_smem(const double* XXt, int64_t M, double* comps, double* sigma, cudaStream_t stream);

namespace {

// pca_reg for `count` matrices, one cluster each; false when the device cannot
// hold a cluster of that size.
template <int CS, int NW, int CPL, bool GIVE_UP = false>
bool launch_pca_reg(const double* XXt, int64_t M, int count, double* comps, double* sigma, cudaStream_t stream,
                    int give_up_step = -1) {
    auto kern = pca_reg<CS, NW, CPL, GIVE_UP>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CS * count), 1, 1);
    cfg.blockDim = dim3(NW * 32, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (CS > 8) {
        MS3_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        if (clusters < 1) return false;
    }
    MS3_CUDA(cudaLaunchKernelEx(&cfg, kern, XXt, (int)M, 10, comps, sigma, give_up_step));
    MS3_LAUNCH_CHECK();
    return true;
}

// Up to 128 channels the matrix fits one CTA's registers (128 KB at most) and
// an exchange through shared memory costs less than one between SMs (128 channels:
// 0.80 us a step in one CTA, 1.04 in a cluster of eight); beyond, 16 CTAs hold it.
// The smallest instance whose column range covers M.
bool pca_registers(const double* XXt, int64_t M, int count, double* comps, double* sigma, cudaStream_t stream) {
    if (const char* give_up = std::getenv("MS3GPU_PCA_GIVE_UP_STEP")) {  // testing: one size per CTA width
        if (M > 192 && M <= 256) return launch_pca_reg<16, 4, 8, true>(XXt, M, count, comps, sigma, stream, std::atoi(give_up));
        if (M > 384 && M <= 512) return launch_pca_reg<16, 8, 16, true>(XXt, M, count, comps, sigma, stream, std::atoi(give_up));
    }
    if (M <= 32) return launch_pca_reg<1, 4, 1>(XXt, M, count, comps, sigma, stream);
    if (M <= 64) return launch_pca_reg<1, 8, 2>(XXt, M, count, comps, sigma, stream);
    if (M <= 96) return launch_pca_reg<1, 8, 3>(XXt, M, count, comps, sigma, stream);
    if (M <= 128) return launch_pca_reg<1, 8, 4>(XXt, M, count, comps, sigma, stream);
    if (M <= 192) return launch_pca_reg<16, 4, 6>(XXt, M, count, comps, sigma, stream);
    if (M <= 256) return launch_pca_reg<16, 4, 8>(XXt, M, count, comps, sigma, stream);
    if (M <= 320) return launch_pca_reg<16, 4, 10>(XXt, M, count, comps, sigma, stream);
    if (M <= 384) return launch_pca_reg<16, 4, 12>(XXt, M, count, comps, sigma, stream);
    if (M <= 512) return launch_pca_reg<16, 8, 16>(XXt, M, count, comps, sigma, stream);
    return false;
}

}  // namespace

void whitening_matrix_device(const double* XXt, int64_t M, double* W, double* comps, double* sigma,
                             cudaStream_t stream, int count) {
    if (M <= 0 || count <= 0) return;
    if (M > 65535) throw_unsupported("whitening matrix for more than 65535 channels");
    DevBuf cbuf, sbuf;
    if (!comps) { cbuf.alloc(sizeof(double) * (size_t)(M * M) * count, stream); comps = cbuf.as<double>(); }
    if (!sigma) { sbuf.alloc(sizeof(double) * (size_t)M * count, stream); sigma = sbuf.as<double>(); }

    // registers hold the working matrix up to 512 channels (MS3GPU_PCA_KERNEL=smem
    // selects the shared-memory kernel, which gives the same values)
    const char* pk = std::getenv("MS3GPU_PCA_KERNEL");
    const bool force_smem = pk && std::string(pk) == "smem";
    const char* force_global0 = std::getenv("MS3GPU_PCA_ROWS_GLOBAL");
    const bool registers = !force_smem && !(force_global0 && force_global0[0] == '1');
    if (!registers || !pca_registers(XXt, M, count, comps, sigma, stream))
        for (int64_t k = 0; k < count; k++)
            pca_launch_smem(XXt + k * M * M, M, comps + k * M * M, sigma + k * M, stream);
    const unsigned wt = (unsigned)ceil_div(M, kWT);
    constexpr int kMaxZ = 65535;  // matrices of one launch
    for (int k = 0; k < count; k += kMaxZ) {
        w_assemble<<<dim3(wt, wt, (unsigned)std::min(count - k, kMaxZ)), 256, 0, stream>>>(
            comps + k * M * M, sigma + k * M, (int)M, W + k * M * M);
        MS3_LAUNCH_CHECK();
    }
}

void whitening_read_timeout(int* flag, cudaStream_t stream) {
    MS3_CUDA(cudaMemcpyFromSymbolAsync(flag, g_pca_timeout, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
}

void whitening_check_timeout(cudaStream_t stream) {
    int h = 0;
    whitening_read_timeout(&h, stream);
    MS3_CUDA(cudaStreamSynchronize(stream));
    whitening_raise_timeout(h, stream);
}

void whitening_raise_timeout(int flag, cudaStream_t stream) {
    if (flag) {
        const int zero = 0;
        MS3_CUDA(cudaMemcpyToSymbolAsync(g_pca_timeout, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
        MS3_CUDA(cudaStreamSynchronize(stream));
        throw Error(MS3GPU_ERR_CUDA, "power iteration: exchange wait timed out");
    }
}

void pca_launch_smem(const double* XXt, int64_t M, double* comps, double* sigma, cudaStream_t stream) {
    int dev = 0, max_optin = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    MS3_CUDA(cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t vec_bytes = sizeof(double) * (size_t)(3 * M + 32);
    int CS = 0, R = 0, in_smem = 0;
    // MS3GPU_PCA_ROWS_GLOBAL=1 keeps the working matrix in global memory
    // even when it fits shared memory (exercises that path in tests).
    const char* force_global = std::getenv("MS3GPU_PCA_ROWS_GLOBAL");
    const bool allow_smem = !(force_global && force_global[0] == '1');
    for (int cs : {8, 16}) {
        if (!allow_smem) break;
        const int r = (int)ceil_div(M, cs);
        const size_t need = vec_bytes + sizeof(double) * (size_t)r * (size_t)(M + 1);
        if (need <= (size_t)max_optin) { CS = cs; R = r; in_smem = 1; break; }
    }
    DevBuf xg;
    if (!in_smem) {
        CS = 16;
        R = (int)ceil_div(M, CS);
        xg.alloc(sizeof(double) * (size_t)CS * R * (size_t)(M + 1), stream);
    }
    const size_t smem = vec_bytes + (in_smem ? sizeof(double) * (size_t)R * (size_t)(M + 1) : 0);
    MS3_CUDA(cudaFuncSetAttribute(pca_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (CS > 8) MS3_CUDA(cudaFuncSetAttribute(pca_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CS, 1, 1);
    cfg.blockDim = dim3(kPcaThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MS3_CUDA(cudaLaunchKernelEx(&cfg, pca_cluster, XXt, (int)M, R, 10, in_smem, xg.as<double>(), comps, sigma));
    MS3_LAUNCH_CHECK();
}

// rows per group and blocks of the two copies above
static void channel_copy_shape(int64_t M2, int64_t N, int& rows, unsigned& blocks) {
    if (M2 > 0x7fffffff) throw_unsupported("more than 2^31 channels");
    rows = (int)std::max<int64_t>(1, kGroupElems / M2);
    blocks = (unsigned)std::min<int64_t>(ceil_div(N, rows), (int64_t)num_sms() * 32);
}

void gather_channels_device(const float* X, int64_t M, int64_t N, const int32_t* ch, int64_t M2, float* out,
                            cudaStream_t stream) {
    if (N <= 0 || M2 <= 0) return;
    int rows;
    unsigned blocks;
    channel_copy_shape(M2, N, rows, blocks);
    gather_channels<<<blocks, 256, 0, stream>>>(X, M, N, ch, (int)M2, rows, out);
    MS3_LAUNCH_CHECK();
}

void scatter_channels_device(const void* Y, int64_t M2, int64_t N, const int32_t* ch, int64_t M, void* out,
                             size_t elem, cudaStream_t stream) {
    if (N <= 0 || M2 <= 0) return;
    int rows;
    unsigned blocks;
    channel_copy_shape(M2, N, rows, blocks);
    if (elem == 2)
        scatter_channels<int16_t><<<blocks, 256, 0, stream>>>(static_cast<const int16_t*>(Y), (int)M2, N, ch, M, rows,
                                                              static_cast<int16_t*>(out));
    else
        scatter_channels<float><<<blocks, 256, 0, stream>>>(static_cast<const float*>(Y), (int)M2, N, ch, M, rows,
                                                            static_cast<float*>(out));
    MS3_LAUNCH_CHECK();
}

void apply_whitening_device(const float* X, int64_t M, int64_t N, const double* W, double quantization_unit,
                            bool mixed, void* out, cudaStream_t stream, int* err, bool round_1e4, int64_t ld,
                            int* host_err) {
    if (M <= 0 || N <= 0) return;
    if (ld == 0) ld = M;
    // MS3GPU_APPLY_FFMA=1 selects the FP32 FMA kernel for the plain form
    const char* ffma = std::getenv("MS3GPU_APPLY_FFMA");
    const bool force_ffma = ffma && ffma[0] == '1';
    if (quantization_unit <= 0 && (mixed || !force_ffma) && apply_f16_supported(X, M, N, out, ld)) {
        apply_whitening_f16(X, M, N, W, /*drain=*/!mixed, out, stream, err, round_1e4, ld, host_err);
        return;
    }
    // int16 output, and float output of many channels or that TMA stores cannot reach
    if (apply_tc_supported(X, M, N, out, ld) && (mixed || !force_ffma)) {
        apply_whitening_tc(X, M, N, W, quantization_unit, /*drain=*/!mixed, out, stream, err, round_1e4, ld, host_err);
        return;
    }
    DevBuf wt(sizeof(float) * (size_t)(M * M), stream);
    w_to_float<<<(unsigned)ceil_div(M * M, 256), 256, 0, stream>>>(W, M * M, wt.as<float>());
    MS3_LAUNCH_CHECK();
    const int64_t blocks = ceil_div(N, kBM) * ceil_div(M, kBN);
    if (blocks > 0x7fffffff) throw_unsupported("too many tiles for the apply kernel");
    apply_gemm<<<(unsigned)blocks, 256, 0, stream>>>(X, wt.as<float>(), M, N, ld, quantization_unit, round_1e4 ? 1 : 0,
                                                     out);
    MS3_LAUNCH_CHECK();
}

int bounds_site_whiten(cudaStream_t s) {
#ifdef MS3GPU_BOUNDS_CHECK
    return take_bounds_site(s);
#else
    (void)s;
    return 0;
#endif
}

}  // namespace ms3gpu
