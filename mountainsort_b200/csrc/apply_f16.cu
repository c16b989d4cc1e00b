// Whitening apply with float output on the 5th-generation tensor cores, kind::f16.
//
// y_t = W^T x_t (p_whiten.cpp:174-183) as OUT[t][m1] = sum_m2 X[t][m2] Wt[m1][m2],
// then the 1e-4 rounding.  (int16 output keeps the TF32 kernel of apply_tc.cu: its
// values are whole numbers that move with the last bit of the sums.)
//
// Precision: x and w as pairs of 11-bit halves, three products per term,
//     x w ~= x_h w_h + x_h w_l + x_l w_h.
// FP16 holds 11 significant bits like TF32 but five bits of exponent, so both sides
// are scaled by powers of two first.  Input channel k's values are multiplied by about
// max_m |W(k, m)| and its row of W divided by it: for a whitening matrix that brings
// channels of any gain to one size.  Then a timepoint's 64 values of a K-block are
// scaled so that their largest lies in [2^14, 2^15), a column of W likewise.  x_h = rn(x
// s), x_l = rn((x s - x_h) 2^11): 22 bits of every value down to 2^-29 of the largest
// (2^-51 of the largest below that).  The cross products x_l w_h + x_h w_l form at 2^11
// times their size, and the first step of x_h w_h scales the accumulator back
// (scale-input-d).  (Without the 2^11, x_l was subnormal from 2^-18 of the largest on.)
// The tensor core's FP32 accumulation rounds toward zero, so each K-block of 64 gets a
// fresh accumulator -- cross products first, while the sum is small, then the four
// steps of x_h w_h -- and the drain warps add it, times the row's scale, into
// round-to-nearest FP32 sums in registers (one FMA: the scale is a power of two).
// Unrounded outputs against 64 bits, relative: 1.4e-7 at 384 channels (the TF32 kernel
// 3.1e-7, its undrained form 2.8e-6), 1.0e-7 at 32 (3.3e-7), the same on channels whose
// gains differ by 10^6.  So both precision forms take this kernel.
//
// Where a value's bits are cut at 2^-51 of the row's largest, the error goes to every
// output that the value contributes to, also to one whose weight for that largest value
// is tiny or zero.  So W decides (split_column): this kernel runs when every weight,
// after the channels' scales, is at least 2^-30 of its column's largest and of the root
// of its K-block's sum of squares; then the cut is below 2^-21 of the terms that the output
// sums, for any x.  Any other W (identity, block-diagonal, sparse) is applied with each
// value held by itself: up to 32 channels by FP32 FMAs in this kernel (apply_rows), beyond
// by the TF32 kernel.  Beyond, both kernels are launched and the one that W's flag does not
// name returns at once (3.5 us).  Whitening matrices of correlated channels have their
// smallest at 2^-24 (384 channels) to 2^-14 (32); uncorrelated noise, 2^-33 at 200.  Only W
// is looked at, so the same W takes the same path in every call and slab.
// A row that holds an infinity or NaN in a K-block, and a column of W that does, come
// out NaN, as they do from the TF32 split.
//
// What bounds it: at 192 columns a K-block of 64 has 1152 cycles of tensor time and 264
// KB of shared-memory traffic (X 32 KB in, 32 read and 32 written by the converter, W 48
// KB in, 12 MMA steps reading 10 KB each: 2062 cycles at 128 B/clk), and takes about
// 4000: the MMAs run at most two K-blocks ahead of the drain (two accumulators of up to
// 256 TMEM columns), and a tile's end costs the drain warps as much as four blocks'
// drains.  Hence the short rounding (quantize.cuh), the scales in shared memory, and
// tiles in turn between the warpgroups where one holds all columns.  12 drain warps of
// 64 columns were no faster (96 registers each: the converter slows down), stores
// straight from registers slower (498 against 462 us), a single accumulation over K
// would be less exact than TF32 with drains.
// 384 channels x 300k: 590 us with TF32 (128 x 128 tiles, 32-wide blocks, FP64 rounding),
// now 407; 200 x 1.5M: 1253 (undrained) and 944; 32 x 1.8M: 213 and 124.
//
// A persistent CTA per SM walks tiles of 128 timepoints x BN channels (BN <= 192):
//   warp 0       TMA: X (two 128 x 32 float boxes) into a ring of kXStages, W_h and
//                W_l (BN x 64 halves) into a ring of kWStages
//   warp 1       TMEM allocation; one thread issues the MMAs (two accumulators)
//   warps 2-5    a thread per row: scale, split, write x_h and x_l over the row's own
//                floats (64 floats are 128 + 128 bytes of halves)
//   warps 6-13   a thread per row and half of the columns, or per row of every other
//                tile: drain, round, store (TMA)
// Every mbarrier wait is bounded (tc::mbar_wait); a timeout raises *err.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "common.cuh"
#include "ms3gpu.h"
#include "quantize.cuh"
#include "tc_sm100.cuh"
#include "whiten.h"

namespace ms3gpu {

namespace {

constexpr int kRows = 128;          // timepoints per tile (MMA M)
constexpr int kKB = 64;             // K elements per block (128 bytes of halves)
constexpr int kMaxBN = 192;         // channels per tile
constexpr int kMaxHalf = kMaxBN / 2;
constexpr int kXStages = 3;
constexpr int kWStages = 2;
constexpr int kXBytes = kRows * kKB * 4;  // floats, then x_h | x_l
constexpr int kXHalf = kXBytes / 2;
constexpr int kKBytes = kKB * 4;          // a K-block's channel scales
// Per K-block: its row scales (exponents, -108 .. 99) and the barriers "MMAs complete"
// (one commit serves the drain warps and the producer) and "scales written".  X of block
// g is loaded after the MMAs of g - 3, which start when g - 5 has been drained: block g
// may be written while g - 4 is still to be read, so the ring holds more than four.
constexpr int kRing = 8;
constexpr int8_t kNotFinite = -128;
constexpr int kConvWarp0 = 2, kConvWarps = 4;
constexpr int kDrainWarp0 = 6, kDrainWarps = 8;
constexpr int kThreads = (kDrainWarp0 + kDrainWarps) * 32;  // 448: 144 registers per thread
constexpr int kBoxCols = 16;        // output box: 32 rows x 16 columns, two per drain warp
constexpr int kBoxBytes = 32 * kBoxCols * 4;
constexpr int kMaxCols = 3072;      // channels (with the last tile's padding): their scales stay in shared memory

constexpr size_t w_stage_bytes(int BN) { return (size_t)2 * BN * 128; }
// staging boxes per drain warp: two where they fit beside the rings
__host__ __device__ constexpr int n_boxes(int BN) { return BN <= 176 ? 2 : 1; }
constexpr size_t smem_bytes(int BN, int cols) {
    return (size_t)kXStages * (kXBytes + kKBytes) + kWStages * w_stage_bytes(BN) +
           (size_t)n_boxes(BN) * kDrainWarps * kBoxBytes + (size_t)cols * sizeof(float) + kRing * kRows * sizeof(int8_t) + 1024 /*align*/ + 256 /*barriers*/;
}
// Channels of a call: equal tiles of up to 192, in steps of 16 (the MMA's N).
constexpr int kMaxM = kMaxCols - 16 * 16;  // 16 column tiles at most, each padded by less than 16
__host__ __device__ constexpr int col_tiles(int M) { return (M + kMaxBN - 1) / kMaxBN; }
__host__ __device__ constexpr int tile_cols(int M) { return ((M + col_tiles(M) - 1) / col_tiles(M) + 15) / 16 * 16; }
// The most that any accepted M asks for.  Not the largest tile's: up to 176 columns there
// are two boxes per warp (1024 channels, six tiles of 176: 228,480 bytes; 192 x 16: 228,352).
constexpr size_t max_smem_bytes() {
    size_t most = 0;
    for (int M = 4; M <= kMaxM; M += 4) {
        const size_t b = smem_bytes(tile_cols(M), col_tiles(M) * tile_cols(M));
        most = b > most ? b : most;
    }
    return most;
}
constexpr bool cols_fit() {
    for (int M = 4; M <= kMaxM; M += 4)
        if (col_tiles(M) * tile_cols(M) > kMaxCols) return false;
    return true;
}
static_assert(max_smem_bytes() <= 232448 && cols_fit(), "shared memory of one CTA");

// 2^k as a float, k within the normal range
__device__ __forceinline__ float pow2f(int k) { return __uint_as_float((uint32_t)(127 + k) << 23); }

constexpr float kLowScale = 2048.0f;  // 2^11: the low halves' factor

// D = A B + 2^-11 D
__device__ __forceinline__ void mma_f16_after_cross(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc)
        : "memory");
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 consecutive columns without the wait
__device__ __forceinline__ void tmem_ld_x16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// the wait, tied to the registers it makes valid
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

__device__ __forceinline__ float quantize_1e4_any(float x) {
    if (fabsf(x) < kQuantizeRange) return quantize_1e4_small(x);
    return (float)__dmul_rn(floor(__dadd_rn(__ddiv_rn((double)x, 0.0001), 0.5)), 0.0001);
}

// The apply by FP32 FMAs for few channels: a thread forms four outputs of two or four
// timepoints.  W lies in shared memory as floats, the outputs side by side; timepoints
// arrive by cp.async, kRowStages - 1 groups ahead.  The line lies where the TF32 kernel in
// its place is as fast (identity, whole calls: 4 channels x 4M 104 us, TF32 830; 12 x 3M 174
// and 770; 32 x 1.8M 255 and 253; 64 x 900k 367 and 240); below it that kernel's launch is
// saved, which small calls notice (300 clips of 32 channels: 57.4 us with it, 53 without).
constexpr int kRowsM = 32;
constexpr int kRowStages = 4;
__host__ __device__ constexpr int row_floats(int M) { return M + 4; }  // of a staged timepoint: no bank conflicts
__host__ __device__ constexpr int rows_of(int M) { return kThreads / (M / 4); }
__host__ __device__ constexpr int rows_each(int M) { return M <= 16 ? 2 : 4; }  // of a thread; what fits
constexpr size_t rows_smem(int M) {
    return 16 + sizeof(float) * ((size_t)M * M + (size_t)kRowStages * rows_each(M) * rows_of(M) * row_floats(M));
}
constexpr bool rows_fit() {
    for (int M = 4; M <= kRowsM; M += 4)
        if (rows_smem(M) > smem_bytes(tile_cols(M), tile_cols(M))) return false;
    return true;
}
static_assert(rows_fit(), "shared memory of the FP32 form");

template <int H>
__device__ __noinline__ void apply_rows(const float* X, const double* __restrict__ W, int M, int64_t N, int64_t ld,
                                        int round_1e4, float* out) {
    extern __shared__ uint8_t smem_raw[];
    constexpr float kMax = 3.402823466e38f;
    float* ws = reinterpret_cast<float*>(smem_raw + ((0u - tc::smem_u32(smem_raw)) & 15u));
    float* staged = ws + M * M;
    const int quads = M / 4, rows = rows_of(M), pitch = row_floats(M);
    const int r = threadIdx.x / quads, q = threadIdx.x - r * quads;
    const bool mine = r < rows;
    const int64_t step = (int64_t)gridDim.x * H * rows;
    auto bring = [&](int64_t t0, int stage) {
#pragma unroll
        for (int h = 0; h < H; h++) {
            const int64_t t = t0 + h * rows + r;
            const bool in = t < N;
            const uint32_t dst = tc::smem_u32(staged + ((size_t)(stage * H + h) * rows + r) * pitch + 4 * q);
            if (mine)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(X + (in ? t * ld + 4 * q : 0)),
                             "r"(in ? 16 : 0)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int64_t t0 = (int64_t)blockIdx.x * H * rows;
#pragma unroll
    for (int i = 0; i < kRowStages - 1; i++) bring(t0 + i * step, i);
    for (int i = threadIdx.x; i < M * M; i += kThreads) {  // W^T[m][k] to ws[k][m]
        const float w = (float)W[i];
        ws[(i % M) * M + i / M] = fabsf(w) <= kMax ? w : __uint_as_float(0x7FC00000u);
    }
    const float4* w = reinterpret_cast<const float4*>(ws) + q;
    for (int stage = 0; t0 < N; t0 += step, stage = (stage + 1) % kRowStages) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRowStages - 2) : "memory");
        __syncthreads();  // the group is here, and every thread is done with the one before
        bring(t0 + (kRowStages - 1) * step, (stage + kRowStages - 1) % kRowStages);
        if (!mine) continue;
        float y[H][4] = {};
        const float* x0 = staged + ((size_t)stage * H * rows + r) * pitch;  // + h rows pitch: this thread's timepoints
        const int next = rows * pitch;
#pragma unroll 2
        for (int c = 0; c < quads; c++) {
            float4 v[H];
#pragma unroll
            for (int h = 0; h < H; h++) v[h] = *reinterpret_cast<const float4*>(x0 + h * next + 4 * c);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 u = w[(4 * c + i) * quads];
#pragma unroll
                for (int h = 0; h < H; h++) {
                    const float x = i == 0 ? v[h].x : i == 1 ? v[h].y : i == 2 ? v[h].z : v[h].w;
                    y[h][0] = __fmaf_rn(x, u.x, y[h][0]);
                    y[h][1] = __fmaf_rn(x, u.y, y[h][1]);
                    y[h][2] = __fmaf_rn(x, u.z, y[h][2]);
                    y[h][3] = __fmaf_rn(x, u.w, y[h][3]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < H; h++) {
            const int64_t t = t0 + h * rows + r;
            if (t >= N) continue;
            // an infinity or NaN in the row leaves no output finite: all of them become NaN
            if (!(fabsf(y[h][0]) <= kMax) && !(fabsf(y[h][1]) <= kMax) && !(fabsf(y[h][2]) <= kMax) && !(fabsf(y[h][3]) <= kMax))
                for (int k = 0; k < M; k++)
                    if (!(fabsf(x0[h * next + k]) <= kMax)) y[h][0] = y[h][1] = y[h][2] = y[h][3] = __uint_as_float(0x7FC00000u);
            if (round_1e4) {
#pragma unroll
                for (int j = 0; j < 4; j++) y[h][j] = quantize_1e4_any(y[h][j]);
            }
            if (MS3_IN_BOUNDS(t * ld + 4 * q + 3, (N - 1) * ld + M, 305))
                *reinterpret_cast<float4*>(out + t * ld + 4 * q) = make_float4(y[h][0], y[h][1], y[h][2], y[h][3]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// COLS: columns of a drain thread, a multiple of 16 that covers them; instances for few
// columns are short enough for the instruction cache.
template <int COLS>
__global__ void __launch_bounds__(kThreads, 1)
    apply_f16_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmWh,
                     const __grid_constant__ CUtensorMap tmWl, const __grid_constant__ CUtensorMap tmOut, int64_t M,
                     int64_t N, int BN, int ncb, int64_t ntiles, const float* __restrict__ in_scale,
                     const float* __restrict__ col_scale, const int* __restrict__ wide, const float* X,
                     const double* __restrict__ W, int64_t ld, float* out, int round_1e4, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    if (*wide) {  // beyond kRowsM the TF32 kernel's
        if (COLS <= kRowsM && M <= kRowsM) apply_rows<rows_each(COLS)>(X, W, (int)M, N, ld, round_1e4, out);
        return;
    }
    const uint32_t w_bytes = (uint32_t)BN * 128u;  // one of W_h, W_l
    uint8_t* xs = smem;
    uint8_t* ws = xs + kXStages * kXBytes;
    uint8_t* boxes = ws + (size_t)kWStages * 2 * w_bytes;
    float* ks = reinterpret_cast<float*>(boxes + (size_t)n_boxes(BN) * kDrainWarps * kBoxBytes);  // [kXStages][kKB]
    float* cols = ks + kXStages * kKB;                                     // [ncb * BN] column scales
    int8_t* rs = reinterpret_cast<int8_t*>(cols + ncb * BN);               // scale exponents
    uint64_t* bars = reinterpret_cast<uint64_t*>(rs + kRing * kRows);
    uint64_t* x_full = bars;                     // [kXStages] TMA bytes landed
    uint64_t* hl_full = x_full + kXStages;       // [kXStages] halves written
    uint64_t* w_full = hl_full + kXStages;       // [kWStages]
    uint64_t* acc_free = w_full + kWStages;      // [2] accumulator read back
    uint64_t* done = acc_free + 2;               // [kRing] a K-block's MMAs complete
    uint64_t* rs_full = done + kRing;            // [kRing] row scales written
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rs_full + kRing);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nkb = (int)((M + kKB - 1) / kKB);
    const int64_t my_tiles = (blockIdx.x < ntiles) ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int64_t total = my_tiles * nkb;  // K-blocks of this CTA
    // More than half a warpgroup's columns: the two drain warpgroups share a tile, each
    // with its columns.  Up to that many: they take tiles in turn, so that one's
    // epilogue overlaps the other's.
    const bool share = BN > kMaxHalf;
    // 32-column boxes of X in K-block kb
    auto boxes_of = [&](int kb) { return M - (int64_t)kb * kKB > 32 ? 2 : 1; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kXStages; s++) {
            tc::mbar_init(&x_full[s], 1);
            tc::mbar_init(&hl_full[s], kConvWarps);
        }
        for (int s = 0; s < kWStages; s++) tc::mbar_init(&w_full[s], 1);
        for (int b = 0; b < 2; b++) tc::mbar_init(&acc_free[b], share ? kDrainWarps : kDrainWarps / 2);
        for (int b = 0; b < kRing; b++) {
            tc::mbar_init(&done[b], 1);
            tc::mbar_init(&rs_full[b], kConvWarps);
        }
        tc::fence_mbar_init();
    }
    for (int j = threadIdx.x; j < ncb * BN; j += kThreads) cols[j] = j < M ? col_scale[j] : 0.f;
    if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t taddr = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int64_t gx = 0, gw = 0;  // K-blocks whose X and W were issued
            int sx = 0, sw = 0, kb = 0;
            auto mmas_done = [&](int64_t h) { return tc::mbar_wait(&done[h & (kRing - 1)], (uint32_t)((h / kRing) & 1), err); };
            int64_t tile = blockIdx.x;
            for (int64_t g = 0; g < total; g++) {
                const int t0 = (int)(tile / ncb) * kRows, n0 = (int)(tile % ncb) * BN;
                if (g >= kXStages && !mmas_done(g - kXStages)) break;
                const int nb = boxes_of(kb);
                tc::mbar_expect_tx(&x_full[sx], (uint32_t)(nb * kXHalf + kKBytes));
                tc::bulk_load_1d(ks + sx * kKB, in_scale + kb * kKB, kKBytes, &x_full[sx]);
                for (int h = 0; h < nb; h++)
                    tc::tma_load_2d(xs + sx * kXBytes + h * kXHalf, &tmX, &x_full[sx], kb * kKB + h * 32, t0);
                gx = g + 1;
                if (++sx == kXStages) sx = 0;
                if (g >= kWStages && !mmas_done(g - kWStages)) break;
                uint8_t* w = ws + (size_t)sw * 2 * w_bytes;
                tc::mbar_expect_tx(&w_full[sw], 2 * w_bytes);
                tc::tma_load_2d(w, &tmWh, &w_full[sw], kb * kKB, n0);
                tc::tma_load_2d(w + w_bytes, &tmWl, &w_full[sw], kb * kKB, n0);
                gw = g + 1;
                if (++sw == kWStages) sw = 0;
                if (++kb == nkb) kb = 0, tile += gridDim.x;
            }
            // no copy may still be landing in shared memory when the CTA exits
            for (int64_t g = (gx > kXStages ? gx - kXStages : 0); g < gx; g++)
                tc::mbar_wait(&x_full[g % kXStages], (uint32_t)((g / kXStages) & 1), err);
            for (int64_t g = (gw > kWStages ? gw - kWStages : 0); g < gw; g++)
                tc::mbar_wait(&w_full[g % kWStages], (uint32_t)((g / kWStages) & 1), err);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // One thread issues: what it computes per MMA is on the critical path, so the
            // descriptors of stage 0 are formed once and advanced by additions.
            const uint32_t idesc = tc::instr_desc(0u /*F16*/, kRows, BN);
            const uint64_t x0 = tc::smem_desc_k_sw128(tc::smem_u32(xs)), d_w0 = tc::smem_desc_k_sw128(tc::smem_u32(ws));
            int sx = 0, sw = 0, kb = 0;
            uint32_t px = 0, pw = 0;
            int64_t g = 0;
            for (; g < total; g++) {
                const int b = (int)(g & 1);
                if (!tc::mbar_wait(&w_full[sw], pw, err) || !tc::mbar_wait(&hl_full[sx], px, err)) break;
                if (g >= 2 && !tc::mbar_wait(&acc_free[b], (uint32_t)(((g >> 1) - 1) & 1), err)) break;
                tc::tc_fence_after();
                const uint32_t acc = taddr + (uint32_t)(b * 256);
                const uint64_t xh = x0 + (uint64_t)(sx * (kXBytes >> 4)), xl = xh + (kXHalf >> 4);
                const uint64_t wh = d_w0 + (uint64_t)(sw * ((2 * w_bytes) >> 4)), wl = wh + (w_bytes >> 4);
                const int left = (int)M - kb * kKB;
                // 16 halves are 32 bytes, 2 in a descriptor's address field
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (left > 16 * k) mma_f16(acc, xl + 2 * k, wh + 2 * k, idesc, k != 0);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (left > 16 * k) mma_f16(acc, xh + 2 * k, wl + 2 * k, idesc, 1);
                mma_f16_after_cross(acc, xh, wh, idesc);
#pragma unroll
                for (int k = 1; k < 4; k++)
                    if (left > 16 * k) mma_f16(acc, xh + 2 * k, wh + 2 * k, idesc, 1);
                tc::mma_commit(&done[g & (kRing - 1)]);
                if (++sx == kXStages) sx = 0, px ^= 1;
                if (++sw == kWStages) sw = 0, pw ^= 1;
                if (++kb == nkb) kb = 0;
            }
            // no MMA may still be writing TMEM when it is freed
            for (int64_t h = (g > 2 ? g - 2 : 0); h < g; h++)
                tc::mbar_wait(&done[h & (kRing - 1)], (uint32_t)((h / kRing) & 1), err);
        }
    } else if (warp < kDrainWarp0) {
        const int row = (warp - kConvWarp0) * 32 + lane;
        int sx = 0, kb = 0;
        uint32_t px = 0;
        for (int64_t g = 0; g < total; g++) {
            const bool ok = tc::mbar_wait(&x_full[sx], px, err);
            if (!__all_sync(0xffffffffu, ok)) break;
            uint8_t* tile = xs + sx * kXBytes + row * 128;
            const int nb = boxes_of(kb);
            float4 v[16];
            float top = 0.f;  // largest magnitude (a NaN passes by: it stays NaN as a half)
#pragma unroll
            for (int c = 0; c < 16; c++) {
                if (c < 8 * nb) {
                    v[c] = *reinterpret_cast<const float4*>(tile + (c >> 3) * kXHalf + (((c & 7) ^ (row & 7)) << 4));
                    const float4 k = *reinterpret_cast<const float4*>(ks + sx * kKB + 4 * c);
                    v[c] = make_float4(v[c].x * k.x, v[c].y * k.y, v[c].z * k.z, v[c].w * k.w);
                    top = fmaxf(fmaxf(top, fabsf(v[c].x)), fabsf(v[c].y));
                    top = fmaxf(fmaxf(top, fabsf(v[c].z)), fabsf(v[c].w));
                }
            }
            const int e = max((int)(__float_as_uint(top) >> 23) - 127, -80);  // rows below 2^-80 keep that scale
            const bool finite = top <= 3.402823466e38f;
            const float s = finite ? pow2f(14 - e) : 1.0f;
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
                if (c < 8 * nb) {
                    const float f[8] = {v[c].x, v[c].y, v[c].z, v[c].w, v[c + 1].x, v[c + 1].y, v[c + 1].z, v[c + 1].w};
                    uint4 h, l;
                    uint32_t* hw = reinterpret_cast<uint32_t*>(&h);
                    uint32_t* lw = reinterpret_cast<uint32_t*>(&l);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const __half2 hi = __floats2half2_rn(f[2 * i] * s, f[2 * i + 1] * s);
                        const float2 hf = __half22float2(hi);
                        // the remainders and their multiples are exact
                        const __half2 lo = __floats2half2_rn(__fmaf_rn(f[2 * i], s, -hf.x) * kLowScale,
                                                             __fmaf_rn(f[2 * i + 1], s, -hf.y) * kLowScale);
                        hw[i] = *reinterpret_cast<const uint32_t*>(&hi);
                        lw[i] = *reinterpret_cast<const uint32_t*>(&lo);
                    }
                    const int at = ((c >> 1) ^ (row & 7)) << 4;
                    *reinterpret_cast<uint4*>(tile + at) = h;
                    *reinterpret_cast<uint4*>(tile + kXHalf + at) = l;
                }
            }
            // the accumulator is 2^(14 - e) x times 2^(14 - E) w: the sums are out / 2^E
            rs[(g & (kRing - 1)) * kRows + row] = finite ? (int8_t)(e - 28) : kNotFinite;
            tc::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                tc::mbar_arrive(&hl_full[sx]);
                tc::mbar_arrive(&rs_full[g & (kRing - 1)]);
            }
            if (++sx == kXStages) sx = 0, px ^= 1;
            if (++kb == nkb) kb = 0;
        }
    } else {
        const int q = warp & 3;  // TMEM lanes 32 q .. 32 q + 31
        const int row = q * 32 + lane;
        const int w0 = warp - kDrainWarp0;
        const int group = w0 >> 2;
        const int first = ((BN / 2 + 15) / 16) * 16;  // columns of the first group when they share
        const int c_base = share && group ? first : 0, nc = share ? (group ? BN - first : first) : BN;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const bool two_boxes = n_boxes(BN) == 2;
        uint8_t* box = boxes + (size_t)w0 * n_boxes(BN) * kBoxBytes;
        int sbuf = 0;
        int64_t g = share ? 0 : (int64_t)group * nkb;
        bool ok = true;
        for (int64_t i = share ? 0 : group; i < my_tiles && ok; i += share ? 1 : 2, g += share ? 0 : nkb) {
            const int64_t tile = blockIdx.x + i * gridDim.x;
            const int64_t trow = (tile / ncb) * kRows + q * 32;
            const int n0 = (int)(tile % ncb) * BN + c_base;
            float y[COLS];
#pragma unroll
            for (int j = 0; j < COLS; j++) y[j] = 0.f;
            for (int kb = 0; kb < nkb; kb++, g++) {
                const int b = (int)(g & 1), rb = (int)(g & (kRing - 1));
                ok = tc::mbar_wait(&done[rb], (uint32_t)((g / kRing) & 1), err) &&
                     tc::mbar_wait(&rs_full[rb], (uint32_t)((g / kRing) & 1), err);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc::tc_fence_after();
                const int re = rs[rb * kRows + row];
                const float r = re == kNotFinite ? __uint_as_float(0x7FC00000u) : pow2f(re);
                const uint32_t acc = taddr + (uint32_t)(b * 256 + c_base) + lane_base;
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    if (c < nc) {
                        uint32_t a[16];
                        tmem_ld_x16_nowait(acc + (uint32_t)c, a);
                        tmem_ld_wait(a);
#pragma unroll
                        for (int j = 0; j < 16; j++) y[c + j] = __fmaf_rn(__uint_as_float(a[j]), r, y[c + j]);
                    }
                }
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&acc_free[b]);
            }
            if (!ok) break;
#pragma unroll
            for (int c = 0; c < COLS; c += 16) {
                const int n = n0 + c;
                // a box wholly beyond the last row or column would be clipped whole
                if (c < nc && n < M && trow < N) {
                    uint8_t* st = box + (size_t)sbuf * kBoxBytes;
                    float z[16];
                    float big = 0.f;
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const float4 s = *reinterpret_cast<const float4*>(cols + n + j);
                        z[j] = __fmul_rn(y[c + j], s.x);
                        z[j + 1] = __fmul_rn(y[c + j + 1], s.y);
                        z[j + 2] = __fmul_rn(y[c + j + 2], s.z);
                        z[j + 3] = __fmul_rn(y[c + j + 3], s.w);
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++) big = fmaxf(big, fabsf(z[j]));
                    const bool fp32 = round_1e4 && big < kQuantizeRange;
                    if (fp32) {
#pragma unroll
                        for (int j = 0; j < 16; j++) z[j] = quantize_1e4_small(z[j]);
                    }
                    if (lane == 0) {  // the store before has read this box
                        if (two_boxes)
                            tc::bulk_wait_group_read<1>();
                        else
                            tc::bulk_wait_group_read<0>();
                    }
                    __syncwarp();
                    float* own = reinterpret_cast<float*>(st + lane * 64);
                    const int sw = (lane >> 1) & 3;  // 64-byte swizzle
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        *reinterpret_cast<float4*>(own + 4 * (k ^ sw)) = make_float4(z[4 * k], z[4 * k + 1], z[4 * k + 2], z[4 * k + 3]);
                    if (round_1e4 && !fp32) {
#pragma unroll 1
                        for (int k = 0; k < 16; k++) own[k] = quantize_1e4_any(own[k]);
                    }
                    tc::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && MS3_IN_BOUNDS(n, M, 303) && MS3_IN_BOUNDS(trow, N, 304)) {
                        tc::tma_store_2d(&tmOut, st, n, (int)trow);
                        tc::bulk_commit_group();
                    }
                    if (two_boxes) sbuf ^= 1;
                }
            }
        }
        if (lane == 0) tc::bulk_wait_group<0>();  // stores complete before the CTA exits
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(taddr, 512);
    }
}

// floor(log2 a) of a finite a, at least -126 (0 for a = 0)
__device__ __forceinline__ int exponent_of(double a) {
    return a == 0.0 ? 0 : max((int)((__double2hiint(a) >> 20) & 0x7FF) - 1023, -126);
}
__device__ __forceinline__ double finite_abs(double w) {  // 0 beyond the float range
    const double a = fabs(w);
    return a < 0x1p128 ? a : 0.0;
}

// 1 / s for a power of two s (2^1023 for 0: those weights are zero)
__device__ __forceinline__ double inverse_pow2(float s) {
    return __hiloint2double((2046 - (__double2hiint((double)s) >> 20)) << 20, 0);
}

// Where the halves of W go: FP16 for this kernel, TF32 (as apply_tc.cu forms them) for
// the other, the scales, and the flag for a W that the other takes.
struct SplitW {
    __half *hi, *lo;        // [M][Kp]
    float *hi32, *lo32;     // [M][M], or null (kRowsM)
    float *in_scale, *col_scale;
    int *wide, *err;        // err: null, or cleared
};

// Column m of W^T divided by the channels' scales, WARPS warps: E = floor(log2 max), the
// column's scale 2^E, the column times 2^(14 - E) as halves w_h = rn(w), w_l = rn((w -
// w_h) 2^11), Kp of them (zeros beyond M).  A column with magnitudes beyond the float
// range, infinities or NaN gets the scale NaN.  *wide is set for a weight below 2^-30 of
// the column's largest or of its K-block's root sum of squares.
// The warps take the K-blocks in turn.  (One warp a column took 13.5 us at 384 channels,
// a third of the time of a call with few timepoints.)
template <int WARPS>
__device__ __forceinline__ void split_column(const double* __restrict__ w, int64_t m, int64_t M, int64_t Kp,
                                             const float* in_scale, const SplitW& o) {
    const int l = threadIdx.x & 31, first = WARPS > 1 ? threadIdx.x >> 5 : 0;
    double top = 0.0, least = 1e300;  // of the magnitudes; of their squares
    bool finite = true, narrow = true;
#pragma unroll 2
    for (int64_t k0 = first * kKB; k0 < M; k0 += WARPS * kKB) {
        double sum = 0.0, low = 1e300;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int64_t k = k0 + l + 32 * i;
            const double v = k < M ? w[k] : 0.0;
            const float scale = k < M ? in_scale[k] : 0.f;
            finite &= fabs(v) < 0x1p128;
            const double a = finite_abs(v) * inverse_pow2(scale);
            top = fmax(top, a);
            sum += a * a;
            if (scale != 0.f) low = fmin(low, a * a);
        }
        for (int s = 16; s > 0; s >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, s);
            low = fmin(low, __shfl_xor_sync(0xffffffffu, low, s));
        }
        narrow &= low >= 0x1p-60 * sum;
        least = fmin(least, low);
    }
    for (int s = 16; s > 0; s >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, s));
    finite = __all_sync(0xffffffffu, finite);
    if (WARPS > 1) {
        __shared__ double tops[WARPS], leasts[WARPS];
        if (l == 0) {
            tops[first] = top;
            leasts[first] = least;
        }
        finite = __syncthreads_and(finite);
        narrow = __syncthreads_and(narrow);
        for (int i = 0; i < WARPS; i++) {
            top = fmax(top, tops[i]);
            least = fmin(least, leasts[i]);
        }
    }
    const int e = exponent_of(top);
    if (l == 0 && first == 0) {
        if (finite && !(narrow && least >= 0x1p-60 * (top * top))) *o.wide = 1;
        o.col_scale[m] = finite ? pow2f(e) : __uint_as_float(0x7FC00000u);
    }
    const double s = __hiloint2double((1023 + 14 - e) << 20, 0);
    __half* hi = o.hi + m * Kp;
    __half* lo = o.lo + m * Kp;
#pragma unroll 4
    for (int64_t k = first * 32 + l; k < Kp; k += WARPS * 32) {
        const double v = k < M ? w[k] : 0.0;
        const double x = k < M ? v * inverse_pow2(in_scale[k]) * s : 0.0;
        const __half h = __double2half(x);
        hi[k] = h;
        lo[k] = __double2half((x - (double)__half2float(h)) * (double)kLowScale);
        if (o.hi32 && k < M) {
            const float h32 = __uint_as_float(tc::cvt_rna_tf32((float)v));
            o.hi32[m * M + k] = h32;
            o.lo32[m * M + k] = __uint_as_float(tc::cvt_rna_tf32((float)(v - (double)h32)));
        }
    }
}

__device__ __forceinline__ float in_scale_of(double top) { return top > 0.0 ? pow2f(exponent_of(top)) : 0.f; }

// in_scale[k] = 2^floor(log2 max_m |W^T[m][k]|), 0 for a channel without weights (so
// that its values, which no output holds, set no row's scale) and beyond M.  Block: 32
// channels x 32 parts of m.
__global__ void __launch_bounds__(1024) w_in_scales(const double* __restrict__ W, int64_t M, int64_t n_in, SplitW o) {
    __shared__ double part[32][33];
    if (blockIdx.x == 0 && threadIdx.x == 0) *o.wide = 0;
    const int l = threadIdx.x & 31, p = threadIdx.x >> 5;
    const int64_t k = (int64_t)blockIdx.x * 32 + l;
    double top = 0.0;
    if (k < M) {
#pragma unroll 8
        for (int64_t m = p; m < M; m += 32) top = fmax(top, finite_abs(W[m * M + k]));
    }
    part[p][l] = top;
    __syncthreads();
    // warp p reduces channel p of the block
    top = part[l][p];
    for (int o16 = 16; o16 > 0; o16 >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o16));
    const int64_t kp = (int64_t)blockIdx.x * 32 + p;
    if (l == 0 && kp < n_in) o.in_scale[kp] = in_scale_of(top);
}

__global__ void __launch_bounds__(128) w_split_f16(const double* __restrict__ W, int64_t M, int64_t Kp, SplitW o) {
    if (o.err && blockIdx.x == 0 && threadIdx.x == 0) *o.err = 0;
    const int64_t m = blockIdx.x;
    split_column<4>(W + m * M, m, M, Kp, o.in_scale, o);
}

// Both in one block for up to 64 channels, where a launch costs more than the work.
constexpr int kSmallM = 64;
__global__ void __launch_bounds__(1024) w_prepare_small(const double* __restrict__ W, int M, int Kp, SplitW o) {
    if (threadIdx.x == 0) {
        *o.wide = 0;
        if (o.err) *o.err = 0;
    }
    __shared__ double part[16][kSmallM];
    __shared__ double copy[kSmallM * kSmallM];
    __shared__ float scale[kSmallM];
    const int k = threadIdx.x & (kSmallM - 1), p = threadIdx.x / kSmallM;
    double top = 0.0;
    if (k < M) {
#pragma unroll
        for (int i = 0; i < kSmallM / 16; i++) {
            const int m = p + 16 * i;
            if (m < M) {
                const double w = W[m * M + k];
                copy[m * M + k] = w;
                top = fmax(top, finite_abs(w));
            }
        }
    }
    part[p][k] = top;
    __syncthreads();
    if (p == 0) {
        for (int i = 1; i < 16; i++) top = fmax(top, part[i][k]);
        o.in_scale[k] = scale[k] = in_scale_of(top);
    }
    __syncthreads();
    for (int m = threadIdx.x >> 5; m < M; m += 32) split_column<1>(copy + m * M, m, M, Kp, scale, o);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn_f16() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    if (!fn) throw_unsupported("cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// Row-major [rows][cols] matrix with `pitch` bytes between rows.
CUtensorMap matrix_map(CUtensorMapDataType type, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch,
                       uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {pitch};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = encode_fn_f16()(&m, type, 2, const_cast<void*>(base), dims, strides, box, es,
                                       CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw_unsupported("cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return m;
}

// Per device, once.  The kernels that prepare W ask for the apply's split of the
// SM's memory too: changing it between two launches costs a few microseconds.
void set_kernel_attributes(int dev) {
    static std::once_flag once[64];
    auto set = [] {
        for (auto k : {apply_f16_kernel<16>, apply_f16_kernel<32>, apply_f16_kernel<64>, apply_f16_kernel<96>})
            MS3_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)max_smem_bytes()));
        for (const void* k : {(const void*)w_prepare_small, (const void*)w_in_scales, (const void*)w_split_f16})
            MS3_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                          (int)cudaSharedmemCarveoutMaxShared));
    };
    if (dev < 64)
        std::call_once(once[dev], set);
    else
        set();
}

}  // namespace

bool apply_f16_supported(const float* X, int64_t M, int64_t N, const void* out, int64_t ld) {
    return apply_tc_supported(X, M, N, out, ld) && M <= kMaxM && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && N < (1LL << 31) - kRows;
}

void apply_whitening_f16(const float* X, int64_t M, int64_t N, const double* W, bool drain, void* out,
                         cudaStream_t stream, int* ext_err, bool round_1e4, int64_t ld, int* host_err) {
    int dev = 0;
    MS3_CUDA(cudaGetDevice(&dev));
    set_kernel_attributes(dev);
    const int ncb = col_tiles((int)M), BN = tile_cols((int)M);
    const int64_t Kp = ceil_div(M, 8) * 8;  // 16-byte rows
    const int64_t n_in = ceil_div(M, kKB) * kKB;
    const size_t n_scales = (size_t)n_in + (size_t)ncb * (size_t)BN;
    auto padded = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t half_bytes = padded((size_t)(M * Kp) * sizeof(__half)), tf32_bytes = M > kRowsM ? padded((size_t)(M * M) * sizeof(float)) : 0;
    DevBuf buf(2 * half_bytes + 2 * tf32_bytes + n_scales * sizeof(float) + 256, stream);
    SplitW w;
    char* at = buf.as<char>();
    w.hi = reinterpret_cast<__half*>(at);
    w.lo = reinterpret_cast<__half*>(at += half_bytes);
    w.hi32 = reinterpret_cast<float*>(at += half_bytes);
    w.lo32 = reinterpret_cast<float*>(at += tf32_bytes);
    w.in_scale = reinterpret_cast<float*>(at += tf32_bytes);
    if (!tf32_bytes) w.hi32 = w.lo32 = nullptr;
    w.col_scale = w.in_scale + n_in;
    w.wide = reinterpret_cast<int*>(w.in_scale + n_scales);
    w.err = ext_err ? nullptr : w.wide + 1;  // the call's own flag: cleared with the preparation of W
    int* err = ext_err ? ext_err : w.err;
    if (M <= kSmallM) {
        w_prepare_small<<<1, 1024, 0, stream>>>(W, (int)M, (int)Kp, w);
    } else {
        w_in_scales<<<(unsigned)ceil_div(n_in, 32), 1024, 0, stream>>>(W, M, n_in, w);
        MS3_LAUNCH_CHECK();
        w_split_f16<<<(unsigned)M, 128, 0, stream>>>(W, M, Kp, w);
    }
    MS3_LAUNCH_CHECK();
    const CUtensorMap mx = matrix_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, X, (uint64_t)M, (uint64_t)N,
                                      (uint64_t)ld * sizeof(float), 32, kRows, CU_TENSOR_MAP_SWIZZLE_128B);
    const CUtensorMap mh = matrix_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w.hi, (uint64_t)Kp, (uint64_t)M,
                                      (uint64_t)Kp * sizeof(__half), kKB, (uint32_t)BN, CU_TENSOR_MAP_SWIZZLE_128B);
    const CUtensorMap ml = matrix_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w.lo, (uint64_t)Kp, (uint64_t)M,
                                      (uint64_t)Kp * sizeof(__half), kKB, (uint32_t)BN, CU_TENSOR_MAP_SWIZZLE_128B);
    const CUtensorMap mo = matrix_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, (uint64_t)M, (uint64_t)N,
                                      (uint64_t)ld * sizeof(float), kBoxCols, 32, CU_TENSOR_MAP_SWIZZLE_64B);
    const int64_t ntiles = ceil_div(N, kRows) * ncb;
    int nsm = 0;
    MS3_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t sm = smem_bytes(BN, ncb * BN);
    const int cols = BN > kMaxHalf ? ((BN / 2 + 15) / 16) * 16 : BN;
    auto kern = cols <= 16   ? apply_f16_kernel<16>
                : cols <= 32 ? apply_f16_kernel<32>
                : cols <= 64 ? apply_f16_kernel<64>
                             : apply_f16_kernel<96>;
    kern<<<(unsigned)std::min<int64_t>(ntiles, nsm), kThreads, sm, stream>>>(
        mx, mh, ml, mo, M, N, BN, ncb, ntiles, w.in_scale, w.col_scale, w.wide, X, W, ld, static_cast<float*>(out),
        round_1e4 ? 1 : 0, err);
    MS3_LAUNCH_CHECK();
    if (M > kRowsM)
        apply_tc_launch(X, M, N, ld, w.hi32, w.lo32, /*quantization_unit=*/0.0, drain, round_1e4, out, err, w.wide,
                        stream);
    if (ext_err) return;  // the caller checks the flag once for many calls
    if (host_err) {  // the caller looks at it after its own synchronisation
        MS3_CUDA(cudaMemcpyAsync(host_err, err, sizeof(int), cudaMemcpyDeviceToHost, stream));
        return;
    }
    int herr = 0;
    MS3_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, stream));
    MS3_CUDA(cudaStreamSynchronize(stream));
    if (herr) throw Error(MS3GPU_ERR_CUDA, "tensor-core apply: pipeline wait timed out");
}

int bounds_site_apply_f16(cudaStream_t s) {
#ifdef MS3GPU_BOUNDS_CHECK
    return take_bounds_site(s);
#else
    (void)s;
    return 0;
#endif
}

}  // namespace ms3gpu
