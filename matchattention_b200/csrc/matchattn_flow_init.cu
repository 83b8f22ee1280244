// Flow branch of GlobalCorrelation after its matmul, with local_flow_estimator
// (models/cost_volume.py:61-69 and :71-121), as four kernels:
//
//   corr [B, N, N] (N = H*W; scaled q.k^T, reference token then target token)
//   prob [2B, N, N]   written: softmax over the last axis of corr[b] and of corr[b]^T
//   flow [2B, H, W, 2] written
//
// The reference materialises the concatenation [corr; corr^T] (2 x N^2), its softmax, the 5x5-pooled copy
// (avg_pool2d over the N x N "image"), arg max, a [2B, N, 25, 2] gather of coordinates and a dozen
// elementwise temporaries.  Here:
//   1. flow_max_kernel        one read of corr: partial maxima of rows AND columns
//   2. flow_sum_kernel        one read for the rows, one for the columns: maximum and sum of exponentials
//   3. flow_prob_pool_kernel  reads corr again, writes both halves of prob and, from the values in registers,
//                             the maximum of the 5x5 box sums per (token, chunk of targets); no second pass over prob
//   4. flow_window_kernel     per token: the chunks that can hold the arg max are pooled once more to find it, then
//                             the 5x5 window estimate
// The window hangs on an arg max, and box averages that differ in their last bit are common in the 16-bit types; so
// prob and the deciding averages are formed in one fixed order (sums of exponentials in 256 interleaved partial sums
// per row and four per column, box sums row by row) whatever the split of the work, and only the screening in step 3
// adds in another.
// Measured on a B200, float16, 128x128 tokens (1.61 GB are the least possible, 3.2 GB move): 1.01 to 1.04 ms in a row of
// calls = 0.09 + 0.25 + 0.62 + 0.05; with a pooling pass over the stored probabilities and separate statistics passes it was
// 6.59 ms, of which the pooling took 4.1.  48x48 tokens: 44 us, before 196.
// Rounding of the 16-bit types as eager PyTorch on the GPU: softmax, pooling and sums accumulate in float32
// and round once, every elementwise op rounds.
#include "../../include/matchattn.h"

#include <stdint.h>

#include <type_traits>

#include "matchattn_kernels.cuh"

namespace matchattn {
namespace {

constexpr int kFlowThreads = 256;
constexpr int kFlowWarps = kFlowThreads / 32;
constexpr int kLaneCols = 4;                          // consecutive columns of corr that a lane owns
constexpr int kWarpCols = 32 * kLaneCols;
constexpr int kMaxRows = 16;                          // rows of corr that a lane holds at a time in the maximum pass
constexpr int kPoolCols = kWarpCols - 2 * kLaneCols;  // columns a warp pools: its outer lanes are the halo
constexpr int kPoolStep = 4;                          // rows per step of the pooling kernel, the next four on their way
constexpr int kTransBytes = 64;                       // run of a prob row that a transposed store writes
constexpr int kPoolSmemPerWarp = kWarpCols * (kTransBytes + 16);
constexpr int kPoolWarps = 4;                         // warps per block of the pooling kernel
constexpr int kSumGroups = 4;                         // interleaved partial sums per column
constexpr int kWindowTokens = kFlowWarps;             // tokens per block of the window kernel: one per warp
// Rows per warp of the maximum and the pooling kernel: long columns amortise the start of a warp (the halo rows, the
// merges of the partials), from so many tokens on; below there are not enough warps to fill the chip with long ones, and
// the single-element accesses of odd token counts want more of them.  Measured, float16, long against short: 64x64 tokens
// 117.4 / 113.1 us, 68x72 145.9 / 148.3, 76x76 181.9 / 189.5, 128x128 1142 / 1231; odd: 67x71 208 / 186, 79x83 352 / 331,
// 97x101 692 / 691; float32: 60x60 105.3 / 103.9, 68x72 167.9 / 173.0, 79x83 356 / 333.
constexpr int64_t kLongBands = 5000, kLongBandsOdd = 10000;
// Column sums: 32-column blocks from so many tokens on, 16-column blocks below, where the wider ones leave SMs without work.
// Measured, the whole call, wide against narrow: float16 48x48 tokens 45.8 / 45.0 us, 64x64 103.6 / 102.4, 72x72 145.8 / 144.8,
// 80x80 200.4 / 208.0, 96x96 365.2 / 387.6; float32 64x64 119.9 / 119.5, 76x76 206.3 / 201.8, 88x88 343.4 / 356.2; in
// rows aligned to single elements 70x73 224.1 / 231.6, 78x75 265.7 / 279.3, 79x83 311.2 / 334.3.  Single 16-bit elements
// (strided): the narrow blocks read 32 rows ahead, the wide ones 16; float16 96x96 418.2 / 407.9, 96x100 433.3 / 445.5.
template <typename T>
constexpr int64_t kWideSums = sizeof(T) == 2 ? 5800 : 6600;
constexpr int64_t kWideStrided = 9400, kWideOdd = 5000;

// Column sums of a block: batches of exponentials, two of them in shared memory.
template <int COLUMNS>
struct SumTile {
    static constexpr int kPieces = COLUMNS / 8;                    // threads per row of a batch, eight columns each
    static constexpr int kPasses = 2, kPassRows = kFlowThreads / kPieces, kRows = kPasses * kPassRows;
    static constexpr int kPitch = COLUMNS + 4;                     // floats: keeps the 16-byte stores of neighbouring rows apart
    static constexpr int kBytes = 2 * kRows * kPitch * static_cast<int>(sizeof(float));
};

// Sizes and scratch areas of one call, computed alike by the size query and the launcher.
struct FlowPlan {
    int64_t N;
    int max_rows;       // rows per warp of the maximum kernel
    int row_parts;      // partials per row of corr (one per kWarpCols columns)
    int col_parts;      // partials per column of corr (one per max_rows rows)
    int band;           // rows per warp of the pooling kernel
    int chunks, bands;  // chunks of kPoolCols columns, bands of rows
    size_t off_col, off_stats, off_row_max, off_col_max, bytes;
};

FlowPlan flow_plan(int B, int H, int W)
{
    FlowPlan pl{};
    pl.N = static_cast<int64_t>(H) * W;
    const auto parts = [&](int64_t of) { return static_cast<int>((pl.N + of - 1) / of); };
    const bool long_bands = pl.N >= (pl.N % 2 == 0 ? kLongBands : kLongBandsOdd);
    pl.max_rows = long_bands ? 128 : 32;
    pl.band = long_bands ? 64 : 32;
    pl.row_parts = parts(kWarpCols);
    pl.col_parts = parts(pl.max_rows);
    pl.chunks = parts(kPoolCols);
    pl.bands = parts(pl.band);
    const auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
    const size_t n = static_cast<size_t>(B) * pl.N;
    size_t off = up(n * pl.row_parts * sizeof(float));
    pl.off_col = off;     off = up(off + n * pl.col_parts * sizeof(float));
    pl.off_stats = off;   off = up(off + 2 * n * sizeof(float2));
    pl.off_row_max = off; off = up(off + n * pl.chunks * sizeof(float));
    pl.off_col_max = off; off = up(off + n * pl.bands * sizeof(float));
    pl.bytes = off;
    return pl;
}

// maximum over a warp in one instruction (PTX ISA 8.6, sm_100a)
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// Four consecutive elements of a row of corr, raw (two words of pairs, or four words).  ALIGN: rows
// start at a multiple of so many elements (1, 2, 4, 8), so that a lane's group is four loads, two (16-bit types), or one.
// FULL: the group lies inside the row; otherwise columns outside [0, N) and rows outside [0, N) read as -infinity
// (probability 0).
template <typename T>
__device__ __forceinline__ uint32_t word_max(uint32_t a, uint32_t b)
{
    if constexpr (sizeof(T) == 4) {
        return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
    } else if constexpr (std::is_same_v<T, __half>) {
        const __half2 m = __hmax2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
        return *reinterpret_cast<const uint32_t *>(&m);
    } else {
        const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
        return *reinterpret_cast<const uint32_t *>(&m);
    }
}

template <typename T>
struct Group {
    uint32_t w[kLaneCols / DT<T>::kElemsPerWord];
    __device__ __forceinline__ float get(int k) const { return DT<T>::unpack(w[k / DT<T>::kElemsPerWord], k % DT<T>::kElemsPerWord); }
    // element k + x, the element converted in the addition
    __device__ __forceinline__ float plus(int k, float x) const
    {
        if constexpr (sizeof(T) == 4) return __uint_as_float(w[k]) + x;
        else {
            const unsigned short h = static_cast<unsigned short>(k % 2 ? w[k / 2] >> 16 : w[k / 2] & 0xffffu);
            if constexpr (std::is_same_v<T, __half>) return add_f32_f16(x, h);
            else return add_f32_bf16(x, h);
        }
    }
    __device__ __forceinline__ void max_with(const Group &o)      // element by element
    {
#pragma unroll
        for (int i = 0; i < kLaneCols / DT<T>::kElemsPerWord; ++i) w[i] = word_max<T>(w[i], o.w[i]);
    }
    __device__ __forceinline__ float max4() const
    {
        if constexpr (sizeof(T) == 4) return fmaxf(fmaxf(get(0), get(1)), fmaxf(get(2), get(3)));
        const uint32_t m = word_max<T>(w[0], w[1]);
        return fmaxf(DT<T>::unpack(m, 0), DT<T>::unpack(m, 1));
    }
    __device__ __forceinline__ void mask()
    {
        constexpr uint32_t kMinusInf = sizeof(T) == 4 ? 0xff800000u : std::is_same_v<T, __nv_bfloat16> ? 0xff80ff80u : 0xfc00fc00u;
#pragma unroll
        for (uint32_t &x : w) x = kMinusInf;
    }
};

__device__ __forceinline__ float plus_float(float a, float x) { return a + x; }
__device__ __forceinline__ float plus_float(__half a, float x) { return add_f32_f16(x, __half_as_ushort(a)); }
__device__ __forceinline__ float plus_float(__nv_bfloat16 a, float x) { return add_f32_bf16(x, __bfloat16_as_ushort(a)); }

template <typename T>
__device__ __forceinline__ uint32_t raw_bits(const T *p)
{
    if constexpr (sizeof(T) == 4) return *reinterpret_cast<const uint32_t *>(p);
    else return *reinterpret_cast<const unsigned short *>(p);
}

template <typename T, int ALIGN, bool FULL>
__device__ __forceinline__ Group<T> load_group(const T *row, int64_t col, int64_t N, bool row_ok)
{
    Group<T> g;
    constexpr int EPW = DT<T>::kElemsPerWord;
    if constexpr (ALIGN == 2 && EPW == 2) {
        g.mask();
#pragma unroll
        for (int k = 0; k < kLaneCols; k += 2)
            if (FULL || (row_ok && col + k >= 0 && col + k < N)) g.w[k / 2] = *reinterpret_cast<const uint32_t *>(row + col + k);
    } else if constexpr (FULL || ALIGN >= kLaneCols) {
        if (!FULL && (!row_ok || col < 0 || col >= N)) {
            g.mask();
            return g;
        }
        if constexpr (ALIGN < kLaneCols) {
#pragma unroll
            for (int k = 0; k < kLaneCols; k += EPW) {
                uint32_t w = raw_bits(row + col + k);
                if constexpr (EPW == 2) w |= raw_bits(row + col + k + 1) << 16;
                g.w[k / EPW] = w;
            }
        } else if constexpr (EPW == 1) {
            const uint4 t = *reinterpret_cast<const uint4 *>(row + col);
            g.w[0] = t.x; g.w[1] = t.y; g.w[2] = t.z; g.w[3] = t.w;
        } else {
            const uint2 t = *reinterpret_cast<const uint2 *>(row + col);
            g.w[0] = t.x; g.w[1] = t.y;
        }
    } else {
        g.mask();
        if (!row_ok) return g;
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k)
            if (col + k >= 0 && col + k < N) {
                const uint32_t w = raw_bits(row + col + k);
                if constexpr (EPW == 1) g.w[k] = w;
                else g.w[k / 2] = (k & 1) ? __byte_perm(g.w[k / 2], w, 0x5410) : __byte_perm(g.w[k / 2], w, 0x3254);
            }
    }
    return g;
}

// Partial maxima of the rows and columns of corr.  A warp takes 128 columns (four per lane) and walks down its rows,
// sixteen at a time; the maxima are taken on pairs of 16-bit values.  Memory-bound.
template <typename T, int ALIGN, bool FULL>
__device__ __forceinline__ void max_tile(const T *src, int64_t col, int64_t r0, int64_t last, int64_t N, Group<T> &cm, float *row_part, int lane)
{
    Group<T> g[kMaxRows];
#pragma unroll
    for (int r = 0; r < kMaxRows; ++r) g[r] = load_group<T, ALIGN, FULL>(src + (r0 + r) * N, col, N, r0 + r < last);
    float mine = -INFINITY;
#pragma unroll
    for (int r = 0; r < kMaxRows; ++r) {
        const float m = warp_max(g[r].max4());
        mine = lane == r ? m : mine;
        cm.max_with(g[r]);
    }
    if (lane < kMaxRows && r0 + lane < last) row_part[r0 + lane] = mine;
}

template <typename T, int ALIGN>
__global__ void __launch_bounds__(kFlowThreads) flow_max_kernel(const T *corr, float *__restrict__ row_part,
                                                                float *__restrict__ col_part, int64_t N, int rows_per_warp,
                                                                int row_parts, int col_parts)
{
    chain_begin();
    const int lane = threadIdx.x & 31;
    const int64_t unit = static_cast<int64_t>(blockIdx.x) * kFlowWarps + (threadIdx.x >> 5);
    const int band = static_cast<int>(unit / row_parts), chunk = static_cast<int>(unit - static_cast<int64_t>(band) * row_parts);
    if (band >= col_parts) return;
    const int64_t b = blockIdx.y;
    const T *src = corr + b * N * N;
    const int64_t col0 = static_cast<int64_t>(chunk) * kWarpCols, col = col0 + lane * kLaneCols;
    const int64_t first = static_cast<int64_t>(band) * rows_per_warp, last = min(first + rows_per_warp, N);
    float *rows = row_part + (b * row_parts + chunk) * N;
    Group<T> cm;
    cm.mask();
    for (int64_t r0 = first; r0 < last; r0 += kMaxRows) {
        if (col0 + kWarpCols <= N && r0 + kMaxRows <= last) max_tile<T, ALIGN, true>(src, col, r0, last, N, cm, rows, lane);
        else max_tile<T, ALIGN, false>(src, col, r0, last, N, cm, rows, lane);
    }
#pragma unroll
    for (int k = 0; k < kLaneCols; ++k)
        if (col + k < N) col_part[(b * col_parts + band) * N + col + k] = cm.get(k);
}

// Maximum and sum of a row of corr by a warp: 256 partial sums (element j goes to sum j mod 256), then a tree over each 32
// of them and a running sum over the eight results.
template <typename T, int ALIGN>
__device__ __forceinline__ void row_sum(const T *src, const float *row_part, float2 *stats, int64_t row, int64_t N, int row_parts)
{
    const int lane = threadIdx.x & 31;
    if (row >= N) return;
    float mx = -INFINITY;
    for (int i = lane; i < row_parts; i += 32) mx = fmaxf(mx, row_part[i * N + row]);
    mx = warp_max(mx);
    const T *p = src + row * N;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float total = 0.f;
    if constexpr (ALIGN >= 4) {     // lane l holds the partial sums 8 l .. 8 l + 7; elements past the end add exp(-inf)
        constexpr bool kWhole = ALIGN >= 8;
#pragma unroll 4
        for (int64_t j = lane * 8; j < N; j += 256) {
            const Group<T> g0 = load_group<T, ALIGN, kWhole>(p, j, N, true), g1 = load_group<T, ALIGN, kWhole>(p, j + 4, N, true);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s[k] += expf(g0.plus(k, -mx));
                s[k + 4] += expf(g1.plus(k, -mx));
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            s[k] += __shfl_xor_sync(0xffffffffu, s[k], 2);
            s[k] += __shfl_xor_sync(0xffffffffu, s[k], 1);
        }
        const float sum = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
#pragma unroll
        for (int w = 0; w < 8; ++w) total += __shfl_sync(0xffffffffu, sum, 4 * w);
    } else {                  // lane l holds the partial sums l, l + 32, .. l + 224
        int64_t j = lane;
        for (; j + 224 < N; j += 256) {
            float x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = load_one<T>(p + j + 32 * k);
#pragma unroll
            for (int k = 0; k < 8; ++k) s[k] += expf(x[k] - mx);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (j + 32 * k < N) s[k] += expf(load_one<T>(p + j + 32 * k) - mx);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
            total += s[k];
        }
    }
    if (lane == 0) stats[row] = make_float2(mx, total);
}

// stats[half, b, token] = (maximum, sum of exp(x - maximum)) of row `token` of corr[b] (half 0) or of column `token`
// (half 1).  The first blocks serve COLUMNS columns each: all threads take the exponentials of a batch of rows into shared
// memory, eight columns of a row at a time, then a thread per column and remainder of the row by four adds them up in order
// while the others are at the next batch.  The other blocks serve one row per warp: 256 partial sums (element j goes to sum
// j mod 256), then a tree over each 32 of them and a running sum over the eight results.
// Bound by instruction issue (one exponential per element and half), on small maps by the chain of batches.  Measured, float16,
// the sums alone: 96x96 tokens 106 -> 91 us, 128x128 259 -> 249, 82x79 81 -> 60; 48x48 14.4 -> 13.2 (a thread per column and
// remainder that read, exponentiated and added one column, at 156 registers).
template <typename T, int ALIGN, int COLUMNS>
__global__ void __launch_bounds__(kFlowThreads, 4) flow_sum_kernel(const T *corr, const float *row_part,
                                                                const float *col_part, float2 *__restrict__ stats,
                                                                int64_t N, int row_parts, int col_parts, int col_blocks)
{
    chain_begin();
    const int64_t b = blockIdx.y;
    const T *src = corr + b * N * N;
    if (static_cast<int>(blockIdx.x) < col_blocks) {
        using Tile = SumTile<COLUMNS>;
        extern __shared__ __align__(16) float e_s[];
        __shared__ float part[kFlowThreads / COLUMNS][COLUMNS];
        const int tid = threadIdx.x, c = tid % COLUMNS, g = tid / COLUMNS;
        const int64_t c0 = static_cast<int64_t>(blockIdx.x) * COLUMNS, col = c0 + c;
        float mx = -INFINITY;
        if (col < N) {
#pragma unroll 4
            for (int i = g; i < col_parts; i += kFlowThreads / COLUMNS) mx = fmaxf(mx, col_part[(b * col_parts + i) * N + col]);
        }
        part[g][c] = mx;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kFlowThreads / COLUMNS; ++i) mx = fmaxf(mx, part[i][c]);
        __syncthreads();
        if (g == 0) part[0][c] = mx;
        __syncthreads();
        const int piece = tid % Tile::kPieces, first = tid / Tile::kPieces;        // eight columns, first row of a batch
        float neg_max[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) neg_max[k] = -part[0][8 * piece + k];
        const int64_t at = c0 + 8 * piece;
        Group<T> raw[Tile::kPasses][2];
        const auto load = [&](int64_t r0) {
            const bool full = c0 + COLUMNS <= N && r0 + Tile::kRows <= N;
#pragma unroll
            for (int p = 0; p < Tile::kPasses; ++p) {
                const int64_t row = r0 + first + p * Tile::kPassRows;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (full) raw[p][i] = load_group<T, ALIGN, true>(src + row * N, at + 4 * i, N, true);
                    else raw[p][i] = load_group<T, ALIGN, false>(src + row * N, at + 4 * i, N, row < N);
                }
            }
        };
        float den = 0.f;
        load(0);
        float *buffer = e_s;
        for (int64_t r0 = 0; r0 < N; r0 += Tile::kRows) {
#pragma unroll
            for (int p = 0; p < Tile::kPasses; ++p) {
                float *out = buffer + (first + p * Tile::kPassRows) * Tile::kPitch + 8 * piece;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const Group<T> &v = raw[p][i];
                    *reinterpret_cast<float4 *>(out + 4 * i) = make_float4(expf(v.plus(0, neg_max[4 * i])), expf(v.plus(1, neg_max[4 * i + 1])),
                                                                           expf(v.plus(2, neg_max[4 * i + 2])), expf(v.plus(3, neg_max[4 * i + 3])));
                }
            }
            if (r0 + Tile::kRows < N) load(r0 + Tile::kRows);
            __syncthreads();
            if (g < kSumGroups) {
                const float *in = buffer + g * Tile::kPitch + c;
                if (r0 + Tile::kRows <= N) {
#pragma unroll 16
                    for (int r = 0; r < Tile::kRows; r += kSumGroups) den += in[r * Tile::kPitch];
                } else {
                    for (int r = 0; r0 + g + r < N; r += kSumGroups) den += in[r * Tile::kPitch];
                }
            }
            buffer = buffer == e_s ? e_s + Tile::kRows * Tile::kPitch : e_s;      // the barrier of the next batch guards this one
        }
        if (g < kSumGroups) part[g][c] = den;
        __syncthreads();
        if (g == 0 && col < N)
            stats[(gridDim.y + b) * N + col] = make_float2(mx, (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]));
        return;
    }
    row_sum<T, ALIGN>(src, row_part + b * row_parts * N, stats + b * N, (static_cast<int64_t>(blockIdx.x) - col_blocks) * kFlowWarps + (threadIdx.x >> 5), N, row_parts);
}

// The same where rows of 16-bit elements are aligned to single elements only: a thread per column and remainder of the row by
// four reads, exponentiates and adds, BATCH rows ahead.  Measured, float16, the sums alone, this / the one above: 67x71 tokens
// 40 / 55 us, 79x83 85 / 89, 97x101 141 / 166, bfloat16 111x113 204 / 240.
template <typename T, int COLUMNS, int BATCH>
__global__ void __launch_bounds__(COLUMNS * kSumGroups) flow_sum_strided_kernel(const T *corr, const float *row_part,
                                                                const float *col_part, float2 *__restrict__ stats,
                                                                int64_t N, int row_parts, int col_parts, int col_blocks)
{
    chain_begin();
    const int64_t b = blockIdx.y;
    const T *src = corr + b * N * N;
    if (static_cast<int>(blockIdx.x) < col_blocks) {
        __shared__ float sm[kSumGroups][COLUMNS];
        const int c = threadIdx.x % COLUMNS, g = threadIdx.x / COLUMNS;
        const int64_t col = static_cast<int64_t>(blockIdx.x) * COLUMNS + c;
        float mx = -INFINITY;
        if (col < N) {
#pragma unroll 8
            for (int i = g; i < col_parts; i += kSumGroups) mx = fmaxf(mx, col_part[(b * col_parts + i) * N + col]);
        }
        sm[g][c] = mx;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSumGroups; ++i) mx = fmaxf(mx, sm[i][c]);
        __syncthreads();
        float den = 0.f;
        if (col < N) {
            const T *p = src + g * N + col;
            const int64_t step = kSumGroups * N;
            int64_t left = (N - g + kSumGroups - 1) / kSumGroups;
            T now[BATCH], next[BATCH];      // the next batch is read while this one is summed
            if (left >= BATCH) {
#pragma unroll
                for (int i = 0; i < BATCH; ++i) now[i] = p[i * step];
                while (left >= BATCH) {
                    p += BATCH * step;
                    left -= BATCH;
                    const bool more = left >= BATCH;
                    if (more) {
#pragma unroll
                        for (int i = 0; i < BATCH; ++i) next[i] = p[i * step];
                    }
#pragma unroll
                    for (int i = 0; i < BATCH; ++i) den += expf(plus_float(now[i], -mx));
                    if (more) {
#pragma unroll
                        for (int i = 0; i < BATCH; ++i) now[i] = next[i];
                    }
                }
            }
            for (; left > 0; --left, p += step) den += expf(load_one<T>(p) - mx);
        }
        sm[g][c] = den;
        __syncthreads();
        if (g == 0 && col < N)
            stats[(gridDim.y + b) * N + col] = make_float2(mx, (sm[0][c] + sm[1][c]) + (sm[2][c] + sm[3][c]));
        return;
    }
    row_sum<T, 1>(src, row_part + b * row_parts * N, stats + b * N,
                  (static_cast<int64_t>(blockIdx.x) - col_blocks) * (COLUMNS * kSumGroups / 32) + (threadIdx.x >> 5), N, row_parts);
}

// Softmax of an element: the quotient exp(x - max) / sum by one Newton step on the product with the rounded reciprocal
// (Markstein, IBM J. Res. Dev. 34, 1990): to the last bit as long as the residual does not underflow, which it does for
// float32 quotients below 2^-102; there the last bit may differ.
struct Softmax {
    float neg_max, sum, inv;
};
// Elements k and k + 1, each by its own statistics, in packed arithmetic (the pooling kernel at 128x128 tokens 621 -> 615 us).
template <typename T>
__device__ __forceinline__ float2 softmax_pair(const Group<T> &g, int k, const Softmax &a, const Softmax &b)
{
    const float2 e = make_float2(expf(g.plus(k, a.neg_max)), expf(g.plus(k + 1, b.neg_max))), inv = make_float2(a.inv, b.inv);
    const float2 q = mul_f32x2(e, inv);
    return fma_f32x2(fma_f32x2(q, make_float2(-a.sum, -b.sum), e), inv, q);
}

template <typename T>
__device__ __forceinline__ Softmax softmax_of(float2 st) { return Softmax{-st.x, st.y, __frcp_rn(st.y)}; }

// Sliding 5-sum down the rows of a pair of columns: push(p) returns p(a-4) + .. + p(a), from the pair sums it keeps.
struct PairSums {
    float2 p1, s1, s2, s3;   // p(a-1); pair sums ending at a-1, a-2, a-3
    __device__ __forceinline__ void reset() { p1 = s1 = s2 = s3 = make_float2(0.f, 0.f); }
    __device__ __forceinline__ float2 push(float2 p)
    {
        const float2 v = add_f32x2(add_f32x2(s3, s1), p);
        s3 = s2;
        s2 = s1;
        s1 = add_f32x2(p1, p);
        p1 = p;
        return v;
    }
};

// box[k] = v(c-2) + .. + v(c+2) around the lane's column k; the outer two columns come from the neighbouring lanes
__device__ __forceinline__ void box_sums(const float2 a, const float2 b, float (&box)[kLaneCols])
{
    const float pa = a.x + a.y, pb = b.x + b.y;
    const float left2 = __shfl_up_sync(0xffffffffu, pb, 1), left1 = __shfl_up_sync(0xffffffffu, b.y, 1);
    const float right1 = __shfl_down_sync(0xffffffffu, a.x, 1), right2 = __shfl_down_sync(0xffffffffu, pa, 1);
    const float mid = pa + pb;
    box[0] = (left2 + pa) + b.x;
    box[1] = left1 + mid;
    box[2] = mid + right1;
    box[3] = (a.y + pb) + right2;
}

struct PoolParams {
    const float2 *stats;
    float *row_max, *col_max;
    int64_t N;
    int B, band_rows, chunks, bands;
};

// role "rows": prob[b][row][col], statistics per row; the box maximum per (row, chunk) by a warp reduction
template <typename T, int ALIGN, bool FULL>
__device__ __forceinline__ void pool_rows(const PoolParams &pp, const T *src, T *dst, char *smem, int64_t b, int64_t a0, int64_t c0, int chunk, int lane)
{
    const int64_t N = pp.N;
    float4 *st = reinterpret_cast<float4 *>(smem);          // rows a0 - 2 .. a0 + band_rows + 1: maximum, sum, reciprocal
    float *row_max = reinterpret_cast<float *>(st + pp.band_rows + 4);
    for (int i = lane; i < pp.band_rows + 4; i += 32) {
        const int64_t a = a0 - 2 + i;
        const Softmax s = softmax_of<T>(FULL || (a >= 0 && a < N) ? pp.stats[b * N + a] : make_float2(0.f, 1.f));
        st[i] = make_float4(s.neg_max, s.sum, s.inv, 0.f);
    }
    __syncwarp();
    const bool inner = lane != 0 && lane != 31;
    PairSums lo, hi;
    lo.reset();
    hi.reset();
    // one row: probabilities, store, box sums of the row two above, their maximum over the warp
    const auto row_step = [&](const Group<T> &g, const Softmax &sm, int64_t a, bool store, bool pool) {
        float2 p01 = softmax_pair(g, 0, sm, sm), p23 = softmax_pair(g, 2, sm, sm);
        uint32_t w[kLaneCols / DT<T>::kElemsPerWord];
        if constexpr (sizeof(T) == 2) {
            w[0] = DT<T>::aw_from(p01.x, p01.y);
            w[1] = DT<T>::aw_from(p23.x, p23.y);
            p01 = make_float2(DT<T>::unpack(w[0], 0), DT<T>::unpack(w[0], 1));
            p23 = make_float2(DT<T>::unpack(w[1], 0), DT<T>::unpack(w[1], 1));
        } else {
            w[0] = __float_as_uint(p01.x); w[1] = __float_as_uint(p01.y);
            w[2] = __float_as_uint(p23.x); w[3] = __float_as_uint(p23.y);
        }
        if (store && inner && (FULL || a < N)) {
            T *out = dst + a * N + c0;
            if constexpr (ALIGN >= kLaneCols) {
                if (FULL || c0 < N) store_words<kLaneCols / DT<T>::kElemsPerWord>(out, w);
            } else if constexpr (ALIGN == 2 && sizeof(T) == 2) {
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (FULL || c0 + 2 * k < N) reinterpret_cast<uint32_t *>(out)[k] = w[k];
            } else {
                const float p[kLaneCols] = {p01.x, p01.y, p23.x, p23.y};
#pragma unroll
                for (int k = 0; k < kLaneCols; ++k)
                    if (FULL || c0 + k < N) store_one<T>(out + k, p[k]);
            }
        }
        const float2 va = lo.push(p01), vb = hi.push(p23);
        if (!pool) return;
        float box[kLaneCols];
        box_sums(va, vb, box);
        float m;
        if constexpr (FULL || ALIGN >= kLaneCols) m = fmaxf(fmaxf(box[0], box[1]), fmaxf(box[2], box[3]));
        else {
            m = 0.f;
#pragma unroll
            for (int k = 0; k < kLaneCols; ++k) m = c0 + k < N ? fmaxf(m, box[k]) : m;
        }
        m = warp_max(inner && (FULL || c0 < N) ? m : 0.f);
        if (lane == 0) row_max[a - 2 - a0] = m;
    };
    const auto load = [&](int64_t a) {
        return load_group<T, ALIGN, FULL>(src + (FULL ? min(a, N - 1) : a) * N, c0, N, a >= 0 && a < N);
    };
    const auto stat = [&](int64_t a) {
        const float4 v = st[a - (a0 - 2)];
        return Softmax{v.x, v.y, v.z};
    };
    Group<T> now[kPoolStep], next[kPoolStep];
#pragma unroll
    for (int i = 0; i < kPoolStep; ++i) now[i] = load(a0 - 2 + i);
    const int64_t end = a0 + pp.band_rows;
#pragma unroll 1
    for (int64_t a = a0 - 2; a < end + 2; a += kPoolStep) {
#pragma unroll
        for (int i = 0; i < kPoolStep; ++i) next[i] = load(a + kPoolStep + i);
#pragma unroll
        for (int i = 0; i < kPoolStep; ++i) {
            row_step(now[i], stat(a + i), a + i, i < 2 ? a >= a0 : a + i < end, i < 2 ? a > a0 : a >= a0);
            now[i] = next[i];
        }
    }
    __syncwarp();
    for (int i = lane; i < pp.band_rows; i += 32)
        if (FULL || a0 + i < N) pp.row_max[(b * pp.chunks + chunk) * N + a0 + i] = row_max[i];
}

// role "columns": prob[B + b][col][row], statistics per column; the box maximum per (column, band) stays in the lane
template <typename T, int ALIGN, bool FULL>
__device__ __forceinline__ void pool_cols(const PoolParams &pp, const T *src, T *dst, char *smem, int64_t b, int64_t a0, int64_t c0,
                                          int chunk, int band, int lane)
{
    constexpr int kTransRows = kTransBytes / sizeof(T);     // rows gathered before a transposed store
    // a column's slot in shared memory: the pitch keeps the stores of four rows (8 or 16 bytes) free of bank conflicts
    constexpr int kPitch = kTransBytes + (sizeof(T) == 2 ? 8 : 16);
    const int64_t N = pp.N;
    const bool inner = lane != 0 && lane != 31;
    PairSums lo, hi;
    lo.reset();
    hi.reset();
    Softmax sm[kLaneCols];
    float best[kLaneCols];
#pragma unroll
    for (int k = 0; k < kLaneCols; ++k) {
        sm[k] = softmax_of<T>(FULL || (c0 + k >= 0 && c0 + k < N) ? pp.stats[(pp.B + b) * N + c0 + k] : make_float2(0.f, 1.f));
        best[k] = 0.f;
    }
    // probabilities of two rows (16-bit types: a word per column, first row low), then the box sums two rows above each
    const auto two_rows = [&](const Group<T> &g0, const Group<T> &g1, int64_t a, bool pool, uint32_t (&w)[kLaneCols][2]) {
        float2 p[2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            p[0][k] = softmax_pair(g0, 2 * k, sm[2 * k], sm[2 * k + 1]);
            p[1][k] = softmax_pair(g1, 2 * k, sm[2 * k], sm[2 * k + 1]);
            if constexpr (sizeof(T) == 2) {
                const uint32_t wx = DT<T>::aw_from(p[0][k].x, p[1][k].x), wy = DT<T>::aw_from(p[0][k].y, p[1][k].y);
                w[2 * k][0] = wx;
                w[2 * k + 1][0] = wy;
                p[0][k] = make_float2(DT<T>::unpack(wx, 0), DT<T>::unpack(wy, 0));
                p[1][k] = make_float2(DT<T>::unpack(wx, 1), DT<T>::unpack(wy, 1));
            } else {
                w[2 * k][0] = __float_as_uint(p[0][k].x);
                w[2 * k][1] = __float_as_uint(p[1][k].x);
                w[2 * k + 1][0] = __float_as_uint(p[0][k].y);
                w[2 * k + 1][1] = __float_as_uint(p[1][k].y);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float2 va = lo.push(p[i][0]), vb = hi.push(p[i][1]);
            if (!pool) continue;
            float box[kLaneCols];
            box_sums(va, vb, box);
#pragma unroll
            for (int k = 0; k < kLaneCols; ++k)
                if (FULL || a + i - 2 < N) best[k] = fmaxf(best[k], box[k]);
        }
    };
    const auto load = [&](int64_t a) {
        return load_group<T, ALIGN, FULL>(src + (FULL ? min(a, N - 1) : a) * N, c0, N, a >= 0 && a < N);
    };
    uint32_t w[kLaneCols][2];
    Group<T> now[kPoolStep], next[kPoolStep];
#pragma unroll
    for (int i = 0; i < kPoolStep; ++i) now[i] = load(a0 - 2 + i);
    uint32_t pend[kLaneCols][2];          // rows a - 2 and a - 1
#pragma unroll 1
    for (int64_t a = a0 - 2; a < a0 + pp.band_rows + 2; a += kPoolStep) {
#pragma unroll
        for (int i = 0; i < kPoolStep; ++i) next[i] = load(a + kPoolStep + i);
        two_rows(now[0], now[1], a, a > a0, w);
        if (a > a0 - 2) {
            const int at = static_cast<int>(a - 2 - a0) & (kTransRows - 1);
            // column k of lane l in slot k * 32 + l
#pragma unroll
            for (int k = 0; k < kLaneCols; ++k) {
                char *slot = smem + (k * 32 + lane) * kPitch + at * sizeof(T);
                if constexpr (sizeof(T) == 2) *reinterpret_cast<uint2 *>(slot) = make_uint2(pend[k][0], w[k][0]);
                else *reinterpret_cast<uint4 *>(slot) = make_uint4(pend[k][0], pend[k][1], w[k][0], w[k][1]);
            }
            if (at == kTransRows - kPoolStep) {
                __syncwarp();
                const int64_t row0 = a + 2 - kTransRows, token0 = static_cast<int64_t>(chunk) * kPoolCols - kLaneCols;
                if constexpr (ALIGN * sizeof(T) >= 16) {      // four lanes per column, eight columns per store
                    const int64_t row = row0 + (lane & 3) * (16 / sizeof(T));
#pragma unroll 4
                    for (int u = 0; u < kWarpCols; u += 8) {
                        const int l = (u + (lane >> 2)) & 31, k = u >> 5;
                        const int64_t token = token0 + l * kLaneCols + k;
                        const char *slot = smem + (k * 32 + l) * kPitch + (lane & 3) * 16;
                        uint4 v;
                        if constexpr (sizeof(T) == 2) {
                            const uint2 v0 = *reinterpret_cast<const uint2 *>(slot), v1 = *reinterpret_cast<const uint2 *>(slot + 8);
                            v = make_uint4(v0.x, v0.y, v1.x, v1.y);
                        } else {
                            v = *reinterpret_cast<const uint4 *>(slot);
                        }
                        if (l != 0 && l != 31 && (FULL || (token < N && row < N))) *reinterpret_cast<uint4 *>(dst + token * N + row) = v;
                    }
                } else {                  // ALIGN rows per lane: 64 bytes of one column to as many of four per store
                    using Piece = std::conditional_t<ALIGN * sizeof(T) == 8, uint2, std::conditional_t<ALIGN * sizeof(T) == 4, uint32_t, uint16_t>>;
                    constexpr int kLanes = kTransRows / ALIGN;
                    const int r = lane % kLanes * ALIGN;
#pragma unroll 4
                    for (int c = kLaneCols + lane / kLanes; c < kWarpCols - kLaneCols; c += 32 / kLanes) {
                        const int64_t token = token0 + c;
                        const Piece v = *reinterpret_cast<const Piece *>(smem + ((c & 3) * 32 + (c >> 2)) * kPitch + r * sizeof(T));
                        if (FULL || (token < N && row0 + r < N)) *reinterpret_cast<Piece *>(dst + token * N + row0 + r) = v;
                    }
                }
                __syncwarp();
            }
        }
        two_rows(now[2], now[3], a + 2, a >= a0, w);
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k) {
            pend[k][0] = w[k][0];
            pend[k][1] = w[k][1];
        }
#pragma unroll
        for (int i = 0; i < kPoolStep; ++i) now[i] = next[i];
    }
    if (inner) {
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k)
            if (FULL || c0 + k < N) pp.col_max[(b * pp.bands + band) * N + c0 + k] = best[k];
    }
}

// Both halves of prob and the maxima of the 5x5 box sums.  A warp takes 128 columns of corr (120 pooled, the outer
// lanes are the halo) and walks down a band of rows (two more on either side); every lane keeps the running pair
// sums of its four columns, so a box sum costs about four additions.  Blocks come in two roles that differ in what
// the softmax runs over (pool_rows, pool_cols); a lane of the second gathers eight rows of its columns and stores
// them as 16 bytes of a prob row, or, where rows of prob are not 16-byte aligned, through shared memory.
// Eight consecutive blocks (four of either role) cover one 4-band x 4-chunk region, so the second role finds corr in L2.
// Bound by instruction issue (about 25 per element and role, a third of them the exponential; 76 % of the slots busy).
// Measured, float16, 16384 x 16384: 0.61 ms (0.72 with eight rows unrolled and the halo rows apart: the instruction cache
// ran short, 2.2 of 8 stalls).  With 16-byte stores straight from the registers to 32 rows of prob the
// second role alone took 0.67 ms; five blocks of four warps hold 20 warps per SM (0.75 ms with four blocks).
template <typename T, int ALIGN>
__global__ void __launch_bounds__(32 * kPoolWarps, sizeof(T) == 2 ? 5 : 4) flow_prob_pool_kernel(const T *corr, T *__restrict__ prob, const PoolParams pp)
{
    chain_begin();
    extern __shared__ __align__(16) char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunk_groups = (pp.chunks + kPoolWarps - 1) / kPoolWarps;
    const int region = blockIdx.x / (2 * kPoolWarps), within = blockIdx.x - region * 2 * kPoolWarps;
    const int bg = region / chunk_groups, cg = region - bg * chunk_groups;
    const bool cols = within >= kPoolWarps;
    const int band = bg * kPoolWarps + (cols ? warp : within);
    const int chunk = cg * kPoolWarps + (cols ? within - kPoolWarps : warp);
    if (band >= pp.bands || chunk >= pp.chunks) return;
    const int64_t b = blockIdx.y, N = pp.N;
    const T *src = corr + b * N * N;
    const int64_t a0 = static_cast<int64_t>(band) * pp.band_rows;
    const int64_t first = static_cast<int64_t>(chunk) * kPoolCols - kLaneCols, c0 = first + lane * kLaneCols;
    char *smem = smem_raw + warp * kPoolSmemPerWarp;
    const bool full = a0 >= 2 && a0 + pp.band_rows + 2 <= N && first >= 0 && first + kWarpCols <= N;
    if (!cols) {
        T *dst = prob + b * N * N;
        if (full) pool_rows<T, ALIGN, true>(pp, src, dst, smem, b, a0, c0, chunk, lane);
        else pool_rows<T, ALIGN, false>(pp, src, dst, smem, b, a0, c0, chunk, lane);
    } else {
        T *dst = prob + (pp.B + b) * N * N;
        if (full) pool_cols<T, ALIGN, true>(pp, src, dst, smem, b, a0, c0, chunk, band, lane);
        else pool_cols<T, ALIGN, false>(pp, src, dst, smem, b, a0, c0, chunk, band, lane);
    }
}

// Per token (b2, i): the first target j whose 5x5 box average, rounded to T, is the largest, and the expected target
// position within the 5x5 window of probabilities around it (clamped to the map) minus the token's own position.
// The box maxima per chunk of targets screen the chunks: the average is monotone in the box sum, and the screening
// sums are within kScreen of the ones that decide.  A block takes eight tokens: its threads read the chunk maxima of
// all of them at once, then every warp serves one: it sums the boxes of the chunks that pass (as a rule one) from prob, one,
// two or four neighbouring targets per lane, then takes the window, lanes = its 25 elements.  Bound by instruction issue and
// a few dependent reads.  Measured, float16: 128x128 tokens 78.7 -> 48.5 us, 48x48 10.3 -> 7.8 (a second walk over the
// maxima with a division per chunk, every box on its own, the 25 terms handed round by shuffles before).
// A chunk maximum below kCoarse * top - kCoarseStep cannot round to the top average: the 16-bit types are at most 2^-7 of a
// value and 2^-24 apart, a box sum is 25 averages.
constexpr float kCoarse = 1.f - 0x1p-6f, kCoarseStep = 25.f * 0x1p-23f;
constexpr int kKeptChunks = 256;      // chunk maxima per token that a block of the window kernel keeps in shared memory
constexpr float kScreen = 4e-6f;      // 24 float32 additions of positive terms in two different orders

template <typename T>
__global__ void __launch_bounds__(kFlowThreads) flow_window_kernel(const T *prob, const float *row_max,
                                                                   const float *col_max, T *__restrict__ flow,
                                                                   T *__restrict__ blur_max, int *__restrict__ centre_out, int B, int H,
                                                                   int W, int chunks, int bands, int band_rows, float tiny)
{
    chain_begin();
    constexpr int kGroups = kFlowThreads / kWindowTokens;
    __shared__ float kept[kWindowTokens][kKeptChunks + 1];
    __shared__ __align__(16) float rows[kFlowWarps][5][kWarpCols];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t N = static_cast<int64_t>(H) * W;
    const int64_t b2 = blockIdx.y, i0 = static_cast<int64_t>(blockIdx.x) * kWindowTokens;
    const bool cols = b2 >= B;
    const int n = cols ? bands : chunks, width = cols ? band_rows : kPoolCols;
    const float *maxima = (cols ? col_max + (b2 - B) * bands * N : row_max + b2 * chunks * N) + i0;
    const auto average = [](float sum) { return DT<T>::rnd(__fdiv_rn(sum, 25.f)); };
    {       // eight tokens' maxima of a chunk lie side by side: a thread reads every 32nd chunk of one token, all under way at once
        const int t = threadIdx.x % kWindowTokens, g = threadIdx.x / kWindowTokens;
        if (i0 + t < N) {
#pragma unroll 8
            for (int c = g; c < min(n, kKeptChunks); c += kGroups) kept[t][c] = maxima[static_cast<int64_t>(c) * N + t];
        }
    }
    __syncthreads();
    const int64_t i = i0 + warp;
    if (i >= N) return;
    const T *base = prob + b2 * N * N;
    const auto chunk_max = [&](int c) {
        return c >= n ? 0.f : c < kKeptChunks ? kept[warp][c] : maxima[static_cast<int64_t>(c) * N + warp];
    };
    float top = 0.f;
    for (int c = lane; c < n; c += 32) top = fmaxf(top, chunk_max(c));
    top = warp_max(top);
    const float least = average(top * (1.f - kScreen));
    const float far = top * kCoarse - kCoarseStep;      // below: rounds to less than `least` whatever the type
    float(*const mine)[kWarpCols] = rows[warp];
    float bv = -INFINITY;
    int bj = 0x7fffffff;
    // boxes of PER neighbouring targets per lane, each summed in the deciding order
    const auto pool = [&](auto per, int64_t first) {
        constexpr int PER = decltype(per)::value;
        if (lane * PER >= width) return;
        float sum[PER];
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            float p[PER + 4];
            if constexpr (PER == 4) {
                const float4 a = *reinterpret_cast<const float4 *>(&mine[d][4 * lane]), c = *reinterpret_cast<const float4 *>(&mine[d][4 * lane + 4]);
                p[0] = a.x; p[1] = a.y; p[2] = a.z; p[3] = a.w; p[4] = c.x; p[5] = c.y; p[6] = c.z; p[7] = c.w;
            } else if constexpr (PER == 2) {
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const float2 a = *reinterpret_cast<const float2 *>(&mine[d][2 * lane + 2 * e]);
                    p[2 * e] = a.x;
                    p[2 * e + 1] = a.y;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 5; ++e) p[e] = mine[d][lane + e];
            }
#pragma unroll
            for (int k = 0; k < PER; ++k)
#pragma unroll
                for (int e = 0; e < 5; ++e) sum[k] = d == 0 && e == 0 ? p[k] : sum[k] + p[k + e];
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int c = lane * PER + k;
            const float v = average(sum[k]);
            if (c < width && first + c < N && v > bv) {
                bv = v;
                bj = static_cast<int>(first) + c;
            }
        }
    };
    for (int c0 = 0; c0 < n; c0 += 32) {
        const float m = chunk_max(c0 + lane);
        if (!__any_sync(0xffffffffu, !(m < far))) continue;
        unsigned pass = __ballot_sync(0xffffffffu, c0 + lane < n && average(m * (1.f + kScreen)) >= least);
        for (; pass != 0; pass &= pass - 1) {
            const int64_t first = static_cast<int64_t>(c0 + __ffs(pass) - 1) * width, j0 = first - 2 + lane;
            const T *at = base + (i - 2) * N + j0;
            for (int c = lane; c < width + 4; c += 32, at += 32) {
                const int64_t j = first - 2 + c;
                const bool in = j >= 0 && j < N;
#pragma unroll
                for (int d = 0; d < 5; ++d) mine[d][c] = in && i + d >= 2 && i + d - 2 < N ? load_one<T>(at + d * N) : 0.f;
            }
            __syncwarp();
            if (width <= 32) pool(std::integral_constant<int, 1>(), first);
            else if (width <= 64) pool(std::integral_constant<int, 2>(), first);
            else pool(std::integral_constant<int, 4>(), first);
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {      // larger value wins, equal values keep the smaller index
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
        if (ov > bv || (ov == bv && oj < bj)) {
            bv = ov;
            bj = oj;
        }
    }
    const int cy = min(max(bj / W, 2), H - 3), cx = min(max(bj % W, 2), W - 3);
    const float mean = DT<T>::rnd(static_cast<float>(1.0 / static_cast<double>(N)));   // the scalar is converted to T first
    const int tx = cx + lane % 5 - 2, ty = cy + lane / 5 - 2;
    float p = lane < 25 ? load_one<T>(base + i * N + static_cast<int64_t>(ty) * W + tx) : 0.f;
    if (p < mean) p = 0.f;
    // sums of 25 in order, the terms read back four at a time
    const auto sum_25 = [](const float *v) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < 24; k += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(v + k);
            sum += q.x; sum += q.y; sum += q.z; sum += q.w;
        }
        return sum + v[24];
    };
    mine[0][lane] = p;
    __syncwarp();
    const float sum = fmaxf(DT<T>::rnd(sum_25(mine[0])), tiny);
    const float np = DT<T>::rnd(__fdiv_rn(p, sum));
    mine[1][lane] = DT<T>::rnd(np * DT<T>::rnd(static_cast<float>(tx)));
    mine[2][lane] = DT<T>::rnd(np * DT<T>::rnd(static_cast<float>(ty)));
    __syncwarp();
    const int64_t at = b2 * N + i;
    const int qy = static_cast<int>(i / W), qx = static_cast<int>(i - static_cast<int64_t>(qy) * W);
    if (lane < 2)       // x, y
        store_one<T>(flow + at * 2 + lane, DT<T>::rnd(DT<T>::rnd(sum_25(mine[1 + lane])) - DT<T>::rnd(static_cast<float>(lane == 0 ? qx : qy))));
    if (lane == 0) {
        if (centre_out != nullptr) centre_out[at] = cy * W + cx;
        if (blur_max != nullptr) store_one<T>(blur_max + at, bv);
    }
}

template <typename T, int ALIGN>
cudaError_t run_flow_kernels(const FlowPlan &pl, const T *corr, T *prob, T *flow, T *blur, int *centre, char *scratch, int B, int H,
                             int W, float tiny, cudaStream_t stream)
{
    const int64_t N = pl.N;
    float *row_part = reinterpret_cast<float *>(scratch), *col_part = reinterpret_cast<float *>(scratch + pl.off_col);
    float2 *stats = reinterpret_cast<float2 *>(scratch + pl.off_stats);
    float *row_max = reinterpret_cast<float *>(scratch + pl.off_row_max), *col_max = reinterpret_cast<float *>(scratch + pl.off_col_max);
    const int64_t units = static_cast<int64_t>(pl.row_parts) * pl.col_parts;
    launch_chained(flow_max_kernel<T, ALIGN>, dim3(static_cast<unsigned>((units + kFlowWarps - 1) / kFlowWarps), B), kFlowThreads, 0, stream, 
        corr, row_part, col_part, N, pl.max_rows, pl.row_parts, pl.col_parts);
    const auto launch_sums = [&](auto kernel, int columns, int threads, int bytes) {
        const int col_blocks = static_cast<int>((N + columns - 1) / columns), rows = threads / 32;
        launch_chained(kernel, dim3(static_cast<unsigned>(col_blocks + (N + rows - 1) / rows), B), threads, bytes, stream, corr, row_part, col_part, stats, N,
                       pl.row_parts, pl.col_parts, col_blocks);
    };
    if constexpr (ALIGN == 1 && sizeof(T) == 2) {
        if (N >= kWideStrided) launch_sums(flow_sum_strided_kernel<T, 32, 16>, 32, 32 * kSumGroups, 0);
        else launch_sums(flow_sum_strided_kernel<T, 16, 32>, 16, 16 * kSumGroups, 0);
    } else {
        if (N >= (ALIGN == 1 ? kWideOdd : kWideSums<T>)) launch_sums(flow_sum_kernel<T, ALIGN, 32>, 32, kFlowThreads, SumTile<32>::kBytes);
        else launch_sums(flow_sum_kernel<T, ALIGN, 16>, 16, kFlowThreads, SumTile<16>::kBytes);
    }
    constexpr int smem = kPoolWarps * kPoolSmemPerWarp;
    const cudaError_t e = cudaFuncSetAttribute(flow_prob_pool_kernel<T, ALIGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int64_t regions = static_cast<int64_t>((pl.bands + kPoolWarps - 1) / kPoolWarps) * ((pl.chunks + kPoolWarps - 1) / kPoolWarps);
    launch_chained(flow_prob_pool_kernel<T, ALIGN>, dim3(static_cast<unsigned>(regions * 2 * kPoolWarps), B), 32 * kPoolWarps, smem, stream, 
        corr, prob, PoolParams{stats, row_max, col_max, N, B, pl.band, pl.chunks, pl.bands});
    launch_chained(flow_window_kernel<T>, dim3(static_cast<unsigned>((N + kWindowTokens - 1) / kWindowTokens), 2 * B), kFlowThreads, 0, stream, 
        prob, row_max, col_max, flow, blur, centre, B, H, W, pl.chunks, pl.bands, pl.band, tiny);
    return cudaGetLastError();
}

template <typename T>
cudaError_t run_flow_init(const void *corr_, void *prob_, void *flow_, void *blur_, int *centre, void *scratch, int B, int H,
                          int W, float tiny, cudaStream_t stream)
{
    const FlowPlan pl = flow_plan(B, H, W);
    const T *corr = static_cast<const T *>(corr_);
    T *prob = static_cast<T *>(prob_), *flow = static_cast<T *>(flow_), *blur = static_cast<T *>(blur_);
    char *ws = static_cast<char *>(scratch);
    // Every row of corr and prob starts at a multiple of ALIGN elements; the loads and stores are that wide, up to 16
    // bytes.  Measured, float16, 2-byte accesses before: 101x100 tokens 652 -> 459 us (4), 82x79 344 -> 251 (2); float32
    // 78x86 335 -> 297 (4).  Odd token counts keep the single elements.
    const auto aligned_to = [&](int elements) {
        const uintptr_t bytes = elements * sizeof(T);
        return pl.N % elements == 0 && reinterpret_cast<uintptr_t>(corr_) % bytes == 0 && reinterpret_cast<uintptr_t>(prob_) % bytes == 0;
    };
    const auto run = [&](auto align) {
        return run_flow_kernels<T, decltype(align)::value>(pl, corr, prob, flow, blur, centre, ws, B, H, W, tiny, stream);
    };
    if constexpr (sizeof(T) == 2) {
        if (aligned_to(8)) return run(std::integral_constant<int, 8>());
        if (aligned_to(4)) return run(std::integral_constant<int, 4>());
        if (aligned_to(2)) return run(std::integral_constant<int, 2>());
    } else {
        if (aligned_to(4)) return run(std::integral_constant<int, 4>());
    }
    return run(std::integral_constant<int, 1>());
}

}  // namespace
}  // namespace matchattn

extern "C" size_t matchattn_flow_init_scratch_bytes(int B, int H, int W)
{
    if (B <= 0 || H <= 0 || W <= 0) return 0;
    return matchattn::flow_plan(B, H, W).bytes;
}

extern "C" int matchattn_flow_init(const void *correlation, void *prob, void *flow, void *blur_max, int *centre,
                                   void *scratch, size_t scratch_bytes, int B, int H, int W, int dtype, void *cuda_stream)
{
    if (!correlation || !prob || !flow || !scratch) return MATCHATTN_ERR_NULL;
    if (B <= 0 || H < 5 || W < 5) return MATCHATTN_ERR_SHAPE;
    const long long N = 1LL * H * W;
    if (N > 65535LL * 32 || 2LL * B > 65535 || N >= (1LL << 31)) return MATCHATTN_ERR_TOO_LARGE;
    if (scratch_bytes < matchattn_flow_init_scratch_bytes(B, H, W) || (reinterpret_cast<uintptr_t>(scratch) & 15))
        return MATCHATTN_ERR_ALIGN;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    cudaError_t err;
    switch (dtype) {
    case MATCHATTN_F32: err = matchattn::run_flow_init<float>(correlation, prob, flow, blur_max, centre, scratch, B, H, W, 1.17549435e-38f, stream); break;
    case MATCHATTN_F16: err = matchattn::run_flow_init<__half>(correlation, prob, flow, blur_max, centre, scratch, B, H, W, 6.103515625e-05f, stream); break;
    case MATCHATTN_BF16: err = matchattn::run_flow_init<__nv_bfloat16>(correlation, prob, flow, blur_max, centre, scratch, B, H, W, 1.17549435e-38f, stream); break;
    default: return MATCHATTN_ERR_DTYPE;
    }
    return matchattn::status_of(err);
}
