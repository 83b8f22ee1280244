// Cost volume of the stereo branch of GlobalCorrelation (models/cost_volume.py:26-51) as one kernel.
//
//   corr [B, H, W, W]  (reference column, then target column, of one image row)
//   vol  [2B, D = W, H, W]
//     left  view: vol[b, d, h, w]   = corr[b, h, w, w-d]  (w >= d, else 0)
//     right view: vol[B+b, d, h, w] = corr[b, h, w+d, w]  (w+d < W, else 0)
//   softmax over d, then the out-of-view fill (left: columns w < d take column d; right: columns
//   w > W-1-d take column W-1-d).
//
// The reference builds this with two Python loops over the W disparities (2 x W slice assignments,
// W more for the fill: about 300 tiny launches at W = 48) around a softmax.  Here one block owns one
// (view, batch item, row) and keeps the row's scores in shared memory, column by column of vol: scores[w][d], as either
// view sees them.  A warp takes the maximum and the exponentials of a column (the pairs out of view score 0), a thread
// their sum in the order of d, then the W rows of W outputs leave coalesced along w.
// HBM traffic: corr once per view, vol once.  Latency-bound (136 blocks at 68 x 120): three steps between barriers, every
// load of a warp under way at once, everything but the W additions of a column's sum spread over the whole block.
// Measured, float16, 68 x 120: 6.6 us (the maxima, the exponentials and their places in five steps 9.0; one thread per
// column for all of it 29.5); 8 x 159 x 128 x 159 63.8 -> 51.1.
#include "../../include/matchattn.h"

#include <stdint.h>

#include <type_traits>

#include "matchattn_kernels.cuh"

namespace matchattn {
namespace {

constexpr int kVolumeMaxW = 159;

// pitch of a column of scores in shared memory: odd (a row of vol walks the columns), P - 1 = 2 mod 4 (the right view's scores
// of a row of corr arrive on a diagonal)
__host__ __device__ constexpr int volume_pitch(int W) { return W / 4 * 4 + 3; }

// maximum over a warp in one instruction (PTX ISA 8.6, sm_100a)
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// PIECES: W / 32 rounded up (a warp takes a row of corr, a column or a row of vol in that many pieces at once)
// WARPS: of a block, ROWS: W / WARPS rounded up, rows or columns per warp
template <typename T, int PIECES, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 2) stereo_volume_kernel(const T *corr, T *__restrict__ vol, int B, int H, int W)
{
    chain_begin();
    constexpr int ROWS = (32 * PIECES + WARPS - 1) / WARPS;
    extern __shared__ float scores[];             // [W][P]: scores[w][d], then exp(score - maximum of its column)
    const int P = volume_pitch(W);
    float *inv = scores + W * P;                  // per column: reciprocal of the sum
    const int h = blockIdx.x, b2 = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool right = b2 >= B;
    const int b = right ? b2 - B : b2;
    const T *src = corr + (static_cast<int64_t>(b) * H + h) * W * W;
    // element (r, j) of the row's correlation, j <= r: disparity r - j at column r of the left view, column j of the right one
    float x[ROWS][PIECES];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int r = warp + i * WARPS, j = lane + 32 * k;
            if (r < W && j <= r) x[i][k] = load_one<T>(src + r * W + j);
        }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int r = warp + i * WARPS, j = lane + 32 * k;
            if (r < W && j <= r) scores[(right ? j : r) * P + r - j] = x[i][k];
        }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int w = warp + i * WARPS;
        if (w >= W) break;
        const int seen = right ? W - w : w + 1;   // disparities in view; the others score 0
        float *column = scores + w * P + lane;
        float m = seen < W ? 0.f : -INFINITY;
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int d = lane + 32 * k;
            x[i][k] = d < seen ? column[32 * k] : 0.f;
            if (d < seen) m = fmaxf(m, x[i][k]);
        }
        m = warp_max(m);
#pragma unroll
        for (int k = 0; k < PIECES; ++k)
            if (lane + 32 * k < W) column[32 * k] = expf(x[i][k] - m);
    }
    __syncthreads();
    for (int w = tid; w < W; w += 32 * WARPS) {
        const float *column = scores + w * P;
        float den = 0.f;
        int d = 0;
        for (; d + 8 <= W; d += 8) {
            float e[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) e[k] = column[d + k];
#pragma unroll
            for (int k = 0; k < 8; ++k) den += e[k];
        }
        for (; d < W; ++d) den += column[d];
        inv[w] = __frcp_rn(den);
    }
    __syncthreads();
    T *dst = vol + (static_cast<int64_t>(b2) * W * H + h) * W;
    const int64_t step = static_cast<int64_t>(H) * W;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int d = warp + i * WARPS;
        if (d >= W) break;
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int w = lane + 32 * k;
            if (w >= W) break;
            const int from = right ? min(w, W - 1 - d) : max(w, d);       // the fill: columns out of view repeat the last one in view
            store_one<T>(dst + d * step + w, scores[from * P + d] * inv[from]);
        }
    }
}

template <typename T>
cudaError_t launch(const void *corr, void *vol, int B, int H, int W, cudaStream_t stream)
{
    const int smem = static_cast<int>(sizeof(float)) * (W * volume_pitch(W) + W);
    const auto go = [&](auto pieces, auto warps) {
        const auto kernel = stereo_volume_kernel<T, decltype(pieces)::value, decltype(warps)::value>;
        if (smem > 48 * 1024) {     // per-device attribute of the kernel: set on every launch (cheap, idempotent, thread-safe)
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
        }
        launch_chained(kernel, dim3(H, 2 * B), 32 * decltype(warps)::value, smem, stream, static_cast<const T *>(corr), static_cast<T *>(vol), B, H, W);
        return cudaGetLastError();
    };
    // as many warps as there are rows to share out, within what two blocks per SM can hold
    using Few = std::integral_constant<int, 16>;
    using Many = std::integral_constant<int, 32>;
    switch ((W + 31) / 32) {
    case 1: return go(std::integral_constant<int, 1>(), Few());
    case 2: return go(std::integral_constant<int, 2>(), Few());
    case 3: return go(std::integral_constant<int, 3>(), Many());
    case 4: return go(std::integral_constant<int, 4>(), Many());
    default: return go(std::integral_constant<int, 5>(), Many());
    }
}

}  // namespace
}  // namespace matchattn

extern "C" int matchattn_stereo_volume(const void *correlation, void *volume, int B, int H, int W, int dtype,
                                       void *cuda_stream)
{
    if (!correlation || !volume) return MATCHATTN_ERR_NULL;
    if (B <= 0 || H <= 0 || W <= 0) return MATCHATTN_ERR_SHAPE;
    if (W > matchattn::kVolumeMaxW || 2LL * B > 65535) return MATCHATTN_ERR_TOO_LARGE;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    cudaError_t err;
    switch (dtype) {
    case MATCHATTN_F32: err = matchattn::launch<float>(correlation, volume, B, H, W, stream); break;
    case MATCHATTN_F16: err = matchattn::launch<__half>(correlation, volume, B, H, W, stream); break;
    case MATCHATTN_BF16: err = matchattn::launch<__nv_bfloat16>(correlation, volume, B, H, W, stream); break;
    default: return MATCHATTN_ERR_DTYPE;
    }
    return matchattn::status_of(err);
}
