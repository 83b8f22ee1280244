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
// (view, batch item, row) and keeps the row's W x W correlation slice in shared memory.  Every pair (d, w) in view is
// one element of the slice, the pairs out of view all score 0 and are never written (the fill replaces them), so the
// exponentials are taken in place: maxima by a warp per column, exponentials by all threads over the triangle in
// view, sums by a thread per column (in the order of d), then the W rows of W outputs, coalesced along w.
// HBM traffic: corr once per view, vol once.  Latency-bound (136 blocks at 68 x 120): everything but the W additions
// of a column's sum is spread over the whole block.  Measured, float16, 68 x 120: 8.8 us; one thread per column for
// all three steps took 29.5 us.
#include "../../include/matchattn.h"

#include <stdint.h>

#include <type_traits>

#include "matchattn_kernels.cuh"

namespace matchattn {
namespace {

constexpr int kVolumeMaxW = 159;

// pitch of the slice in shared memory: P + 1 odd (columns walk the diagonals of the slice), P = 2 mod 4 (and its columns)
__host__ __device__ constexpr int volume_pitch(int W) { return (W + 3) / 4 * 4 + 2; }

// PIECES: W / 32 rounded up (a warp takes a row of the slice, or a column of vol, in that many pieces at once)
template <typename T, int PIECES>
__global__ void __launch_bounds__(1024) stereo_volume_kernel(const T *__restrict__ corr, T *__restrict__ vol, int B, int H, int W)
{
    chain_begin();
    extern __shared__ float slice[];              // [W][P]: corr[w][j], then exp(corr - maximum of its column of vol)
    const int P = volume_pitch(W);
    float *top = slice + W * P, *inv = top + W;   // per column w: maximum, reciprocal of the sum
    const int h = blockIdx.x, b2 = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const bool right = b2 >= B;
    const int b = right ? b2 - B : b2;
    const T *src = corr + (static_cast<int64_t>(b) * H + h) * W * W;
    // element (w, j) of the slice: the left view sees it at column w, disparity w - j, the right one at column j
    for (int r0 = warp; r0 < W; r0 += 2 * warps) {        // two rows of a warp in flight
        float x[2][PIECES];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < PIECES; ++k) {
                const int r = r0 + i * warps, j = lane + 32 * k;
                x[i][k] = r < W && j <= r ? load_one<T>(src + r * W + j) : 0.f;
            }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < PIECES; ++k) {
                const int r = r0 + i * warps, j = lane + 32 * k;
                if (r < W && j <= r) slice[r * P + j] = x[i][k];
            }
    }
    __syncthreads();
    for (int w = warp; w < W; w += warps) {
        const int seen = right ? W - w : w + 1;   // disparities in view
        float m = seen < W ? 0.f : -INFINITY;     // those out of view score 0
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int d = lane + 32 * k;
            if (d < seen) m = fmaxf(m, right ? slice[(w + d) * P + w] : slice[w * P + w - d]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) top[w] = m;
    }
    __syncthreads();
    for (int r = warp; r < W; r += warps) {
        float x[PIECES];
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int j = lane + 32 * k;
            x[k] = j <= r ? slice[r * P + j] - top[right ? j : r] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int j = lane + 32 * k;
            if (j <= r) slice[r * P + j] = expf(x[k]);
        }
    }
    __syncthreads();
    for (int w = tid; w < W; w += blockDim.x) {
        const int seen = right ? W - w : w + 1;
        const float *p = slice + w * P + w;
        const int step = right ? P : -1;
        float den = 0.f;
#pragma unroll 8
        for (int d = 0; d < seen; ++d) den += p[d * step];
        const float none = expf(0.f - top[w]);
#pragma unroll 8
        for (int d = seen; d < W; ++d) den += none;
        inv[w] = __frcp_rn(den);
    }
    __syncthreads();
    T *dst = vol + (static_cast<int64_t>(b2) * W * H + h) * W;
    for (int d = warp; d < W; d += warps)
#pragma unroll
        for (int k = 0; k < PIECES; ++k) {
            const int w = lane + 32 * k;
            if (w >= W) break;
            const int from = right ? min(w, W - 1 - d) : max(w, d);       // the fill: columns out of view repeat the last one in view
            const float e = right ? slice[(from + d) * P + from] : slice[from * P + from - d];
            store_one<T>(dst + static_cast<int64_t>(d) * H * W + w, e * inv[from]);
        }
}

template <typename T>
cudaError_t launch(const void *corr, void *vol, int B, int H, int W, cudaStream_t stream)
{
    const int smem = static_cast<int>(sizeof(float)) * (W * volume_pitch(W) + 2 * W);
    const auto go = [&](auto pieces) {
        constexpr int kPieces = decltype(pieces)::value;
        if (smem > 48 * 1024) {     // per-device attribute of the kernel: set on every launch (cheap, idempotent, thread-safe)
            const cudaError_t e = cudaFuncSetAttribute(stereo_volume_kernel<T, kPieces>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
        }
        // as many warps as there are rows to share out, within what two blocks per SM can hold
        const int threads = W > 64 ? 1024 : 512;
        launch_chained(stereo_volume_kernel<T, kPieces>, dim3(H, 2 * B), threads, smem, stream, static_cast<const T *>(corr), static_cast<T *>(vol), B, H, W);
        return cudaGetLastError();
    };
    switch ((W + 31) / 32) {
    case 1: return go(std::integral_constant<int, 1>());
    case 2: return go(std::integral_constant<int, 2>());
    case 3: return go(std::integral_constant<int, 3>());
    case 4: return go(std::integral_constant<int, 4>());
    default: return go(std::integral_constant<int, 5>());
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
    return err == cudaSuccess ? MATCHATTN_OK : MATCHATTN_ERR_CUDA + static_cast<int>(err);
}
