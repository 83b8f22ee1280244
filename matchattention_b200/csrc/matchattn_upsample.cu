// Convex upsampling of a field: MatchStereo.upsample_field of the reference
// (models/match_stereo.py:73-84) as one kernel.
//
//   field [B, H, W, D], mask [B, 9*f*f, H, W]  ->  out [B, f*H, f*W, D]
//   out[b, h*f+i, w*f+j, d] = sum_k softmax_k(mask[b, (k*f+i)*f+j, h, w]) * (f * field[b, h+ky-1, w+kx-1, d])
//
// The reference does this with a view, a softmax, an unfold, a broadcast multiply that materialises
// a [B, D, 9, f, f, H, W] tensor, a sum and a permute: about six passes over 4-5x the data.  Here one
// thread owns one coarse cell (b, h, w): it reads its 9*f*f mask logits (each a coalesced read across
// the threads of a warp, the mask is the bulk of the traffic and is read exactly once), the 3x3
// neighbourhood of the field, and writes the f x f block of fine cells.  HBM-bound: 9*f*f + ~D reads and
// f*f*D writes per thread.  Rounding in the 16-bit types follows eager PyTorch: softmax result, field*f
// and every product rounded to the tensor type, nine-term sum in float32.
#include "../../include/matchattn.h"

#include <stdint.h>

#include <type_traits>

#include "matchattn_kernels.cuh"

namespace matchattn {
namespace {

constexpr int kMaxD = 8;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float exp2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// exp(l - top), top the largest logit: one way per type, whatever the width, the address or the kernel.  float32: expf.  The
// 16-bit types round the weight to the type right after and take the special-function unit alone; bfloat16 takes the
// difference first, since log2e times a logit near its largest value overflows, which float16 is far from (the rounding of
// top * log2e is a factor common to the nine weights).  Relative error of the result against 64 bits, 2 x 384x384 by 4:
// float16 3.597e-4 and bfloat16 2.875e-3, with expf the same; float32 8.55e-8 (8.71e-8 with the special-function unit).
template <typename T>
__device__ __forceinline__ float weight_exp(float l, float top)
{
    if constexpr (sizeof(T) == 4) return expf(l - top);
    else if constexpr (std::is_same_v<T, __half>) return exp2_approx(fmaf(l, kLog2e, top * -kLog2e));
    else return exp2_approx((l - top) * kLog2e);
}
template <typename T>
__device__ __forceinline__ float2 weight_exp(float2 l, float2 top)
{
    const float2 log2e = make_float2(kLog2e, kLog2e);
    float2 t;
    if constexpr (std::is_same_v<T, __half>) {
        t = fma_f32x2(l, log2e, make_float2(top.x * -kLog2e, top.y * -kLog2e));
    } else {
        t = add_f32x2(l, make_float2(-top.x, -top.y));
        if constexpr (sizeof(T) == 4) return make_float2(expf(t.x), expf(t.y));
        t = mul_f32x2(t, log2e);
    }
    return make_float2(exp2_approx(t.x), exp2_approx(t.y));
}

template <typename T, int F>
__global__ void __launch_bounds__(128) upsample_field_kernel(const T *field, const T *mask,
                                                             T *__restrict__ out, int B, int H, int W, int D)
{
    chain_begin();
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y, b = blockIdx.z;
    if (w >= W) return;
    const int64_t plane = static_cast<int64_t>(H) * W;

    // 3x3 neighbourhood of the field, times f, rounded to T; zero outside the map
    float nb[9][kMaxD];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int hh = h + k / 3 - 1, ww = w + k % 3 - 1;
        const bool inside = hh >= 0 && hh < H && ww >= 0 && ww < W;
        const T *src = field + ((static_cast<int64_t>(b) * H + (inside ? hh : h)) * W + (inside ? ww : w)) * D;
#pragma unroll
        for (int d = 0; d < kMaxD; ++d)
            nb[k][d] = (inside && d < D) ? DT<T>::rnd(load_one<T>(src + d) * static_cast<float>(F)) : 0.f;
    }

    const T *mrow = mask + static_cast<int64_t>(b) * 9 * F * F * plane + static_cast<int64_t>(h) * W + w;
    // the logits of a fine cell are asked for before the cell ahead of it is stored: loads do not pass stores
    float next[9];
    const auto ask = [&](int cell) {
#pragma unroll
        for (int k = 0; k < 9; ++k) next[k] = load_one<T>(mrow + static_cast<int64_t>(k * F * F + cell) * plane);
    };
    ask(0);
    for (int i = 0; i < F; ++i) {
        T *orow = out + ((static_cast<int64_t>(b) * H * F + static_cast<int64_t>(h) * F + i) * W * F + static_cast<int64_t>(w) * F) * D;
#pragma unroll
        for (int j = 0; j < F; ++j) {
            float p[9];
            float mx = -INFINITY;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                p[k] = next[k];
                mx = fmaxf(mx, p[k]);
            }
            if (i * F + j + 1 < F * F) ask(i * F + j + 1);
            float den = 0.f;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                p[k] = weight_exp<T>(p[k], mx);
                den += p[k];
            }
            const float inv = __frcp_rn(den);
#pragma unroll
            for (int k = 0; k < 9; ++k) p[k] = DT<T>::rnd(p[k] * inv);
#pragma unroll
            for (int d = 0; d < kMaxD; ++d) {
                if (d >= D) break;
                float acc = 0.f;
#pragma unroll
                for (int k = 0; k < 9; ++k) acc += DT<T>::rnd(p[k] * nb[k][d]);
                store_one<T>(orow + j * D + d, acc);
            }
        }
    }
}

// a packed 32-bit word of two 16-bit values as the pair type of the element-wise helpers
template <typename T>
__device__ __forceinline__ typename DT<T>::Bcast word_as_pair(uint32_t w);
template <>
__device__ __forceinline__ __half2 word_as_pair<__half>(uint32_t w) { return *reinterpret_cast<const __half2 *>(&w); }
template <>
__device__ __forceinline__ __nv_bfloat162 word_as_pair<__nv_bfloat16>(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162 *>(&w); }


// element-wise maximum of two pairs
__device__ __forceinline__ __half2 pair_max(__half2 a, __half2 b) { return __hmax2(a, b); }
__device__ __forceinline__ __nv_bfloat162 pair_max(__nv_bfloat162 a, __nv_bfloat162 b) { return __hmax2(a, b); }
template <typename P>
__device__ __forceinline__ uint32_t pair_word(P p) { return *reinterpret_cast<const uint32_t *>(&p); }

// Nine logits of two cells as loaded: a word of two neighbours, or two values, which stay apart (put into a word first, 2 x 543x541
// by 4 took 66 us in float16 and 106 in bfloat16, now 62 and 63).
template <typename T, bool EVEN>
struct Logits {
    uint32_t w[9];
    __device__ __forceinline__ void load(int k, const T *at, int w0, int) { w[k] = *reinterpret_cast<const uint32_t *>(at + w0); }
    __device__ __forceinline__ float2 get(int k) const { return make_float2(DT<T>::unpack(w[k], 0), DT<T>::unpack(w[k], 1)); }
    __device__ __forceinline__ float2 top() const
    {
        typename DT<T>::Bcast top = word_as_pair<T>(w[0]);
#pragma unroll
        for (int k = 1; k < 9; ++k) top = pair_max(top, word_as_pair<T>(w[k]));
        const uint32_t tw = pair_word(top);
        return make_float2(DT<T>::unpack(tw, 0), DT<T>::unpack(tw, 1));
    }
};
template <typename T>
struct Logits<T, false> {
    T a[9], b[9];
    __device__ __forceinline__ void load(int k, const T *at, int w0, int w1)
    {
        a[k] = at[w0];
        b[k] = at[w1];
    }
    __device__ __forceinline__ float2 get(int k) const { return make_float2(static_cast<float>(a[k]), static_cast<float>(b[k])); }
    __device__ __forceinline__ float2 top() const
    {
        T ta = a[0], tb = b[0];
#pragma unroll
        for (int k = 1; k < 9; ++k) {
            ta = __hmax(ta, a[k]);
            tb = __hmax(tb, b[k]);
        }
        return make_float2(static_cast<float>(ta), static_cast<float>(tb));
    }
};

// One fine row of two cells: softmax of the logits at m0, weighted sums of the neighbours' components, F fine cells to either.
// (place: gives the row's output, asked for at the end: one row per thread needs no register for it before that)
template <typename T, int F, bool EVEN, typename Place>
__device__ __forceinline__ void fine_row(const T *m0, Place place, const uint32_t (&nx)[9], const uint32_t (&ny)[9], int w0, int w1, bool second, int64_t plane)
{
    uint32_t o0[F], o1[F];
#pragma unroll
    for (int j = 0; j < F; ++j) {
        Logits<T, EVEN> logits;
#pragma unroll
        for (int k = 0; k < 9; ++k) logits.load(k, m0 + static_cast<int64_t>(k * F * F + j) * plane, w0, w1);
        const float2 mx = logits.top();
        float2 p[9], den;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            p[k] = weight_exp<T>(logits.get(k), mx);
            den = k == 0 ? p[0] : add_f32x2(den, p[k]);
        }
        const float2 inv = make_float2(__frcp_rn(den.x), __frcp_rn(den.y));
        float sx[2] = {0.f, 0.f}, sy[2] = {0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const float2 q = mul_f32x2(p[k], inv);
            const typename DT<T>::Bcast w = word_as_pair<T>(DT<T>::aw_from(q.x, q.y));
            DT<T>::wmul(w, nx[k], sx);
            DT<T>::wmul(w, ny[k], sy);
        }
        o0[j] = DT<T>::aw_from(sx[0], sy[0]);
        o1[j] = DT<T>::aw_from(sx[1], sy[1]);
    }
    uint32_t *row = place();
    if constexpr (F == 4) {
        st_128(row + static_cast<int64_t>(w0) * F, o0);
        if (second) st_128(row + static_cast<int64_t>(w1) * F, o1);
    } else {
        st_64(row + static_cast<int64_t>(w0) * F, o0);
        if (second) st_64(row + static_cast<int64_t>(w1) * F, o1);
    }
}

// 16-bit types, two-component fields (the model's), factors 2 and 4, any width.  A thread owns two cells of a row and
// ROWS fine rows, one after the other, and takes them through everything in pairs: a weight word holds both cells' weights,
// multiplied by the pair of their neighbours' components, packed float32 arithmetic in between.  EVEN: the two cells are
// neighbours and a mask read is one word; otherwise they lie 32 apart, so that a warp's 2-byte reads are contiguous.  A cell's
// F fine cells are one aligned store of 8 or 16 bytes.
// Two rows share the neighbours and their addresses; one is half as long where the blocks do not fill the chip (pair_rows).
// Two: issue 65 %, then the latency of the mask reads (4.7 stalls per issue).  Measured, float16, 2 x 384x384 by 4: 27.3 us
// (one row 28.9, two without the limit of 64 registers 54, four cells and five blocks per SM 33); by 2 9.1 (10.5).
template <typename T, int F, bool EVEN, int ROWS>
__global__ void __launch_bounds__(128, ROWS == 1 ? 0 : 8) upsample_pair_kernel(const T *field, const T *mask, T *__restrict__ out,
                                                            int B, int H, int W, int segments)
{
    chain_begin();
    constexpr int G = F / ROWS;                    // threads' shares of a cell
    constexpr int COLS = EVEN ? 4 : 6;             // columns of neighbours: -1 .. 2 around the pair, or -1 .. 1 around either
    const int lane = threadIdx.x & 31;
    const uint32_t warp = blockIdx.x * 4u + (threadIdx.x >> 5);
    const uint32_t line = warp / static_cast<uint32_t>(segments);              // b, ROWS fine rows
    const int w0 = static_cast<int>(warp - line * segments) * 64 + (EVEN ? 2 * lane : lane);
    const uint32_t b = line / static_cast<uint32_t>(H * G);
    if (b >= static_cast<uint32_t>(B) || w0 >= W) return;
    const int hi = static_cast<int>(line - b * (H * G)), h = hi / G, i0 = (hi - h * G) * ROWS;
    const int w1 = EVEN ? w0 + 1 : min(w0 + 32, W - 1);
    const bool second = EVEN || w0 + 32 < W;
    const int64_t plane = static_cast<int64_t>(H) * W;

    // neighbours times F, rounded to T, zero outside the map: the pair of x and the pair of y components per tap
    uint32_t nx[9], ny[9];
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(field) + b * plane;
        const uint32_t factor = DT<T>::aw_bcast(static_cast<float>(F));
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            const int hh = h + ky - 1;
            uint32_t v[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const int ww = EVEN || c < 3 ? w0 + c - 1 : w1 + c - 4;
                const bool inside = hh >= 0 && hh < H && ww >= 0 && ww < W;
                v[c] = inside ? DT<T>::aw_mul(src[hh * W + ww], factor) : 0u;
            }
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
                nx[3 * ky + kx] = __byte_perm(v[kx], v[EVEN ? kx + 1 : kx + 3], 0x5410);
                ny[3 * ky + kx] = __byte_perm(v[kx], v[EVEN ? kx + 1 : kx + 3], 0x7632);
            }
        }
    }

    const T *m0 = mask + static_cast<int64_t>(b) * 9 * F * F * plane + static_cast<int64_t>(i0) * F * plane + static_cast<int64_t>(h) * W;
    if constexpr (ROWS == 1) {
        fine_row<T, F, EVEN>(m0, [&] { return reinterpret_cast<uint32_t *>(out) + static_cast<int64_t>(line) * W * F; }, nx, ny, w0, w1, second, plane);
    } else {
        uint32_t *row = reinterpret_cast<uint32_t *>(out) + static_cast<int64_t>(line) * ROWS * W * F;
#pragma unroll 1
        for (int i = 0; i < ROWS; ++i, m0 += F * plane, row += static_cast<int64_t>(W) * F)
            fine_row<T, F, EVEN>(m0, [row] { return row; }, nx, ny, w0, w1, second, plane);
    }
}

// float32, two-component fields, factors 2 and 4, even widths: a thread owns two neighbouring cells of a row and ONE fine
// row i, as above; the cells go through the softmax and the components through the sums in pairs (packed float32
// arithmetic), and its 2*F fine cells are one contiguous run of the output row, stored 16 bytes at a time.
// Measured, 2 x 384x384 by 4: 43.8 us (four cells per thread, exponentials by the special-function unit alone: 47.7; with
// expf 50.7, in pairs 64.2 at 137 registers); 2 x 201x302 by 4: 22.7 (one cell and all its fine rows per thread: 55.5).
template <int F>
__global__ void __launch_bounds__(128) upsample_f32_kernel(const float *field, const float *mask,
                                                           float *__restrict__ out, int B, int H, int W, int segments)
{
    chain_begin();
    const uint32_t warp = blockIdx.x * 4u + (threadIdx.x >> 5);
    const uint32_t line = warp / static_cast<uint32_t>(segments);              // b, fine row
    const int w0 = static_cast<int>(warp - line * segments) * 64 + 2 * (threadIdx.x & 31);
    const uint32_t b = line / static_cast<uint32_t>(H * F);
    if (b >= static_cast<uint32_t>(B) || w0 >= W) return;
    const int hi = static_cast<int>(line - b * (H * F)), h = hi / F, i = hi - h * F;
    const int64_t plane = static_cast<int64_t>(H) * W;

    // neighbours times F in columns w0 - 1 .. w0 + 2, zero outside the map
    float2 nb[3][4];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
        const int hh = h + ky - 1;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int ww = w0 + c - 1;
            const bool inside = hh >= 0 && hh < H && ww >= 0 && ww < W;
            const float *src = field + (b * plane + (inside ? static_cast<int64_t>(hh) * W + ww : 0)) * 2;
            nb[ky][c] = inside ? make_float2(load_one<float>(src) * F, load_one<float>(src + 1) * F) : make_float2(0.f, 0.f);
        }
    }

    const float *m0 = mask + static_cast<int64_t>(b) * 9 * F * F * plane + static_cast<int64_t>(i) * F * plane + static_cast<int64_t>(h) * W + w0;
    float2 first[F], second[F];
#pragma unroll
    for (int j = 0; j < F; ++j) {
        float2 p[9], den;
#pragma unroll
        for (int k = 0; k < 9; ++k) p[k] = *reinterpret_cast<const float2 *>(m0 + static_cast<int64_t>(k * F * F + j) * plane);
        float2 mx = p[0];
#pragma unroll
        for (int k = 1; k < 9; ++k) mx = make_float2(fmaxf(mx.x, p[k].x), fmaxf(mx.y, p[k].y));
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            p[k] = weight_exp<float>(p[k], mx);
            den = k == 0 ? p[0] : add_f32x2(den, p[k]);
        }
        const float2 inv = make_float2(__frcp_rn(den.x), __frcp_rn(den.y));
        first[j] = second[j] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const float2 q = mul_f32x2(p[k], inv);
            first[j] = fma_f32x2(make_float2(q.x, q.x), nb[k / 3][k % 3], first[j]);
            second[j] = fma_f32x2(make_float2(q.y, q.y), nb[k / 3][k % 3 + 1], second[j]);
        }
    }
    float4 *row = reinterpret_cast<float4 *>(out + (static_cast<int64_t>(line) * W + w0) * F * 2);
#pragma unroll
    for (int j = 0; j < F / 2; ++j) {
        row[j] = make_float4(first[2 * j].x, first[2 * j].y, first[2 * j + 1].x, first[2 * j + 1].y);
        row[F / 2 + j] = make_float4(second[2 * j].x, second[2 * j].y, second[2 * j + 1].x, second[2 * j + 1].y);
    }
}

// Fine rows per thread of the kernel for pairs; `blocks`: of a launch with one.  Two pay once the chip is full: one row in even
// widths by 4 is held by 64 registers, eight blocks per SM, in other builds by up to 80, six.  Even by 4, three rounds of one row
// beat two of two.  Measured, one row / two, us, float16, 2 maps: by 4 48x48 3.4 / 5.2, 192x192 (0.97 rounds) 9.1 / 11.4, 200x304
// (1.7) 14.5 / 13.9, 272x272 (2.3) 19.1 / 21.3, 352x352 (3.6) 26.9 / 25.7, 544x544 57.4 / 56.0, 161x161 (1.1 of six) 10.6 / 9.3,
// 96x97 5.3 / 7.0, 543x541 83.7 / 62.4; by 2 192x192 3.5 / 3.7, 240x240 (1.1 of six) 4.8 / 4.5, 96x97 3.4 / 3.9, 201x303 6.2 / 5.6.
int pair_rows(long long blocks, int factor, bool even)
{
    const long long eight = 8LL * sm_count(), held = even && factor == 4 ? eight : eight * 6 / 8;
    if (blocks <= held || (held == eight && (blocks + eight - 1) / eight == 3)) return 1;
    return 2;
}

template <typename T>
cudaError_t launch(const void *field, const void *mask, void *out, int B, int H, int W, int D, int factor,
                   cudaStream_t stream)
{
    const dim3 grid((W + 127) / 128, H, B), block(128);
    const T *f = static_cast<const T *>(field), *m = static_cast<const T *>(mask);
    T *o = static_cast<T *>(out);
    // the model's shapes: a 2-component field, factor 2 between stages and 4 at the end
    const int64_t segments = (W + 63) / 64, warps = segments * H * factor * B;
    const unsigned blocks = static_cast<unsigned>((warps + 3) / 4);
    const int seg = static_cast<int>(segments);
    const bool even = W % 2 == 0 && reinterpret_cast<uintptr_t>(m) % (2 * sizeof(T)) == 0;
    if (D == 2 && (factor == 2 || factor == 4) && (reinterpret_cast<uintptr_t>(o) & 15u) == 0 &&
        static_cast<int64_t>(H) * W < (1LL << 31) && warps < (1LL << 31)) {
        if constexpr (sizeof(T) == 2) {
            if ((reinterpret_cast<uintptr_t>(f) & 3u) == 0) {
                const auto go = [&](auto rows) {
                    constexpr int ROWS = decltype(rows)::value;
                    const auto kernel = even ? (factor == 4 ? upsample_pair_kernel<T, 4, true, ROWS> : upsample_pair_kernel<T, 2, true, ROWS>)
                                             : (factor == 4 ? upsample_pair_kernel<T, 4, false, ROWS> : upsample_pair_kernel<T, 2, false, ROWS>);
                    launch_chained(kernel, (blocks + ROWS - 1) / ROWS, 128, 0, stream, f, m, o, B, H, W, seg);
                };
                if (pair_rows(blocks, factor, even) == 2) go(std::integral_constant<int, 2>());
                else go(std::integral_constant<int, 1>());
                return cudaGetLastError();
            }
        } else if (even) {
            const auto kernel = factor == 4 ? upsample_f32_kernel<4> : upsample_f32_kernel<2>;
            launch_chained(kernel, blocks, 128, 0, stream, f, m, o, B, H, W, seg);
            return cudaGetLastError();
        }
    }
    switch (factor) {
    case 1: launch_chained(upsample_field_kernel<T, 1>, grid, block, 0, stream, f, m, o, B, H, W, D); break;
    case 2: launch_chained(upsample_field_kernel<T, 2>, grid, block, 0, stream, f, m, o, B, H, W, D); break;
    case 4: launch_chained(upsample_field_kernel<T, 4>, grid, block, 0, stream, f, m, o, B, H, W, D); break;
    case 8: launch_chained(upsample_field_kernel<T, 8>, grid, block, 0, stream, f, m, o, B, H, W, D); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace
}  // namespace matchattn

extern "C" int matchattn_upsample_field(const void *field, const void *mask, void *out, int B, int H, int W, int D,
                                        int factor, int dtype, void *cuda_stream)
{
    if (!field || !mask || !out) return MATCHATTN_ERR_NULL;
    if (B <= 0 || H <= 0 || W <= 0 || D <= 0 || D > matchattn::kMaxD) return MATCHATTN_ERR_SHAPE;
    if (factor != 1 && factor != 2 && factor != 4 && factor != 8) return MATCHATTN_ERR_SHAPE;
    if (H > 65535 || B > 65535 || 1LL * B * 9 * factor * factor * H * W >= (1LL << 40)) return MATCHATTN_ERR_TOO_LARGE;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    cudaError_t err;
    switch (dtype) {
    case MATCHATTN_F32: err = matchattn::launch<float>(field, mask, out, B, H, W, D, factor, stream); break;
    case MATCHATTN_F16: err = matchattn::launch<__half>(field, mask, out, B, H, W, D, factor, stream); break;
    case MATCHATTN_BF16: err = matchattn::launch<__nv_bfloat16>(field, mask, out, B, H, W, D, factor, stream); break;
    default: return MATCHATTN_ERR_DTYPE;
    }
    return matchattn::status_of(err);
}
