// Backward of the MatchAttention operator.
//
// The reference's native path has no backward (models/match_former_ops.py registers none; the attn_sum
// buffer "for backward" of models/src/match_former_fused_forward.cu:409,495 is never read); only its 'pytorch'
// path can be trained, through autograd over the five functions of models/mat_pytorch_impl.py.  This kernel
// computes what that autograd computes: gradients with respect to q, k, v and max_offset, given the
// gradients of both outputs (out and attn_out: the cross branch feeds the attention weights to its output
// projection, models/attention_blocks.py:95-98).
//
//   s_m   = -scale * sum_c |q_c - k_mc|                         scores of the (2r+2)^2 taps
//   p_t   = softmax of s over sub-window t (t = nw, ne, sw, se)  a_m = sum_t w_t p_tm,  out_c = sum_m a_m v_mc
//   da_m  = sum_c dout_c v_mc + dattn_m                          dv_mc += a_m dout_c
//   ds_m  = sum_t w_t p_tm (da_m - sum_m' p_tm' da_m')           dw_t   = sum_m p_tm da_m
//   dq_c  = -scale sum_m ds_m sign(q_c - k_mc)                   dk_mc += scale ds_m sign(q_c - k_mc)
//   d(max_offset) follows from dw through w = [(1-dx)(1-dy), dx(1-dy), (1-dx)dy, dx dy] (floor has no gradient)
//
// The forward quantities are recomputed (nothing is saved by the forward); all arithmetic in float32 whatever the
// tensor type.  Several queries look at the same token, so dk and dv are sums over queries.  Two ways:
//
//   gathered (matchattn_fused_backward_ws; head widths that are multiples of 8, r = 1 or 2: every model shape)
//     The (query, head) items are bucketed by the origin of their window; one kernel computes dq, d(max_offset) and the
//     coefficients (scale * ds_m, a_m) of every item, another sums them up per token, which finds its contributions in
//     the (2r+2)^2 buckets whose windows cover it.  dk and dv are written once, in the tensor type.
//     Measured on a B200, float16, 384x384 tokens, 8 heads x 16, r = 1, centres spread over +-24 tokens: 353 us in all,
//     against 785 us for the scattered kernel with its clearing and conversion passes (bound by the rate of the
//     reductions at L2).
//   scattered (matchattn_fused_backward; any head width and radius)
//     One thread per item adds its contributions to float32 arrays with atomic adds, on top of what the caller has there.
//     Two kernels: one element at a time, and eight channels at a time with four-float vector reductions for the
//     shapes above.
#include "../../include/matchattn.h"

#include <stdint.h>

#include <initializer_list>
#include <type_traits>

#include "matchattn_kernels.cuh"

namespace matchattn {
namespace {

struct BwdParams {
    const void *mo, *q, *k, *v, *dout, *dattn;   // dattn may be null
    void *dq, *dmo;                               // tensor type; dmo may be null
    float *dk, *dv;                               // float32, pre-zeroed
    int B, H, W, h, hd, C, r, rows, Nq, N;
    float scale;
};

template <typename T>
__global__ void __launch_bounds__(128) backward_kernel(const BwdParams p)
{
    chain_begin();
    const int64_t per_item = static_cast<int64_t>(p.Nq) * p.h;
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= per_item) return;
    const int b = blockIdx.y;
    const int head = static_cast<int>(t % p.h);
    const int64_t bq = static_cast<int64_t>(b) * p.Nq + t / p.h;
    const int r = p.r, side = 2 * r + 2, sub = 2 * r + 1, M = side * side;

    const T *mo = static_cast<const T *>(p.mo) + (bq * p.h + head) * 2;
    const float x = load_one<T>(mo), y = load_one<T>(mo + 1);
    const float xf = floorf(x), yf = floorf(y);
    const float dx = x - xf, dy = y - yf;
    const float wgt[4] = {(1.f - dx) * (1.f - dy), dx * (1.f - dy), (1.f - dx) * dy, dx * dy};
    const int x0 = window_origin(xf, r, p.W) - r, y0 = window_origin(yf, r, p.H) - r;

    const int64_t qoff = bq * p.C + head * p.hd;
    const T *qp = static_cast<const T *>(p.q) + qoff;
    const T *gop = static_cast<const T *>(p.dout) + qoff;
    const int64_t kv_base = static_cast<int64_t>(b) * p.N * p.C + head * p.hd;
    const T *kb = static_cast<const T *>(p.k) + kv_base;
    const T *vb = static_cast<const T *>(p.v) + kv_base;

    // forward: scores, sub-window softmaxes, attention weights; da from dout.v (+ dattn)
    float s[kMaxTaps], a[kMaxTaps], da[kMaxTaps];
    int tok[kMaxTaps];
    for (int j = 0; j < side; ++j) {
        const int ty = min(max(y0 + j, 0), p.H - 1);
        for (int i = 0; i < side; ++i) {
            const int tx = min(max(x0 + i, 0), p.W - 1);
            const int m = j * side + i;
            tok[m] = ty * p.W + tx;
            const T *kp = kb + static_cast<int64_t>(tok[m]) * p.C;
            const T *vp = vb + static_cast<int64_t>(tok[m]) * p.C;
            float l1 = 0.f, dot = 0.f;
            for (int c = 0; c < p.hd; ++c) {
                l1 += fabsf(load_one<T>(qp + c) - load_one<T>(kp + c));
                dot = fmaf(load_one<T>(gop + c), load_one<T>(vp + c), dot);
            }
            s[m] = -l1 * p.scale;
            a[m] = 0.f;
            da[m] = dot;
        }
    }
    if (p.dattn != nullptr) {
        const T *gap = static_cast<const T *>(p.dattn) + (bq * p.h + head) * M;
        for (int m = 0; m < M; ++m) da[m] += load_one<T>(gap + m);
    }
    float ds[kMaxTaps], dw[4];
    for (int m = 0; m < M; ++m) ds[m] = 0.f;
    for (int tq = 0; tq < 4; ++tq) {
        const int oy = tq >> 1, ox = tq & 1;
        float mx = -INFINITY;
        for (int j = 0; j < sub; ++j)
            for (int i = 0; i < sub; ++i) mx = fmaxf(mx, s[(j + oy) * side + i + ox]);
        float den = 0.f;
        for (int j = 0; j < sub; ++j)
            for (int i = 0; i < sub; ++i) den += expf(s[(j + oy) * side + i + ox] - mx);
        const float inv = 1.f / den;
        float pda = 0.f;                                   // sum_m p_tm da_m
        for (int j = 0; j < sub; ++j)
            for (int i = 0; i < sub; ++i) {
                const int m = (j + oy) * side + i + ox;
                const float pr = expf(s[m] - mx) * inv;
                a[m] += wgt[tq] * pr;
                pda = fmaf(pr, da[m], pda);
            }
        dw[tq] = pda;
        for (int j = 0; j < sub; ++j)
            for (int i = 0; i < sub; ++i) {
                const int m = (j + oy) * side + i + ox;
                const float pr = expf(s[m] - mx) * inv;
                ds[m] = fmaf(wgt[tq] * pr, da[m] - pda, ds[m]);
            }
    }

    // gradient of the sampling centre through the bilinear weights
    if (p.dmo != nullptr) {
        T *gmo = static_cast<T *>(p.dmo) + (bq * p.h + head) * 2;
        store_one<T>(gmo, (1.f - dy) * (dw[1] - dw[0]) + dy * (dw[3] - dw[2]));
        store_one<T>(gmo + 1, (1.f - dx) * (dw[2] - dw[0]) + dx * (dw[3] - dw[1]));
    }

    // dq, and the scatter into dk / dv
    T *gq = static_cast<T *>(p.dq) + qoff;
    for (int c = 0; c < p.hd; ++c) {
        const float qc = load_one<T>(qp + c), go = load_one<T>(gop + c);
        float acc = 0.f;
        for (int m0 = 0; m0 < M; m0 += 4) {       // four loads, then what they lead to: loads do not pass the additions
            float kv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) kv[i] = load_one<T>(kb + static_cast<int64_t>(tok[m0 + i]) * p.C + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int m = m0 + i;
                const int64_t off = static_cast<int64_t>(tok[m]) * p.C + c;
                const float d = qc - kv[i];
                const float sg = d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f);
                const float g = p.scale * ds[m] * sg;
                acc -= g;
                if (g != 0.f) atomicAdd(p.dk + kv_base + off, g);
                const float gv = a[m] * go;
                if (gv != 0.f) atomicAdd(p.dv + kv_base + off, gv);
            }
        }
        store_one<T>(gq + c, acc);
    }
}

__device__ __forceinline__ float sign_of(float a, float b)      // sign(a - b), 0 where one of them is no number
{
    float gt, lt;
    asm("set.gt.f32.f32 %0, %1, %2;" : "=f"(gt) : "f"(a), "f"(b));
    asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(lt) : "f"(a), "f"(b));
    return gt - lt;
}

// ---- the same computation for head widths that are multiples of 8 and r = 1 or 2 -----------------------
// Eight channels at a time through 16- or 32-byte loads, the window in registers (R is a template
// argument), and the scatter into dk / dv as four-float vector reductions (red.global.add.v4.f32 through
// atomicAdd(float4 *), a quarter of the scalar kernel's atomic instructions).

template <typename T>
__device__ __forceinline__ void load8(const T *p, float (&f)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float *p, float (&f)[8])
{
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__half>(const __half *p, float (&f)[8])
{
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16 *p, float (&f)[8])
{
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

template <typename T>
__device__ __forceinline__ void store8(T *p, const float (&f)[8]);
template <>
__device__ __forceinline__ void store8<float>(float *p, const float (&f)[8])
{
    reinterpret_cast<float4 *>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
template <>
__device__ __forceinline__ void store8<__half>(__half *p, const float (&f)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 t = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&t);
    }
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16 *p, const float (&f)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&t);
    }
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// (measured: the kernel is bound by the rate of the reductions into dk / dv, L2 throughput 62 % at 18 %
// occupancy; four blocks per SM instead of three change nothing at r = 1 and gain 25 % at r = 2)
template <typename T, int R>
__global__ void __launch_bounds__(128, R == 2 ? 4 : 3) backward_vec_kernel(const BwdParams p)
{
    chain_begin();
    constexpr int SIDE = 2 * R + 2, SUB = 2 * R + 1, M = SIDE * SIDE;
    const int64_t per_item = static_cast<int64_t>(p.Nq) * p.h;
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= per_item) return;
    const int b = blockIdx.y;
    const int head = static_cast<int>(t % p.h);
    const int64_t bq = static_cast<int64_t>(b) * p.Nq + t / p.h;

    const T *mo = static_cast<const T *>(p.mo) + (bq * p.h + head) * 2;
    const float x = load_one<T>(mo), y = load_one<T>(mo + 1);
    const float xf = floorf(x), yf = floorf(y);
    const float dx = x - xf, dy = y - yf;
    const float wgt[4] = {(1.f - dx) * (1.f - dy), dx * (1.f - dy), (1.f - dx) * dy, dx * dy};
    const int x0 = window_origin(xf, R, p.W) - R, y0 = window_origin(yf, R, p.H) - R;
    int col[SIDE], row[SIDE];                      // element offsets of the window's columns and rows
#pragma unroll
    for (int i = 0; i < SIDE; ++i) {
        col[i] = min(max(x0 + i, 0), p.W - 1) * p.C;
        row[i] = min(max(y0 + i, 0), p.H - 1) * p.W * p.C;
    }

    const int64_t qoff = bq * p.C + head * p.hd;
    const T *qp = static_cast<const T *>(p.q) + qoff;
    const T *gop = static_cast<const T *>(p.dout) + qoff;
    const int64_t kv_base = static_cast<int64_t>(b) * p.N * p.C + head * p.hd;
    const T *kb = static_cast<const T *>(p.k) + kv_base;
    const T *vb = static_cast<const T *>(p.v) + kv_base;
    const int chunks = p.hd >> 3;

    float s[M], da[M];
#pragma unroll
    for (int m = 0; m < M; ++m) s[m] = da[m] = 0.f;
    for (int ch = 0; ch < chunks; ++ch) {
        float qv[8], gv[8];
        load8<T>(qp + 8 * ch, qv);
        load8<T>(gop + 8 * ch, gv);
#pragma unroll
        for (int j = 0; j < SIDE; ++j)
#pragma unroll
            for (int i = 0; i < SIDE; ++i) {
                float kv[8], vv[8];
                load8<T>(kb + row[j] + col[i] + 8 * ch, kv);
                load8<T>(vb + row[j] + col[i] + 8 * ch, vv);
                float l1 = 0.f, dot = 0.f;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    l1 += fabsf(qv[c] - kv[c]);
                    dot = fmaf(gv[c], vv[c], dot);
                }
                s[j * SIDE + i] += l1;
                da[j * SIDE + i] += dot;
            }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) s[m] = -s[m] * p.scale;
    if (p.dattn != nullptr) {
        const T *gap = static_cast<const T *>(p.dattn) + (bq * p.h + head) * M;
#pragma unroll
        for (int m = 0; m < M; ++m) da[m] += load_one<T>(gap + m);
    }
    float a[M], ds[M], dw[4];
#pragma unroll
    for (int m = 0; m < M; ++m) a[m] = ds[m] = 0.f;
#pragma unroll
    for (int tq = 0; tq < 4; ++tq) {
        const int oy = tq >> 1, ox = tq & 1;
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < SUB; ++j)
#pragma unroll
            for (int i = 0; i < SUB; ++i) mx = fmaxf(mx, s[(j + oy) * SIDE + i + ox]);
        float pr[SUB * SUB], den = 0.f;
#pragma unroll
        for (int j = 0; j < SUB; ++j)
#pragma unroll
            for (int i = 0; i < SUB; ++i) {
                pr[j * SUB + i] = expf(s[(j + oy) * SIDE + i + ox] - mx);
                den += pr[j * SUB + i];
            }
        const float inv = 1.f / den;
        float pda = 0.f;
#pragma unroll
        for (int j = 0; j < SUB; ++j)
#pragma unroll
            for (int i = 0; i < SUB; ++i) {
                pr[j * SUB + i] *= inv;
                pda = fmaf(pr[j * SUB + i], da[(j + oy) * SIDE + i + ox], pda);
            }
        dw[tq] = pda;
#pragma unroll
        for (int j = 0; j < SUB; ++j)
#pragma unroll
            for (int i = 0; i < SUB; ++i) {
                const int m = (j + oy) * SIDE + i + ox;
                const float wp = wgt[tq] * pr[j * SUB + i];
                a[m] += wp;
                ds[m] = fmaf(wp, da[m] - pda, ds[m]);
            }
    }
    if (p.dmo != nullptr) {
        T *gmo = static_cast<T *>(p.dmo) + (bq * p.h + head) * 2;
        store_one<T>(gmo, (1.f - dy) * (dw[1] - dw[0]) + dy * (dw[3] - dw[2]));
        store_one<T>(gmo + 1, (1.f - dx) * (dw[2] - dw[0]) + dx * (dw[3] - dw[1]));
    }
#pragma unroll
    for (int m = 0; m < M; ++m) ds[m] *= p.scale;

    T *gq = static_cast<T *>(p.dq) + qoff;
    float *dkb = p.dk + kv_base, *dvb = p.dv + kv_base;
    for (int ch = 0; ch < chunks; ++ch) {
        float qv[8], gv[8], acc[8];
        load8<T>(qp + 8 * ch, qv);
        load8<T>(gop + 8 * ch, gv);
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = 0.f;
#pragma unroll
        for (int j = 0; j < SIDE; ++j)
#pragma unroll
            for (int i = 0; i < SIDE; ++i) {
                const int m = j * SIDE + i;
                const int off = row[j] + col[i] + 8 * ch;
                float kv[8], gk[8];
                load8<T>(kb + off, kv);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    gk[c] = ds[m] * sign_of(qv[c], kv[c]);       // not finite where ds is not, as the product is in every other kernel
                    acc[c] -= gk[c];
                }
                if (ds[m] != 0.f) {
                    atomicAdd(reinterpret_cast<float4 *>(dkb + off), make_float4(gk[0], gk[1], gk[2], gk[3]));
                    atomicAdd(reinterpret_cast<float4 *>(dkb + off) + 1, make_float4(gk[4], gk[5], gk[6], gk[7]));
                }
                if (a[m] != 0.f) {
                    atomicAdd(reinterpret_cast<float4 *>(dvb + off),
                              make_float4(a[m] * gv[0], a[m] * gv[1], a[m] * gv[2], a[m] * gv[3]));
                    atomicAdd(reinterpret_cast<float4 *>(dvb + off) + 1,
                              make_float4(a[m] * gv[4], a[m] * gv[5], a[m] * gv[6], a[m] * gv[7]));
                }
            }
        store8<T>(gq + 8 * ch, acc);
    }
}

// ---- gathered ---------------------------------------------------------------------------------------------
//
// A window that sticks out of the map has its outer taps on the border tokens; the coefficients of such taps are
// added to those of the border token, which leaves a full window inside the map: origins (x0, y0) in
// [0, W-SIDE] x [0, H-SIDE], one bucket each and per head and batch item.  The four (six) buckets of one row that a
// token needs are consecutive, and so are their items: the rows of buckets get their place in the list from an atomic
// cursor, the buckets within a row in order.
//
// Where all heads of every query share one centre (the cross branch, whose field has no head axis) one list of queries
// serves all heads and a warp sums whole token rows; a first kernel finds out, the others read its verdict.

// Tile of a block of the staged sums and chunks of eight channels of a head: a thread per token and chunk.
constexpr int kStagedX = 16, kStagedY = 8, kStagedChunks = 2;

// Split of the direct sums: chunks per lane, lanes per token, tokens per warp, tile of a block.
struct SumTiles {
    int cpt, lanes, per_warp, x, y, tiles_x;
};

struct GatherParams {
    BwdParams b;                 // b.dk, b.dv unused
    void *dk, *dv;               // tensor type, written
    int cells_x, cells_y;        // W - SIDE + 1, H - SIDE + 1
    int lph, lph_shift;          // coefficient kernel: lanes per head
    int64_t items;               // B * Nq * h
    int *counts, *cursor, *differ;   // [B * h * cells_y][cells_x]; one word each: next free slot, heads differ
    int *starts;                 // [B * h * cells_y][cells_x + 1]: first slot of a bucket
    int *rank;                   // [items]: place of an item within its bucket
    int2 *meta;                  // [slot]: row of q in its batch item (elements), x0 -- shared centres: slot * taps - x0
    float2 *coef;                // (scale * ds, a) per slot, tap -- shared centres: slot, tap, head
    int batch;                                          // staged sums: items at a time
    SumTiles all_heads, one_head;                       // direct sums: shared centres, one head
};

template <typename T, int R>
__device__ __forceinline__ void gather_window(const BwdParams &p, int64_t item, float &dx, float &dy, int &x0, int &y0)
{
    const T *mo = static_cast<const T *>(p.mo) + item * 2;
    const float x = load_one<T>(mo), y = load_one<T>(mo + 1);
    const float xf = floorf(x), yf = floorf(y);
    dx = x - xf;
    dy = y - yf;
    x0 = window_origin(xf, R, p.W) - R;
    y0 = window_origin(yf, R, p.H) - R;
}

// An item's query (over all batch items), head and batch item.
struct ItemIndex {
    uint32_t bq, head, b;
    __device__ __forceinline__ ItemIndex(const BwdParams &p, uint32_t item)
        : bq(item / static_cast<uint32_t>(p.h)), head(item - bq * p.h), b(bq / static_cast<uint32_t>(p.Nq)) {}
    __device__ __forceinline__ int64_t bucket_row(const GatherParams &g, bool shared, int y0) const
    {
        return static_cast<int64_t>((shared ? b : b * g.b.h + head) * static_cast<uint32_t>(g.cells_y) + y0);
    }
};

// Sets *differ if some query's heads have different centres.
template <typename T>
__global__ void __launch_bounds__(256) gather_check_kernel(const GatherParams g, uint32_t queries)
{
    chain_begin();
    using Pair = typename std::conditional<sizeof(T) == 4, uint2, uint32_t>::type;       // one (x, y)
    const uint32_t bq = blockIdx.x * 256u + threadIdx.x;
    if (bq >= queries) return;
    const Pair *mo = static_cast<const Pair *>(g.b.mo) + static_cast<int64_t>(bq) * g.b.h;
    const Pair first = *mo;
    bool same = true;
#pragma unroll 4
    for (int i = 1; i < g.b.h; ++i) {
        const Pair v = mo[i];
        if constexpr (sizeof(T) == 4) same = same && v.x == first.x && v.y == first.y;
        else same = same && v == first;
    }
    if (!same) *g.differ = 1;
}

// Every item takes a place in its bucket.
template <typename T, int R>
__global__ void __launch_bounds__(256) gather_count_kernel(const GatherParams g)
{
    chain_begin();
    constexpr int SIDE = 2 * R + 2;
    const uint32_t item = blockIdx.x * 256u + threadIdx.x;
    if (item >= g.items) return;
    const bool shared = *g.differ == 0;
    const ItemIndex at(g.b, item);
    if (shared && at.head != 0) return;
    float dx, dy;
    int x0, y0;
    gather_window<T, R>(g.b, item, dx, dy, x0, y0);
    x0 = min(max(x0, 0), g.b.W - SIDE);
    y0 = min(max(y0, 0), g.b.H - SIDE);
    g.rank[item] = atomicAdd(g.counts + at.bucket_row(g, shared, y0) * g.cells_x + x0, 1);
}

// A warp per row of buckets: the buckets' first slots, the row's place from the cursor.
__global__ void __launch_bounds__(256) gather_starts_kernel(const GatherParams g, int64_t rows)
{
    chain_begin();
    const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= (*g.differ == 0 ? rows / g.b.h : rows)) return;
    const int *count = g.counts + row * g.cells_x;
    int total = 0;
    for (int c = lane; c < g.cells_x; c += 32) total += count[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    int at = lane == 0 ? atomicAdd(g.cursor, total) : 0;
    at = __shfl_sync(0xffffffffu, at, 0);
    int *start = g.starts + row * (g.cells_x + 1);
    for (int c0 = 0; c0 < g.cells_x; c0 += 32) {
        const int n = c0 + lane < g.cells_x ? count[c0 + lane] : 0;
        int sum = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int left = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += left;
        }
        if (c0 + lane < g.cells_x) start[c0 + lane] = at + sum - n;
        at += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) start[g.cells_x] = at;
}

// float32 accumulator += product of two 16-bit values, exact product (PTX ISA 8.6, sm_100+)
template <typename T>
__device__ __forceinline__ float fma_f32_16(unsigned short a, unsigned short b, float acc)
{
    if constexpr (std::is_same_v<T, __half>) asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc) : "h"(a), "h"(b));
    else asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(acc) : "h"(a), "h"(b));
    return acc;
}
template <typename T>
__device__ __forceinline__ float add_f32_16(float acc, unsigned short h)
{
    if constexpr (std::is_same_v<T, __half>) return add_f32_f16(acc, h);
    else return add_f32_bf16(acc, h);
}
__device__ __forceinline__ unsigned short half_of(uint32_t w, int hi) { return static_cast<unsigned short>(hi ? w >> 16 : w & 0xffffu); }

// sign(a - b) of the elements of a word, as floats.  16-bit types: (a > b) - (a < b), two elements per instruction.
template <typename T>
__device__ __forceinline__ float2 sign_pair(uint32_t a, uint32_t b)
{
    uint32_t w;
    if constexpr (std::is_same_v<T, __half>) {
        const __half2 x = *reinterpret_cast<const __half2 *>(&a), y = *reinterpret_cast<const __half2 *>(&b);
        const __half2 d = __hsub2(__hgt2(x, y), __hlt2(x, y));
        w = *reinterpret_cast<const uint32_t *>(&d);
    } else {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162 *>(&a), y = *reinterpret_cast<const __nv_bfloat162 *>(&b);
        const __nv_bfloat162 d = __hsub2(__hgt2(x, y), __hlt2(x, y));
        w = *reinterpret_cast<const uint32_t *>(&d);
    }
    return make_float2(DT<T>::unpack(w, 0), DT<T>::unpack(w, 1));
}

// A lane's slice (NW words) of q or dout against one tap's words of K or V.
template <typename T, int NW>
struct Distance {                // sum of |q - k|, exact differences
    float neg_q[NW * DT<T>::kElemsPerWord];
    __device__ __forceinline__ explicit Distance(const uint32_t (&q)[NW])
    {
#pragma unroll
        for (int c = 0; c < NW * DT<T>::kElemsPerWord; ++c) neg_q[c] = -DT<T>::unpack(q[c / DT<T>::kElemsPerWord], c % DT<T>::kElemsPerWord);
    }
    __device__ __forceinline__ float operator()(const uint32_t (&k)[NW]) const
    {
        float a = 0.f, b = 0.f;
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int w = 0; w < NW; w += 2) {
                a += fabsf(neg_q[w] + __uint_as_float(k[w]));
                b += fabsf(neg_q[w + 1] + __uint_as_float(k[w + 1]));
            }
        } else {
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                a += fabsf(add_f32_16<T>(neg_q[2 * w], half_of(k[w], 0)));
                b += fabsf(add_f32_16<T>(neg_q[2 * w + 1], half_of(k[w], 1)));
            }
        }
        return a + b;
    }
};

template <typename T, int NW>
__device__ __forceinline__ float dot_words(const uint32_t (&g)[NW], const uint32_t (&v)[NW])
{
    float a = 0.f, b = 0.f;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int w = 0; w < NW; w += 2) {
            a = fmaf(__uint_as_float(g[w]), __uint_as_float(v[w]), a);
            b = fmaf(__uint_as_float(g[w + 1]), __uint_as_float(v[w + 1]), b);
        }
    } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            a = fma_f32_16<T>(half_of(g[w], 0), half_of(v[w], 0), a);
            b = fma_f32_16<T>(half_of(g[w], 1), half_of(v[w], 1), b);
        }
    }
    return a + b;
}

template <typename T, int NW>
struct QueryGradient {           // dq -= ds * sign(q - k)
    static constexpr int EPW = DT<T>::kElemsPerWord;
    float dq[NW * EPW];
    __device__ __forceinline__ QueryGradient()
    {
#pragma unroll
        for (int c = 0; c < NW * EPW; ++c) dq[c] = 0.f;
    }
    __device__ __forceinline__ void step(const uint32_t (&q)[NW], const uint32_t (&k)[NW], float ds)
    {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if constexpr (EPW == 1) {
                dq[w] = fmaf(ds, sign_of(__uint_as_float(k[w]), __uint_as_float(q[w])), dq[w]);
            } else {
                const float2 s = sign_pair<T>(k[w], q[w]);
                dq[2 * w] = fmaf(ds, s.x, dq[2 * w]);
                dq[2 * w + 1] = fmaf(ds, s.y, dq[2 * w + 1]);
            }
        }
    }
    __device__ __forceinline__ void result(uint32_t (&o)[NW]) const
    {
#pragma unroll
        for (int w = 0; w < NW; ++w) o[w] = DT<T>::aw_from(dq[w * EPW], dq[w * EPW + EPW - 1]);
    }
};

// dq, d(max_offset) and the coefficients of one item, by one lane or (wide heads) a few that share its channels.
// With e_m the exponentials around the largest score, den_t and v_t the sums of e_m and e_m da_m over sub-window t and
// c_t = w_t / den_t:   a_m = e_m C_m,  ds_m = e_m (da_m C_m - U_m),  C_m = sum of c_t, U_m = sum of c_t v_t / den_t
// over the sub-windows t that hold m, so one exponential per tap serves all four.
// Bound by the latency of the taps at four blocks of 128 threads per SM (issue 59 %, L1 49 %; with a centre per head the
// slots' stores bring L1 to 79 %): the window of V once, of K twice, 128 bytes of coefficients out.
// Measured, float16, 384x384 tokens, 8 heads x 16, r = 1: 163 us (207 us with per-head slots, whose stores touch a line
// per lane), at 128 registers; the rows of the second walk over K as a loop, or the compiler moves all its loads up and
// spills (266 us).
template <typename T, int R, int CPL>
__global__ void __launch_bounds__(128, R == 1 && CPL <= 2 ? 4 : 3) gather_coef_kernel(const GatherParams g)
{
    chain_begin();
    constexpr int SIDE = 2 * R + 2, SUB = 2 * R + 1, M = SIDE * SIDE;
    constexpr int NW = CPL * DT<T>::kWordsPerChunk;
    const BwdParams &p = g.b;
    const int64_t t = static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x;
    const bool valid = (t >> g.lph_shift) < g.items;
    const uint32_t item = static_cast<uint32_t>(valid ? t >> g.lph_shift : g.items - 1);   // idle lanes redo the last item for the shuffles
    const int sl = static_cast<int>(t) & (g.lph - 1);
    const ItemIndex at(p, item);
    const int64_t bq = at.bq, b = at.b;
    const int head = static_cast<int>(at.head);

    float dx, dy;
    int x0, y0;
    gather_window<T, R>(p, item, dx, dy, x0, y0);
    // a tap's address is its row's pointer plus an unsigned 32-bit byte offset of its column
    uint32_t col[SIDE];
    int row[SIDE];
#pragma unroll
    for (int i = 0; i < SIDE; ++i) {
        col[i] = static_cast<uint32_t>(min(max(x0 + i, 0), p.W - 1) * p.C) * static_cast<uint32_t>(sizeof(T));
        row[i] = min(max(y0 + i, 0), p.H - 1) * p.W * p.C;
    }
    const int lane_off = head * p.hd + sl * CPL * 8;
    const int64_t q_off = bq * p.C + lane_off, kv_base = b * p.N * p.C + lane_off;
    const T *kb = static_cast<const T *>(p.k) + kv_base;
    const T *vb = static_cast<const T *>(p.v) + kv_base;
    // V first, then K, so that the second walk over K comes soon after the first
    float s[M], da[M];
    uint32_t qw[NW];
    load_words<NW>(qw, static_cast<const T *>(p.dout) + q_off);
#pragma unroll
    for (int j = 0; j < SIDE; ++j)
#pragma unroll
        for (int i = 0; i < SIDE; ++i) {
            uint32_t vw[NW];
            load_words<NW>(vw, tap_ptr(vb + row[j], col[i]));
            da[j * SIDE + i] = dot_words<T, NW>(qw, vw);
        }
    load_words<NW>(qw, static_cast<const T *>(p.q) + q_off);
    {
        const Distance<T, NW> distance(qw);
#pragma unroll
        for (int j = 0; j < SIDE; ++j)
#pragma unroll
            for (int i = 0; i < SIDE; ++i) {
                uint32_t kw[NW];
                load_words<NW>(kw, tap_ptr(kb + row[j], col[i]));
                s[j * SIDE + i] = distance(kw);
            }
    }
    for (int o = g.lph >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            s[m] += __shfl_xor_sync(0xffffffffu, s[m], o);
            da[m] += __shfl_xor_sync(0xffffffffu, da[m], o);
        }
    }
    if (p.dattn != nullptr) {
        constexpr int EPW = DT<T>::kElemsPerWord;
        const uint2 *gap = reinterpret_cast<const uint2 *>(static_cast<const T *>(p.dattn) + static_cast<int64_t>(item) * M);
#pragma unroll
        for (int w = 0; w < M / EPW / 2; ++w) {
            const uint2 u = gap[w];
#pragma unroll
            for (int e = 0; e < 2 * EPW; ++e) da[2 * EPW * w + e] += DT<T>::unpack(e < EPW ? u.x : u.y, e % EPW);
        }
    }
    float top = -INFINITY;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        s[m] = -s[m] * p.scale;
        top = fmaxf(top, s[m]);
    }
    float low = top;                               // the lowest of the sub-windows' maxima
#pragma unroll
    for (int tq = 0; tq < 4; ++tq) {
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < SUB; ++j)
#pragma unroll
            for (int i = 0; i < SUB; ++i) mx = fmaxf(mx, s[(j + (tq >> 1)) * SIDE + i + (tq & 1)]);
        low = fminf(low, mx);
    }
    const float wgt[4] = {(1.f - dx) * (1.f - dy), dx * (1.f - dy), (1.f - dx) * dy, dx * dy};
    float dw[4];
    if (top - low < 60.f) {
#pragma unroll
        for (int m = 0; m < M; ++m) s[m] = expf(s[m] - top);
        float den[4], num[4];
#pragma unroll
        for (int tq = 0; tq < 4; ++tq) {
            den[tq] = num[tq] = 0.f;
#pragma unroll
            for (int j = 0; j < SUB; ++j)
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    const int m = (j + (tq >> 1)) * SIDE + i + (tq & 1);
                    den[tq] += s[m];
                    num[tq] = fmaf(s[m], da[m], num[tq]);
                }
        }
        float c[4], u[4];
#pragma unroll
        for (int tq = 0; tq < 4; ++tq) {
            const float inv = 1.f / den[tq];
            dw[tq] = num[tq] * inv;
            c[tq] = wgt[tq] * inv;
            u[tq] = c[tq] * dw[tq];
        }
#pragma unroll
        for (int j = 0; j < SIDE; ++j)
#pragma unroll
            for (int i = 0; i < SIDE; ++i) {
                const int m = j * SIDE + i;
                float cm = 0.f, um = 0.f;
#pragma unroll
                for (int tq = 0; tq < 4; ++tq) {
                    const int oy = tq >> 1, ox = tq & 1;
                    if (j >= oy && j < oy + SUB && i >= ox && i < ox + SUB) {
                        cm += c[tq];
                        um += u[tq];
                    }
                }
                const float e = s[m];
                s[m] = e * fmaf(da[m], cm, -um) * p.scale;       // scale * ds
                da[m] = e * cm;                                  // a
            }
    } else {     // widely spread scores: every sub-window around its own maximum
        float a[M], ds[M];
#pragma unroll
        for (int m = 0; m < M; ++m) a[m] = ds[m] = 0.f;
#pragma unroll
        for (int tq = 0; tq < 4; ++tq) {
            const int oy = tq >> 1, ox = tq & 1;
            float mx = -INFINITY, den = 0.f, num = 0.f;
#pragma unroll
            for (int j = 0; j < SUB; ++j)
#pragma unroll
                for (int i = 0; i < SUB; ++i) mx = fmaxf(mx, s[(j + oy) * SIDE + i + ox]);
#pragma unroll
            for (int j = 0; j < SUB; ++j)
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    const int m = (j + oy) * SIDE + i + ox;
                    const float e = expf(s[m] - mx);
                    den += e;
                    num = fmaf(e, da[m], num);
                }
            const float inv = 1.f / den;
            dw[tq] = num * inv;
#pragma unroll
            for (int j = 0; j < SUB; ++j)
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    const int m = (j + oy) * SIDE + i + ox;
                    const float wp = wgt[tq] * (expf(s[m] - mx) * inv);
                    a[m] += wp;
                    ds[m] = fmaf(wp, da[m] - dw[tq], ds[m]);
                }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            s[m] = ds[m] * p.scale;
            da[m] = a[m];
        }
    }
    if (p.dmo != nullptr && sl == 0 && valid) {
        T *gmo = static_cast<T *>(p.dmo) + static_cast<int64_t>(item) * 2;
        store_one<T>(gmo, (1.f - dy) * (dw[1] - dw[0]) + dy * (dw[3] - dw[2]));
        store_one<T>(gmo + 1, (1.f - dx) * (dw[2] - dw[0]) + dx * (dw[3] - dw[1]));
    }

    const int x_in = min(max(x0, 0), p.W - SIDE), y_in = min(max(y0, 0), p.H - SIDE);
    const bool shared = *g.differ == 0;
    const int64_t slot = g.starts[at.bucket_row(g, shared, y_in) * (g.cells_x + 1) + x_in] + g.rank[shared ? item - head : item];
    float2 *coef = g.coef + (shared ? slot * M * p.h + head : slot * M);     // tap m at coef[m * coef_step]
    const int coef_step = shared ? p.h : 1;
    if (valid) {
        if (sl == 0 && (!shared || head == 0)) g.meta[slot] = make_int2(static_cast<int>((bq - b * p.Nq) * p.C), shared ? static_cast<int>(slot * M) - x_in : x_in);
        if (shared) {
#pragma unroll
            for (int m = 0; m < M; ++m)
                if ((m & (g.lph - 1)) == sl) coef[m * coef_step] = make_float2(s[m], da[m]);
        } else {
            float4 *out = reinterpret_cast<float4 *>(coef);
#pragma unroll
            for (int k = 0; k < M / 2; ++k)
                if ((k & (g.lph - 1)) == sl) out[k] = make_float4(s[2 * k], da[2 * k], s[2 * k + 1], da[2 * k + 1]);
        }
    }
    // dq: a row of the window per step (a loop, or the loads of all rows would be moved up and take the registers)
    {
        QueryGradient<T, NW> grad;
#pragma unroll 1
        for (int j = 0; j < SIDE; ++j) {
#pragma unroll
            for (int i = 0; i < SIDE; ++i) {
                uint32_t kw[NW];
                load_words<NW>(kw, tap_ptr(kb + row[0], col[i]));
                grad.step(qw, kw, s[i]);
            }
#pragma unroll
            for (int m = 0; m + SIDE < M; ++m) s[m] = s[m + SIDE];
#pragma unroll
            for (int i = 0; i + 1 < SIDE; ++i) row[i] = row[i + 1];
        }
        uint32_t ow[NW];
        grad.result(ow);
        if (valid) store_words<NW>(static_cast<T *>(p.dq) + q_off, ow);
    }
    const bool sticks_out = x_in != x0 || y_in != y0;
    if (!__any_sync(0xffffffffu, sticks_out)) return;
    __syncwarp();
    if (!valid || !sticks_out || sl != 0) return;
    // taps outside the map onto the border token: row by row, then column by column, in the slot just written
    const auto fold = [](float2 *at0, int step, int shift) {       // element i goes to min(max(i + shift, 0), SIDE - 1)
        float2 in[SIDE];
#pragma unroll
        for (int i = 0; i < SIDE; ++i) in[i] = at0[i * step];
#pragma unroll
        for (int o = 0; o < SIDE; ++o) {
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < SIDE; ++i)
                if (min(max(i + shift, 0), SIDE - 1) == o) {
                    sum.x += in[i].x;
                    sum.y += in[i].y;
                }
            at0[o * step] = sum;
        }
    };
    if (x_in != x0)
        for (int j = 0; j < SIDE; ++j) fold(coef + j * SIDE * coef_step, coef_step, x0 - x_in);
    if (y_in != y0)
        for (int i = 0; i < SIDE; ++i) fold(coef + i * coef_step, SIDE * coef_step, y0 - y_in);
}

// Eight channels of q and dout as loaded: 16 bytes, or 32 in one piece (float32, 192x192 tokens, 4 heads x 16: 77 -> 71 us).
template <typename T>
struct Piece {
    static constexpr int NW = DT<T>::kWordsPerChunk;
    uint32_t q[NW], go[NW];
    static __device__ __forceinline__ void load(uint32_t (&w)[NW], const T *at)      // (the 32-byte form takes global addresses only)
    {
        if constexpr (NW == 8) {
            ld_256(w, at);
        } else {
            const uint4 u = *reinterpret_cast<const uint4 *>(at);
            w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
        }
    }
    __device__ __forceinline__ void load(const T *qp, const T *gp)         // from global memory
    {
        load(q, qp);
        load(go, gp);
    }
    __device__ __forceinline__ void load_staged(const char *qp, const char *gp)      // from shared memory
    {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            const uint4 u = reinterpret_cast<const uint4 *>(qp)[i], v = reinterpret_cast<const uint4 *>(gp)[i];
            q[4 * i] = u.x; q[4 * i + 1] = u.y; q[4 * i + 2] = u.z; q[4 * i + 3] = u.w;
            go[4 * i] = v.x; go[4 * i + 1] = v.y; go[4 * i + 2] = v.z; go[4 * i + 3] = v.w;
        }
    }
};

// sign(q - k) * ds and a * dout added to the sums of eight channels of a token
template <typename T>
struct Accumulate {
    uint32_t k[4 * sizeof(T) / 2];
    float dk[8], dv[8];
    __device__ __forceinline__ void start(const T *kp)
    {
#pragma unroll
        for (int i = 0; i < static_cast<int>(sizeof(T)) / 2; ++i) {
            const uint4 u = reinterpret_cast<const uint4 *>(kp)[i];
            k[4 * i] = u.x; k[4 * i + 1] = u.y; k[4 * i + 2] = u.z; k[4 * i + 3] = u.w;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) dk[c] = dv[c] = 0.f;
    }
    __device__ __forceinline__ void add(const Piece<T> &pc, float ds, float a)
    {
#pragma unroll
        for (int w = 0; w < Piece<T>::NW; ++w) {
            if constexpr (sizeof(T) == 4) {
                dk[w] = fmaf(ds, sign_of(__uint_as_float(pc.q[w]), __uint_as_float(k[w])), dk[w]);
                dv[w] = fmaf(a, __uint_as_float(pc.go[w]), dv[w]);
            } else {
                const float2 s = sign_pair<T>(pc.q[w], k[w]);
                dk[2 * w] = fmaf(ds, s.x, dk[2 * w]);
                dk[2 * w + 1] = fmaf(ds, s.y, dk[2 * w + 1]);
                dv[2 * w] = fmaf(a, DT<T>::unpack(pc.go[w], 0), dv[2 * w]);
                dv[2 * w + 1] = fmaf(a, DT<T>::unpack(pc.go[w], 1), dv[2 * w + 1]);
            }
        }
    }
};

// Rows of tiles in the order last, first, second, ...: centres that the caller clamps to the map pile up at its borders,
// and the long lists of the last row must not start last.
__device__ __forceinline__ int tile_row(int i, int rows) { return i == 0 ? rows - 1 : i - 1; }

__device__ __forceinline__ void copy16_async(void *smem, const void *global)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))), "l"(global)
                 : "memory");
}

// Has L2 fetch `count` pieces of `bytes` (a multiple of 16, from an address aligned to 16) that lie one after another.
__device__ __forceinline__ void prefetch_l2(const void *global, int count, uint32_t bytes)
{
    // (one request holds a 32-bit size: what does not fit in is left to the loads)
    const uint32_t most = 0x7ffffff0u / bytes, n = min(static_cast<uint32_t>(count), most);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(global), "r"(n * bytes) : "memory");
}

// dk and dv of a tile of tokens, one head of two chunks of channels: a thread per (token, eight channels).  The items
// of all buckets that the tile needs are staged in shared memory, `batch` at a time: coefficients, q and dout.
// A slot of coefficients is padded by 16 bytes: neighbouring tokens read the same tap of neighbouring slots.
// Such narrow heads alone: read straight from global memory, every item of a list is a line of its own for as few bytes
// (float16, 384x384 tokens, 8 heads x 16, a centre per head: 207 to 219 us on several boards, the kernel below 260 where it
// took 219; float32, 2 x 192x192, 4 x 16: 79 and 105; 4 x 8 channels: 54 and 50, 4 x 64: 190 and 160).
// Bound by instruction issue (73 % of the slots; about 57 per token, item and eight channels; two thirds of the lanes busy,
// lists differ in length); walking a token's four ranges as one list costs as much as it saves.
template <typename T, int R>
__global__ void __launch_bounds__(kStagedX * kStagedY * kStagedChunks) gather_sum_staged_kernel(const GatherParams g)
{
    chain_begin();
    constexpr int SIDE = 2 * R + 2, M = SIDE * SIDE, kCoefPitch = M * 8 + 16;
    extern __shared__ __align__(16) char smem[];
    if (*g.differ == 0) return;
    const BwdParams &p = g.b;
    constexpr int threads = kStagedX * kStagedY * kStagedChunks, row_bytes = kStagedChunks * 8 * static_cast<int>(sizeof(T));
    constexpr int rows = kStagedY + SIDE - 1, cols = kStagedX + SIDE;         // bucket rows, bucket starts per row
    const int tid = threadIdx.x, tiles_x = (p.W + kStagedX - 1) / kStagedX;
    const int order = blockIdx.x / tiles_x, tile_x = blockIdx.x - order * tiles_x;
    const int tx0 = tile_x * kStagedX, ty0 = tile_row(order, gridDim.x / tiles_x) * kStagedY;
    const int bh = blockIdx.y, b = bh / p.h, head = bh - b * p.h;
    const int head_off = head * p.hd;

    char *coef_s = smem;
    char *q_s = coef_s + g.batch * kCoefPitch, *go_s = q_s + g.batch * row_bytes;
    int2 *meta_s = reinterpret_cast<int2 *>(go_s + g.batch * row_bytes);      // (row of q, x0) of a staged item
    int *slot_s = reinterpret_cast<int *>(meta_s + g.batch);
    int *start_s = slot_s + g.batch, *base_s = start_s + rows * cols;         // base_s[r]: items of the tile before row r

    for (int e = tid; e < rows * cols; e += threads) {
        const int r = e / cols, c = e - r * cols;
        const int cy = ty0 - (SIDE - 1) + r, cx = min(max(tx0 - (SIDE - 1) + c, 0), g.cells_x);
        start_s[e] = cy >= 0 && cy < g.cells_y ? g.starts[(static_cast<int64_t>(bh) * g.cells_y + cy) * (g.cells_x + 1) + cx] : 0;
    }
    __syncthreads();
    if (tid < 32) {
        int n = tid < rows ? start_s[tid * cols + cols - 1] - start_s[tid * cols] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int left = __shfl_up_sync(0xffffffffu, n, o);
            if (tid >= o) n += left;
        }
        if (tid < rows) base_s[tid + 1] = n;
        if (tid == 0) base_s[0] = 0;
    }
    __syncthreads();
    const int total = base_s[rows];

    const int chunk = tid % kStagedChunks, token = tid / kStagedChunks;
    const int txl = token % kStagedX, tyl = token / kStagedX;
    const int tx = tx0 + txl, ty = ty0 + tyl;
    const bool mine = tx < p.W && ty < p.H;
    const int64_t token_off = (static_cast<int64_t>(b) * p.N + static_cast<int64_t>(ty) * p.W + tx) * p.C + head_off + chunk * 8;
    Accumulate<T> acc;
    acc.start(static_cast<const T *>(p.k) + (mine ? token_off : 0));

    for (int f0 = 0; f0 < total; f0 += g.batch) {
        const int n = min(g.batch, total - f0);
        for (int e = tid; e < n; e += threads) {
            int r = 0;
            while (f0 + e >= base_s[r + 1]) ++r;
            const int slot = start_s[r * cols] + f0 + e - base_s[r];
            slot_s[e] = slot;
            meta_s[e] = g.meta[slot];
        }
        __syncthreads();
        for (int e = tid; e < n * (M / 2); e += threads) {
            const int i = e / (M / 2), k = e - i * (M / 2);
            copy16_async(coef_s + i * kCoefPitch + k * 16, reinterpret_cast<const char *>(g.coef + static_cast<int64_t>(slot_s[i]) * M) + k * 16);
        }
        constexpr int pieces = row_bytes / 16;
        for (int e = tid; e < n * pieces; e += threads) {
            const int i = e / pieces, k = e - i * pieces;
            const int64_t off = static_cast<int64_t>(b) * p.Nq * p.C + meta_s[i].x + head_off;
            copy16_async(q_s + i * row_bytes + k * 16, reinterpret_cast<const char *>(static_cast<const T *>(p.q) + off) + k * 16);
            copy16_async(go_s + i * row_bytes + k * 16, reinterpret_cast<const char *>(static_cast<const T *>(p.dout) + off) + k * 16);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (mine) {
            for (int j = 0; j < SIDE; ++j) {
                const int r = tyl + SIDE - 1 - j;
                const int *st = start_s + r * cols;
                const int lo = max(base_s[r] + st[txl] - st[0] - f0, 0), hi = min(base_s[r] + st[txl + SIDE] - st[0] - f0, n);
                for (int i = lo; i < hi; ++i) {
                    const float2 co = *reinterpret_cast<const float2 *>(coef_s + i * kCoefPitch + (j * SIDE + tx - meta_s[i].y) * 8);
                    Piece<T> piece;
                    piece.load_staged(q_s + i * row_bytes + chunk * 8 * sizeof(T), go_s + i * row_bytes + chunk * 8 * sizeof(T));
                    acc.add(piece, co.x, co.y);
                }
            }
        }
        __syncthreads();
    }
    if (mine) {
        store8<T>(static_cast<T *>(g.dk) + token_off, acc.dk);
        store8<T>(static_cast<T *>(g.dv) + token_off, acc.dv);
    }
}

// resident blocks of the kernel below per SM: as many as the registers of its chunks allow (0: no limit asked for)
// (float16, 384x384 tokens, 8 heads x 16: 183 us with three, 173 with four; float32, r = 1: 126 with four, 79 with three;
// float32, 2 x 45x79, 4 x 32, r = 2: 41 to 48 with three, 34 with two)
template <typename T, int R, int CPT>
constexpr int sum_min_blocks() { return CPT == 4 ? 0 : CPT == 2 ? 2 : sizeof(T) == 2 && R == 1 ? 4 : sizeof(T) == 4 && R == 2 ? 2 : 3; }
// blocks ahead, in the same list, whose coefficients a block asks L2 for (float16, 384x384 tokens, 8 heads x 16: 600 173 us, 300
// 171, 1000 176); the first so many blocks of every list, all those of a small map, go without
constexpr unsigned kPrefetchAhead = 300;

// The same without staging: `lanes` lanes per token, each with CPT chunks of eight channels (chunk = lane + s * lanes),
// `per_warp` tokens per warp; the lanes of a token walk the same list.  SHARED: one list for all heads, a query's row of
// q and dout is read as a whole, a tap's coefficients of all heads lie side by side; otherwise one head.  The rows are
// shared by the tokens of a block through L1.
// The coefficients are read once and come from memory: every block has L2 fetch those of the buckets that a block some
// way ahead starts with, whole runs of slots in one request each.
// Bound by instruction issue with shared centres (73 %; 59 % and the latency of the loads at three blocks per SM without the
// prefetch; more lanes or items side by side add their own start: 230 to 265 us), by the longest lists in small calls.
// Measured, float16, 384x384 tokens, 8 heads x 16, r = 1, shared: 171 us (209 without the prefetch at three blocks).  One
// head: float16, 2 x 192x192, 4 x 64: 160 us (staged 190); float32, 2 x 45x79, 4 x 32, r = 2: 34 us (staged 38).
template <typename T, int R, int CPT, bool SHARED>
__global__ void __launch_bounds__(256, sum_min_blocks<T, R, CPT>()) gather_sum_direct_kernel(const GatherParams g)
{
    chain_begin();
    constexpr int SIDE = 2 * R + 2, M = SIDE * SIDE;
    if ((*g.differ == 0) != SHARED) return;
    const BwdParams &p = g.b;
    const SumTiles &tl = SHARED ? g.all_heads : g.one_head;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane / tl.lanes, own = lane - sub * tl.lanes;
    const int list = blockIdx.y, b = SHARED ? list : list / p.h, tile_rows = gridDim.x / tl.tiles_x;
    const uint32_t coef_step = SHARED ? p.h : 1;         // heads whose coefficients of a tap lie side by side
    const int order = blockIdx.x / tl.tiles_x, tile_x = blockIdx.x - order * tl.tiles_x;
    if (blockIdx.x + kPrefetchAhead < gridDim.x && threadIdx.x < tl.y) {
        const int then = blockIdx.x + kPrefetchAhead, then_row = then / tl.tiles_x;
        const int cy = tile_row(then_row, tile_rows) * tl.y + threadIdx.x, cx = (then - then_row * tl.tiles_x) * tl.x;
        if (cy < g.cells_y && cx < g.cells_x) {
            const int *start = g.starts + (static_cast<int64_t>(list) * g.cells_y + cy) * (g.cells_x + 1);
            const int from = start[cx], slots = start[min(cx + tl.x, g.cells_x)] - from;
            if (slots > 0) prefetch_l2(g.coef + static_cast<int64_t>(from) * M * coef_step, slots, M * coef_step * static_cast<uint32_t>(sizeof(float2)));
        }
    }
    const int t = warp * tl.per_warp + sub, ty_in = t / tl.x;
    const int tx = tile_x * tl.x + t - ty_in * tl.x, ty = tile_row(order, tile_rows) * tl.y + ty_in;
    if (sub >= tl.per_warp || tx >= p.W || ty >= p.H) return;
    const int hd8 = p.hd >> 3;
    const int64_t token_off = (static_cast<int64_t>(b) * p.N + static_cast<int64_t>(ty) * p.W + tx) * p.C + (SHARED ? 0 : (list - b * p.h) * p.hd);

    const int64_t query_off = static_cast<int64_t>(b) * p.Nq * p.C + (SHARED ? 0 : (list - b * p.h) * p.hd) + own * 8;
    const T *q = static_cast<const T *>(p.q) + query_off, *go = static_cast<const T *>(p.dout) + query_off;
    const int step = tl.lanes * 8;                       // channels between the chunks of a lane
    Accumulate<T> acc[CPT];
#pragma unroll
    for (int s = 0; s < CPT; ++s) acc[s].start(static_cast<const T *>(p.k) + token_off + own * 8 + s * step);
    int head[CPT];
#pragma unroll
    for (int s = 0; s < CPT; ++s) head[s] = SHARED ? (own + s * tl.lanes) / hd8 : 0;

    // the token's items, one range of slots per row of buckets, numbered through: item f of row j lies in slot
    // base[j] + f
    int until[SIDE], base[SIDE], total = 0;
    {
        const int c_lo = max(tx - (SIDE - 1), 0), c_hi = min(tx + 1, g.cells_x);
        int lo[SIDE], hi[SIDE];
#pragma unroll
        for (int j = 0; j < SIDE; ++j) {
            const int cy = ty - j;
            const int *start = g.starts + (static_cast<int64_t>(list) * g.cells_y + cy) * (g.cells_x + 1);
            const bool ok = cy >= 0 && cy < g.cells_y;
            lo[j] = ok ? start[c_lo] : 0;
            hi[j] = ok ? start[c_hi] : 0;
        }
#pragma unroll
        for (int j = 0; j < SIDE; ++j) {
            base[j] = lo[j] - total;
            total += hi[j] - lo[j];
            until[j] = total;
        }
    }
    const auto locate = [&](int f, int &slot, int &tap) {
        slot = base[0];
        tap = tx;
#pragma unroll
        for (int j = 1; j < SIDE; ++j)
            if (f >= until[j - 1]) {
                slot = base[j];
                tap = tx + j * SIDE;
            }
        slot += f;
    };
    // two items at a time, so that their loads are under way together; their places are read one step ahead
    using Tap = std::conditional_t<SHARED, uint32_t, uint64_t>;       // fewer than 2^31 (query, tap), or not
    uint32_t row[2] = {0u, 0u};
    Tap tap[2] = {0u, 0u};
    const auto fetch = [&](int f) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            int slot, at;
            locate(min(f + n, total - 1), slot, at);
            const int2 m = g.meta[slot];
            row[n] = static_cast<uint32_t>(m.x);
            tap[n] = SHARED ? static_cast<Tap>(at + m.y) : static_cast<Tap>(slot) * M + static_cast<Tap>(at - m.y);
        }
    };
    if (total > 0) fetch(0);
    for (int f = 0; f < total; f += 2) {
        const bool second = f + 1 < total;
        const uint32_t r0 = row[0], r1 = row[1];
        const float2 *c0 = g.coef + static_cast<uint64_t>(tap[0]) * coef_step, *c1 = g.coef + static_cast<uint64_t>(tap[1]) * coef_step;
#pragma unroll
        for (int s = 0; s < CPT; ++s) {
            Piece<T> first, other;
            first.load(q + r0 + s * step, go + r0 + s * step);
            other.load(q + r1 + s * step, go + r1 + s * step);
            const float2 ca = c0[head[s]], cb = c1[head[s]];
            if (s == CPT - 1 && f + 2 < total) fetch(f + 2);
            acc[s].add(first, ca.x, ca.y);
            if (second) acc[s].add(other, cb.x, cb.y);
        }
    }
#pragma unroll
    for (int s = 0; s < CPT; ++s) {
        store8<T>(static_cast<T *>(g.dk) + token_off + own * 8 + s * step, acc[s].dk);
        store8<T>(static_cast<T *>(g.dv) + token_off + own * 8 + s * step, acc[s].dv);
    }
}

// Sizes of the gathered path; bytes == 0 where it does not apply.
struct GatherPlan {
    size_t off_cursor, off_starts, off_rank, off_meta, off_coef, bytes;
    int64_t bucket_rows;
    int cells_x, cells_y, lph, cpl;
    bool staged;
    int batch, smem;
    SumTiles all_heads, one_head;
};

GatherPlan gather_plan(int B, int H, int W, int h, int hd, int r, int dtype, int64_t Nq)
{
    GatherPlan pl{};
    const int side = 2 * r + 2, M = side * side, esize = dtype == MATCHATTN_F32 ? 4 : 2;
    if (hd % 8 != 0 || (r != 1 && r != 2) || W < side || H < side) return pl;
    const int chunks = hd / 8;
    const int64_t items = static_cast<int64_t>(B) * Nq * h;
    pl.cells_x = W - side + 1;
    pl.cells_y = H - side + 1;
    pl.bucket_rows = static_cast<int64_t>(B) * h * pl.cells_y;
    if (items >= (1LL << 31) || static_cast<int64_t>(B) * Nq * M >= (1LL << 31) || pl.bucket_rows * (pl.cells_x + 1) >= (1LL << 31) || static_cast<int64_t>(B) * h > 65535) return pl;
    // coefficient kernel: 32 bytes per lane and tap where the width allows (three or five chunks where it does not), up to
    // eight lanes per head; float32, r = 2, 2 x 45x79 tokens, 4 heads x 32: 48 us with 64-byte slices, 38 with these
    pl.lph = 1;
    pl.cpl = chunks;
    while (pl.cpl % 2 == 0 && (pl.cpl > 2 || (esize == 4 && pl.lph < 8))) {
        pl.cpl /= 2;
        pl.lph *= 2;
    }
    if (pl.lph > 32) return pl;
    if (pl.cpl > 3 && pl.cpl != 5) return pl;
    // staged sums: room for one and a half items per bucket of the tile (one is the mean), at most four blocks per SM
    // (float16, 384x384 tokens, 8 heads x 16: 219 us, three 238), or the three that float32 has registers for
    pl.staged = chunks == kStagedChunks;
    const int per_item = M * 8 + 16 + 2 * kStagedChunks * 8 * esize + 12;
    const int cells = (kStagedX + side - 1) * (kStagedY + side - 1), room = (esize == 2 ? 54 : 72) * 1024;
    pl.batch = cells * 3 / 2;
    if (pl.batch * per_item > room) pl.batch = room / per_item;
    pl.batch &= ~3;
    pl.smem = pl.batch * per_item + ((kStagedY + side - 1) * (kStagedX + side + 1) + 1) * 4;
    const auto split = [&](int row_chunks, SumTiles &tl) {     // one, two or four chunks per lane, whichever leaves the fewest lanes idle
        int best = 0;
        for (int cpt = 1; cpt <= 4; cpt *= 2) {
            if (row_chunks % cpt != 0 || row_chunks / cpt > 32) continue;
            const int lanes = row_chunks / cpt, used = 32 / lanes * lanes;
            if (used > best) {
                best = used;
                tl.cpt = cpt;
                tl.lanes = lanes;
                tl.per_warp = 32 / lanes;
            }
        }
        const int tokens = 8 * tl.per_warp;
        tl.x = tokens >= 32 ? 8 : 4;
        tl.y = tokens / tl.x;
        tl.tiles_x = (W + tl.x - 1) / tl.x;
        return best != 0;
    };
    if (!split(chunks * h, pl.all_heads) || !split(chunks, pl.one_head)) return pl;
    const auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
    size_t off = static_cast<size_t>(pl.bucket_rows) * pl.cells_x * sizeof(int);    // counts and the two words are cleared together
    pl.off_cursor = off; off = up(off + 2 * sizeof(int));
    pl.off_starts = off; off = up(off + static_cast<size_t>(pl.bucket_rows) * (pl.cells_x + 1) * sizeof(int));
    pl.off_rank = off;   off = up(off + static_cast<size_t>(items) * sizeof(int));
    pl.off_meta = off;   off = up(off + static_cast<size_t>(items) * sizeof(int2));
    pl.off_coef = off;   off = up(off + static_cast<size_t>(items) * M * sizeof(float2));
    pl.bytes = off;
    return pl;
}

template <typename T, int R>
cudaError_t launch_gather(const GatherParams &g, const GatherPlan &pl, cudaStream_t stream)
{
    cudaError_t e = cudaMemsetAsync(g.counts, 0, pl.off_cursor + 2 * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    const uint32_t queries = static_cast<uint32_t>(g.items / g.b.h);
    launch_chained(gather_check_kernel<T>, (queries + 255) / 256, 256, 0, stream, g, queries);
    launch_chained(gather_count_kernel<T, R>, static_cast<unsigned>((g.items + 255) / 256), 256, 0, stream, g);
    launch_chained(gather_starts_kernel, static_cast<unsigned>((pl.bucket_rows + 7) / 8), 256, 0, stream, g, pl.bucket_rows);
    const unsigned coef_blocks = static_cast<unsigned>((g.items * pl.lph + 127) / 128);
    switch (pl.cpl) {
    case 1: launch_chained(gather_coef_kernel<T, R, 1>, coef_blocks, 128, 0, stream, g); break;
    case 2: launch_chained(gather_coef_kernel<T, R, 2>, coef_blocks, 128, 0, stream, g); break;
    case 3: launch_chained(gather_coef_kernel<T, R, 3>, coef_blocks, 128, 0, stream, g); break;
    default: launch_chained(gather_coef_kernel<T, R, 5>, coef_blocks, 128, 0, stream, g); break;
    }
    const auto sums = [&](auto shared, const SumTiles &tl, int lists) {
        constexpr bool SHARED = decltype(shared)::value;
        const dim3 grid(static_cast<unsigned>(tl.tiles_x) * ((g.b.H + tl.y - 1) / tl.y), lists);
        switch (tl.cpt) {
        case 1: launch_chained(gather_sum_direct_kernel<T, R, 1, SHARED>, grid, 256, 0, stream, g); break;
        case 2: launch_chained(gather_sum_direct_kernel<T, R, 2, SHARED>, grid, 256, 0, stream, g); break;
        default: launch_chained(gather_sum_direct_kernel<T, R, 4, SHARED>, grid, 256, 0, stream, g); break;
        }
    };
    if (pl.staged) {
        if (pl.smem > 48 * 1024) {     // per-device attribute of the kernel: set on every launch (cheap, idempotent, thread-safe)
            e = cudaFuncSetAttribute(gather_sum_staged_kernel<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.smem);
            if (e != cudaSuccess) return e;
        }
        const unsigned tiles = static_cast<unsigned>((g.b.W + kStagedX - 1) / kStagedX) * ((g.b.H + kStagedY - 1) / kStagedY);
        launch_chained(gather_sum_staged_kernel<T, R>, dim3(tiles, g.b.B * g.b.h), kStagedX * kStagedY * kStagedChunks, pl.smem, stream, g);
    } else {
        sums(std::false_type(), pl.one_head, g.b.B * g.b.h);
    }
    sums(std::true_type(), pl.all_heads, g.b.B);
    return cudaGetLastError();
}

template <typename T>
void launch_backward(const BwdParams &p, bool vec, dim3 grid, cudaStream_t stream)
{
    if (vec && p.r == 1) launch_chained(backward_vec_kernel<T, 1>, grid, 128, 0, stream, p);
    else if (vec && p.r == 2) launch_chained(backward_vec_kernel<T, 2>, grid, 128, 0, stream, p);
    else launch_chained(backward_kernel<T>, grid, 128, 0, stream, p);
}

}  // namespace
}  // namespace matchattn

namespace matchattn {
namespace {

// Arguments both entry points share: checked here, on the host.
int backward_params(BwdParams &p, const void *max_offset, const void *q, const void *k, const void *v, const void *d_out, const void *d_attn,
                    void *d_q, void *d_max_offset, int B, int H, int W, int h, int hd, int rx, int ry, int dtype, int attn_type,
                    float scale, int q_row_begin, int q_row_end)
{
    if (!max_offset || !q || !k || !v || !d_out || !d_q) return MATCHATTN_ERR_NULL;
    if (dtype != MATCHATTN_F32 && dtype != MATCHATTN_F16 && dtype != MATCHATTN_BF16) return MATCHATTN_ERR_DTYPE;
    if (attn_type != MATCHATTN_L1_NORM) return MATCHATTN_ERR_ATTN_TYPE;
    if (B <= 0 || H <= 0 || W <= 0 || h <= 0 || hd <= 0) return MATCHATTN_ERR_SHAPE;
    if (q_row_begin < 0 || q_row_end > H || q_row_begin >= q_row_end) return MATCHATTN_ERR_SHAPE;
    if (rx != ry || rx < 0 || rx > MATCHATTN_MAX_R) return MATCHATTN_ERR_WINDOW;
    if (2 * rx + 2 > W || 2 * ry + 2 > H) return MATCHATTN_ERR_WINDOW_FIT;
    const long long C = 1LL * h * hd, N = 1LL * H * W, Nq = 1LL * (q_row_end - q_row_begin) * W;
    if (C > 65536 || N * C >= 2147483647LL || Nq * h >= 2147483647LL || B > 65535) return MATCHATTN_ERR_TOO_LARGE;
    const uintptr_t esize = dtype == MATCHATTN_F32 ? 4 : 2;
    const std::initializer_list<const void *> arrays = {max_offset, q, k, v, d_out, d_attn, d_q, d_max_offset};
    for (const void *ptr : arrays)
        if (reinterpret_cast<uintptr_t>(ptr) % esize != 0) return MATCHATTN_ERR_ALIGN;
    p.mo = max_offset; p.q = q; p.k = k; p.v = v; p.dout = d_out; p.dattn = d_attn;
    p.dq = d_q; p.dmo = d_max_offset;
    p.B = B; p.H = H; p.W = W; p.h = h; p.hd = hd; p.C = static_cast<int>(C); p.r = rx;
    p.rows = q_row_end - q_row_begin; p.Nq = static_cast<int>(Nq); p.N = static_cast<int>(N);
    p.scale = scale;
    return MATCHATTN_OK;
}

inline bool aligned16(const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

}  // namespace
}  // namespace matchattn

extern "C" int matchattn_fused_backward(const void *max_offset, const void *q, const void *k, const void *v,
                                        const void *d_out, const void *d_attn, void *d_q, float *d_k, float *d_v,
                                        void *d_max_offset, int B, int H, int W, int h, int hd, int rx, int ry, int dtype,
                                        int attn_type, float scale, int q_row_begin, int q_row_end, void *cuda_stream)
{
    using namespace matchattn;
    if (!d_k || !d_v) return MATCHATTN_ERR_NULL;
    BwdParams p{};
    const int status = backward_params(p, max_offset, q, k, v, d_out, d_attn, d_q, d_max_offset, B, H, W, h, hd, rx, ry, dtype,
                                       attn_type, scale, q_row_begin, q_row_end);
    if (status != MATCHATTN_OK) return status;
    if (((reinterpret_cast<uintptr_t>(d_k) | reinterpret_cast<uintptr_t>(d_v)) & 3u) != 0) return MATCHATTN_ERR_ALIGN;
    p.dk = d_k; p.dv = d_v;
    const dim3 grid(static_cast<unsigned>((1LL * p.Nq * h + 127) / 128), B);
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    // the vector kernel: head width a multiple of 8, r = 1 or 2, 16-byte aligned rows everywhere
    const bool vec = hd % 8 == 0 && (rx == 1 || rx == 2) && aligned16(q) && aligned16(k) && aligned16(v) && aligned16(d_out) &&
                     aligned16(d_q) && aligned16(d_k) && aligned16(d_v);
    switch (dtype) {
    case MATCHATTN_F32: launch_backward<float>(p, vec, grid, stream); break;
    case MATCHATTN_F16: launch_backward<__half>(p, vec, grid, stream); break;
    default: launch_backward<__nv_bfloat16>(p, vec, grid, stream); break;
    }
    const cudaError_t err = cudaGetLastError();
    return status_of(err);
}

extern "C" size_t matchattn_backward_workspace_bytes(int B, int H, int W, int h, int hd, int r, int dtype, int q_row_begin, int q_row_end)
{
    if (B <= 0 || H <= 0 || W <= 0 || h <= 0 || hd <= 0 || q_row_begin < 0 || q_row_end > H || q_row_begin >= q_row_end) return 0;
    return matchattn::gather_plan(B, H, W, h, hd, r, dtype, 1LL * (q_row_end - q_row_begin) * W).bytes;
}

extern "C" int matchattn_fused_backward_ws(const void *max_offset, const void *q, const void *k, const void *v,
                                           const void *d_out, const void *d_attn, void *d_q, void *d_k, void *d_v,
                                           void *d_max_offset, int B, int H, int W, int h, int hd, int rx, int ry, int dtype,
                                           int attn_type, float scale, int q_row_begin, int q_row_end, void *workspace,
                                           size_t workspace_bytes, void *cuda_stream)
{
    using namespace matchattn;
    if (!d_k || !d_v || !workspace) return MATCHATTN_ERR_NULL;
    GatherParams g{};
    const int status = backward_params(g.b, max_offset, q, k, v, d_out, d_attn, d_q, d_max_offset, B, H, W, h, hd, rx, ry, dtype,
                                       attn_type, scale, q_row_begin, q_row_end);
    if (status != MATCHATTN_OK) return status;
    const GatherPlan pl = gather_plan(B, H, W, h, hd, rx, dtype, g.b.Nq);
    const auto aligned32 = [](const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 31u) == 0; };
    // (a centre is read as one word of two elements)
    if (pl.bytes == 0 || workspace_bytes < pl.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0 ||
        reinterpret_cast<uintptr_t>(max_offset) % (dtype == MATCHATTN_F32 ? 8 : 4) != 0 || !aligned32(q) ||
        !aligned32(k) || !aligned32(v) || !aligned32(d_out) || !aligned32(d_attn) || !aligned32(d_q) || !aligned32(d_k) || !aligned32(d_v))
        return MATCHATTN_ERR_VARIANT;
    char *ws = static_cast<char *>(workspace);
    g.dk = d_k; g.dv = d_v;
    g.cells_x = pl.cells_x; g.cells_y = pl.cells_y;
    g.lph = pl.lph;
    while ((1 << g.lph_shift) < pl.lph) ++g.lph_shift;
    g.items = static_cast<int64_t>(B) * g.b.Nq * h;
    g.counts = reinterpret_cast<int *>(ws);
    g.cursor = reinterpret_cast<int *>(ws + pl.off_cursor);
    g.differ = g.cursor + 1;
    g.all_heads = pl.all_heads; g.one_head = pl.one_head;
    g.starts = reinterpret_cast<int *>(ws + pl.off_starts);
    g.rank = reinterpret_cast<int *>(ws + pl.off_rank);
    g.meta = reinterpret_cast<int2 *>(ws + pl.off_meta);
    g.coef = reinterpret_cast<float2 *>(ws + pl.off_coef);
    g.batch = pl.batch;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    const auto run = [&](auto tag) {
        using T = decltype(tag);
        return rx == 1 ? launch_gather<T, 1>(g, pl, stream) : launch_gather<T, 2>(g, pl, stream);
    };
    const cudaError_t err = dtype == MATCHATTN_F32 ? run(float()) : dtype == MATCHATTN_F16 ? run(__half()) : run(__nv_bfloat16());
    return status_of(err);
}
