// MatchAttention forward for heads that several lanes share (L = 2, 4 or 8 lanes of a warp).
//
// Each lane owns CPL chunks of 8 channels.  What does not depend on the channels -- scores, exponentials, the four
// sub-window softmaxes and their blend -- is split over the lanes as well, by rows of the window: the partial L1 sums
// are reduced AND scattered in one go (a lane ends up with the finished sums of its own rows: r = 1, L = 4: 12 shuffles
// per window where a full exchange takes 32), every lane evaluates its rows, and the finished weights, two to a word in
// the 16-bit types, are gathered for the sum over the value taps.
//
// A lane's chunks lie in 32-byte pieces, piece i of lane s at piece i * lanes + s of the head: the lanes of a query read
// whole lines of a token.  Odd chunk counts in the 16-bit types take 16-byte pieces (hd = 80 on two lanes: 58 us where
// 32-byte pieces and a last one of 16 took 71: their eight neighbouring registers leave the compiler less room).
//
// RAGGED (16-bit types, hd = 40): a 32-byte piece per lane and a 16-byte one for lane 0; lane 1 reads that along and
// leaves it out.  Every other head starts half way into a 32-byte piece and has its 16-byte piece in front.
// Measured, float16, r = 2, 4 heads: 2 x 48x48 tokens 13.4 -> 11.4 us, 2 x 160x160 125 -> 112 (one lane per head:
// five loads per tap that touch a line per lane each, L1 71 % busy, issue 29 %).
//
// Bound by instruction issue and the L1 path (61 and 67 % at bfloat16 heads of 64, r = 1); r = 2 by the latency of the taps at
// two blocks per SM (issue 60 %, L1 54 to 63 %).  Measured on a B200 against one lane's full softmax in every lane and
// 64-byte slices: float16, 2 x 272x480 tokens, 4 heads x 64, r = 1: 320 -> 225 us; 2 x 68x120, 4 x 128, r = 2:
// 101 -> 78; float32, 2 x 192x192, 4 x 64, r = 1: 399 -> 160.
#pragma once

#include "matchattn_kernels.cuh"

namespace matchattn {

// Which rows of the window a lane evaluates.
template <int R, int L>
struct RowShare {
    static constexpr int SIDE = 2 * R + 2;
    static constexpr int ROWS = R == 1 ? (L == 2 ? 2 : 1) : (L == 2 ? 3 : L == 4 ? 2 : 1);   // per lane
    static_assert((R == 1 || R == 2) && (L == 2 || L == 4 || L == 8), "");
    static __device__ __forceinline__ int first(int sl)
    {
        if (R == 1) return L == 2 ? 2 * sl : L == 4 ? sl : sl >> 1;
        return L == 2 ? 3 * sl : L == 4 ? min(2 * sl, 4) : sl < 4 ? sl : sl < 6 ? 4 : 5;
    }
    // the lane that speaks for a row, and the row's place among that lane's rows
    static constexpr __host__ __device__ int owner(int j)
    {
        if (R == 1) return L == 2 ? j / 2 : L == 4 ? j : 2 * j;
        return L == 2 ? j / 3 : L == 4 ? j / 2 : j < 4 ? j : 2 * j - 4;
    }
    static constexpr __host__ __device__ int place(int j) { return R == 1 ? (L == 2 ? j % 2 : 0) : L == 2 ? j % 3 : L == 4 ? j % 2 : 0; }
    static __device__ __forceinline__ bool speaks(int sl)
    {
        if (R == 1) return L != 8 || (sl & 1) == 0;
        return L == 2 || (L == 4 ? sl < 3 : sl < 5 || sl == 6);
    }

    // p: this lane's partial sums of one window column, one per row.  out: the sums over the L lanes for this lane's rows.
    static __device__ __forceinline__ void reduce(const float (&p)[SIDE], float (&out)[ROWS], int sl)
    {
        constexpr unsigned kAll = 0xffffffffu;
        const auto swap = [](float keep, float send, int o) { return keep + __shfl_xor_sync(kAll, send, o); };
        const bool hi = (sl & (L / 2)) != 0;
        if constexpr (L == 2) {
#pragma unroll
            for (int k = 0; k < ROWS; ++k) out[k] = swap(hi ? p[k + ROWS] : p[k], hi ? p[k] : p[k + ROWS], 1);
        } else if constexpr (R == 1) {
            float h[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) h[k] = swap(hi ? p[k + 2] : p[k], hi ? p[k] : p[k + 2], L / 2);
            const bool odd = (sl & (L / 4)) != 0;
            out[0] = swap(odd ? h[1] : h[0], odd ? h[0] : h[1], L / 4);
            if constexpr (L == 8) out[0] += __shfl_xor_sync(kAll, out[0], 1);
        } else {
            // the lower half of the lanes takes rows 0-3, the upper half rows 4 and 5
            float h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int up = k < 2 ? k + 4 : k;
                h[k] = swap(hi ? p[up] : p[k], hi ? p[k] : p[up], L / 2);
            }
            const bool odd = (sl & (L / 4)) != 0;
            if constexpr (L == 4) {
#pragma unroll
                for (int k = 0; k < 2; ++k) out[k] = swap(odd && !hi ? h[k + 2] : h[k], odd || hi ? h[k] : h[k + 2], 1);
            } else {
                const float q0 = swap(hi ? (odd ? h[1] : h[0]) : (odd ? h[2] : h[0]), hi ? (odd ? h[0] : h[1]) : (odd ? h[0] : h[2]), 2);
                const float q1 = swap(odd ? h[3] : h[1], odd ? h[1] : h[3], 2);      // lower half only
                const bool last = (sl & 1) != 0;
                out[0] = swap(last && !hi ? q1 : q0, last || hi ? q0 : q1, 1);
            }
        }
    }
};

// N words to an address that is a multiple of 4 * N bytes past one aligned to ALIGN bytes
template <int N, int ALIGN>
__device__ __forceinline__ void store_run(void *p, const uint32_t *w)
{
    constexpr int kBytes = 4 * N;
    constexpr int V = (kBytes % 32 == 0 && ALIGN % 32 == 0) ? 8 : (kBytes % 16 == 0 && ALIGN % 16 == 0) ? 4 : (kBytes % 8 == 0 && ALIGN % 8 == 0) ? 2 : 1;
#pragma unroll
    for (int i = 0; i < N; i += V) {
        char *at = static_cast<char *>(p) + 4 * i;
        if constexpr (V == 8) st_256(at, w + i);
        else if constexpr (V == 4) st_128(at, w + i);
        else if constexpr (V == 2) st_64(at, w + i);
        else *reinterpret_cast<uint32_t *>(at) = w[i];
    }
}

// resident blocks per SM the register allocation is held to.  r = 1 with 32-byte slices: three (80 registers; two measured
// 15 % slower, four equal); r = 2: two (128; three measured 10 % slower at two lanes per head).
template <typename T, int R, int CPL>
constexpr int lanes_min_blocks() { return R == 1 && CPL * DT<T>::kWordsPerChunk <= 8 ? 3 : 2; }

template <typename T, int R, int CPL, int L, bool RAGGED, int BLOCKS = lanes_min_blocks<T, R, CPL>()>
__global__ void __launch_bounds__(kThreads, BLOCKS) lanes_forward_kernel(const Params p)
{
    chain_begin();
    using Share = RowShare<R, L>;
    constexpr int SIDE = Share::SIDE, SUB = 2 * R + 1, ROWS = Share::ROWS;
    constexpr int NW = CPL * DT<T>::kWordsPerChunk, EPW = DT<T>::kElemsPerWord;
    constexpr int PW = RAGGED || NW % 8 == 0 ? 8 : 4, PIECES = RAGGED ? 1 : NW / PW;   // 32-bit words of a piece, pieces per lane and tap
    static_assert(!RAGGED || (NW == 12 && L == 2), "");
    constexpr int WPR = SIDE / EPW;                                // words of a row of weights
    constexpr unsigned kAll = 0xffffffffu;

    // lane -> (query of the tile, head, share of the head); lanes without a query redo a neighbour's work for the shuffles
    const int tid = threadIdx.x;
    const int lq = tid / p.G, g = tid - lq * p.G;
    const int head = g / L, sl = g & (L - 1);
    const int tile_y = blockIdx.x / p.tiles_x, tile_x = blockIdx.x - tile_y * p.tiles_x;
    int qx = tile_x * p.tile_w + (lq & (p.tile_w - 1)), qy = tile_y * p.tile_h + (lq >> p.tile_w_shift);
    const bool valid = (lq >> p.tile_w_shift) < p.tile_h && qx < p.W && qy < p.rows;
    qx = min(qx, p.W - 1);
    qy = min(qy, p.rows - 1);
    const int b = blockIdx.y;
    const int64_t bq = static_cast<int64_t>(b) * p.Nq + qy * p.W + qx;

    // sampling centre -> origin, weights, clamped tap rows / columns
    float x, y;
    DT<T>::load_xy(static_cast<const T *>(p.mo) + (bq * p.h + head) * 2, x, y);
    if (p.clamp) {
        x = clamp_keep_nan(x, p.clamp_lo, p.clamp_hi_x);
        y = clamp_keep_nan(y, p.clamp_lo, p.clamp_hi_y);
    }
    const float xf = floorf(x), yf = floorf(y);
    const int x0 = window_origin(xf, R, p.W) - R, y0 = window_origin(yf, R, p.H) - R;
    uint32_t col[SIDE];
    int row[SIDE];
#pragma unroll
    for (int i = 0; i < SIDE; ++i) {
        col[i] = static_cast<uint32_t>(min(max(x0 + i, 0), p.W - 1) * p.C) * static_cast<uint32_t>(sizeof(T));
        row[i] = min(max(y0 + i, 0), p.H - 1) * p.W * p.C;
    }

    constexpr int kPiece = PW * EPW, kStep = L * kPiece;           // elements of a piece; from one of a lane's pieces to the next
    const int shift = RAGGED && (head & 1) ? kPiece / 2 : 0;
    const int lane_off = head * p.hd + sl * kPiece + shift;
    const int tail = (shift ? -shift : kStep) - sl * kPiece;       // a ragged head's 16-byte piece, from lane_off
    const bool full = !RAGGED || sl == 0;
    const int b_kv = b + p.kv_shift >= p.B ? b + p.kv_shift - p.B : b + p.kv_shift;
    const int64_t kv_base = static_cast<int64_t>(b_kv) * p.N * p.C + lane_off;
    const T *kb = static_cast<const T *>(p.k) + kv_base;
    const T *vb = static_cast<const T *>(p.v) + kv_base;
    const auto load_slice = [&](uint32_t (&w)[NW], const T *at) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            if constexpr (PW == 8) ld_256(&w[8 * i], at + i * kStep);
            else ld_128(&w[4 * i], at + i * kStep);
        }
        if constexpr (RAGGED) ld_128(&w[8], at + tail);
    };

    uint32_t qw[NW];
    load_slice(qw, static_cast<const T *>(p.q) + bq * p.C + lane_off);

    // scores of the lane's rows, a window column at a time
    float s[ROWS][SIDE];
#pragma unroll
    for (int i = 0; i < SIDE; ++i) {
        float part[SIDE], sum[ROWS];
#pragma unroll
        for (int j = 0; j < SIDE; ++j) {
            uint32_t kw[NW];
            load_slice(kw, tap_ptr(kb + row[j], col[i]));
            float a0 = 0.f, a1 = 0.f, t0 = 0.f, t1 = 0.f;          // t: the last piece of a ragged head
            if constexpr (EPW == 1) {
#pragma unroll
                for (int w = 0; w < NW; w += 2) {
                    float d0, d1;
                    sub_f32x2(d0, d1, __uint_as_float(qw[w]), __uint_as_float(qw[w + 1]), __uint_as_float(kw[w]),
                              __uint_as_float(kw[w + 1]));
                    a0 += fabsf(d0);
                    a1 += fabsf(d1);
                }
            } else {
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    if (RAGGED && w >= 8) DT<T>::absdiff(t0, t1, qw[w], kw[w]);
                    else DT<T>::absdiff(a0, a1, qw[w], kw[w]);
                }
            }
            part[j] = a0 + a1;
            if constexpr (RAGGED) part[j] += full ? t0 + t1 : 0.f;
        }
        Share::reduce(part, sum, sl);
#pragma unroll
        for (int k = 0; k < ROWS; ++k) s[k][i] = finish_score<T>(sum[k], p.scale);
    }

    // the first value taps are requested before the softmax so that their latency overlaps it
    constexpr int VPF = (R == 1 && NW <= 8) ? 2 : 0;
    uint32_t vpre[VPF > 0 ? VPF : 1][NW];
#pragma unroll
    for (int t = 0; t < VPF; ++t) load_slice(vpre[t], tap_ptr(vb + row[0], col[t]));

    // BilinearSoftmax (see bilinear_softmax): exponentials around the window's maximum, unless a sub-window could
    // underflow there.  All sub-windows share the inner taps (rows and columns 1 .. SIDE-2): one of those within 60 of
    // the maximum rules that out.
    const int j0 = Share::first(sl);
    const bool speaks = Share::speaks(sl);
    const auto all_max = [&](float v) {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kAll, v, o));
        return v;
    };
    const auto all_sum = [&](float v) {      // neighbouring rows first, as a lane with more rows adds them
        v = speaks ? v : 0.f;
#pragma unroll
        for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(kAll, v, o);
        return v;
    };
    float top = s[0][0], inner = -INFINITY;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        float in_row = s[k][1];
#pragma unroll
        for (int i = 2; i < SIDE - 1; ++i) in_row = fmaxf(in_row, s[k][i]);
        top = fmaxf(top, fmaxf(fmaxf(s[k][0], s[k][SIDE - 1]), in_row));
        if (j0 + k > 0 && j0 + k < SIDE - 1) inner = fmaxf(inner, in_row);
    }
    top = all_max(top);
    const unsigned close = __ballot_sync(kAll, top - inner < 60.f);
    const bool shared = ((close >> (tid & 31 & ~(L - 1))) & ((1u << L) - 1u)) != 0u;      // the same for the lanes of a head

    float wgt[4];
    bilinear_weights<T>(x, xf, y, yf, wgt);
    uint32_t mine[ROWS * WPR];
#pragma unroll
    for (int w = 0; w < ROWS * WPR; ++w) mine[w] = 0u;
    // sum of a row over the columns ox .. ox + SUB - 1
    const auto row_sums = [&](const float (&e)[SIDE], float &left, float &right) {
        float m = e[1];
#pragma unroll
        for (int i = 2; i < SUB; ++i) m += e[i];
        left = e[0] + m;
        right = m + e[SIDE - 1];
    };
    // adds w_t * p_t to the weights of the lane's rows
    const auto blend = [&](const float (&e)[ROWS][SIDE], int t, float inv) {
        const int oy = t >> 1, ox = t & 1;
        const uint32_t wt_w = DT<T>::aw_bcast(wgt[t]);
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            const bool in = oy == 0 ? j0 + k < SIDE - 1 : j0 + k > 0;
            const float f = in ? inv : 0.f;                        // a row outside the sub-window adds w * 0
#pragma unroll
            for (int w = 0; w < WPR; ++w) {
                const int i0 = w * EPW, i1 = i0 + EPW - 1;
                const bool in0 = i0 >= ox && i0 < ox + SUB, in1 = i1 >= ox && i1 < ox + SUB;
                if (!in0 && !in1) continue;
                const float p0 = in0 ? e[k][i0] * f : 0.f, p1 = (EPW == 2 && in1) ? e[k][i1] * f : 0.f;
                uint32_t &dst = mine[k * WPR + w];
                dst = DT<T>::aw_add(dst, DT<T>::aw_mul(wt_w, DT<T>::aw_from(p0, p1)));
            }
        }
    };
    if (__all_sync(kAll, shared)) {
        float den[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
#pragma unroll
            for (int i = 0; i < SIDE; ++i) s[k][i] = softmax_exp(s[k][i] - top);
            float left, right;
            row_sums(s[k], left, right);
            const bool upper = j0 + k < SIDE - 1, lower = j0 + k > 0;
            den[0] += upper ? left : 0.f;
            den[1] += upper ? right : 0.f;
            den[2] += lower ? left : 0.f;
            den[3] += lower ? right : 0.f;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) den[t] = softmax_rcp(all_sum(den[t]));
#pragma unroll
        for (int t = 0; t < 4; ++t) blend(s, t, den[t]);
    } else {   // rare: widely spread scores, or a NaN score, in some head of the warp; the other heads get the same bits as above
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int oy = t >> 1, ox = t & 1;
            float mx = -INFINITY;
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                float m = s[k][ox];
#pragma unroll
                for (int i = 1; i < SUB; ++i) m = fmaxf(m, s[k][i + ox]);
                if (oy == 0 ? j0 + k < SIDE - 1 : j0 + k > 0) mx = fmaxf(mx, m);
            }
            mx = all_max(mx);
            if (shared) mx = top;
            float e[ROWS][SIDE], den = 0.f;
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const bool in = oy == 0 ? j0 + k < SIDE - 1 : j0 + k > 0;
#pragma unroll
                for (int i = 0; i < SIDE; ++i) e[k][i] = in && i >= ox && i < ox + SUB ? softmax_exp(s[k][i] - mx) : 0.f;
                float left, right;
                row_sums(e[k], left, right);
                den += ox == 0 ? left : right;
            }
            blend(e, t, softmax_rcp(all_sum(den)));
        }
    }

    if (p.attn != nullptr && speaks && valid) {
        constexpr int kBytes = SIDE * SIDE * static_cast<int>(sizeof(T)), kAlign = kBytes % 32 == 0 ? 32 : kBytes % 16 == 0 ? 16 : 8;
        store_run<ROWS * WPR, kAlign>(static_cast<T *>(p.attn) + bq * p.attn_stride + head * (SIDE * SIDE) + j0 * SIDE, mine);
    }
    uint32_t aw[SIDE * WPR];
#pragma unroll
    for (int j = 0; j < SIDE; ++j)
#pragma unroll
        for (int w = 0; w < WPR; ++w) aw[j * WPR + w] = __shfl_sync(kAll, mine[Share::place(j) * WPR + w], Share::owner(j), L);

    // weighted sum of the value taps
    float o[NW * EPW];
#pragma unroll
    for (int c = 0; c < NW * EPW; ++c) o[c] = 0.f;
#pragma unroll
    for (int j = 0; j < SIDE; ++j)
#pragma unroll
        for (int i = 0; i < SIDE; ++i) {
            uint32_t vw[NW];
            if (j * SIDE + i < VPF) {
#pragma unroll
                for (int w = 0; w < NW; ++w) vw[w] = vpre[i < VPF ? i : 0][w];
            } else {
                load_slice(vw, tap_ptr(vb + row[j], col[i]));
            }
            if constexpr (EPW == 1) {
#pragma unroll
                for (int w = 0; w < NW; w += 2)
                    fma_f32x2(o[w], o[w + 1], __uint_as_float(aw[j * SIDE + i]), __uint_as_float(vw[w]), __uint_as_float(vw[w + 1]));
            } else {
                const typename DT<T>::Bcast am = DT<T>::aw_tap(aw, j * SIDE + i);
#pragma unroll
                for (int w = 0; w < NW; ++w) DT<T>::wmul(am, vw[w], &o[w * EPW]);
            }
        }

    if (valid) {
        uint32_t ow[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) ow[w] = DT<T>::pack(&o[w * EPW]);
        if (p.gate != nullptr) {
            uint32_t gw[NW];
            load_slice(gw, static_cast<const T *>(p.gate) + bq * p.C + lane_off);
#pragma unroll
            for (int w = 0; w < NW; ++w) ow[w] = DT<T>::gate_mul(ow[w], gw[w]);
        }
        T *out = static_cast<T *>(p.out) + bq * p.out_stride + lane_off;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            if constexpr (PW == 8) st_256(out + i * kStep, &ow[8 * i]);
            else st_128(out + i * kStep, &ow[4 * i]);
        }
        if (RAGGED && full) st_128(out + tail, &ow[NW - 4]);
    }
}

// Runs the kernel above if it is built for these lanes, `err` what the launch returned; false, nothing launched, if it is not.
// load: blocks of 256 threads per SM, rounded up, as many as the launch has threads for.
template <typename T>
bool launch_lanes(const Params &p, int r, int cpl, dim3 grid, int threads, int load, cudaStream_t stream, cudaError_t &err);

}  // namespace matchattn
