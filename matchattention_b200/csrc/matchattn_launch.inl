// Included once per element type with MATCHATTN_T defined: instantiates the
// specialised kernels for that type and the switch that picks one.
#include <type_traits>

#include "matchattn_kernels.cuh"
#include "matchattn_lanes.cuh"
#ifdef MATCHATTN_T_IS_16BIT
#include "matchattn_mma.cuh"
#include "matchattn_binned.cuh"
#include "matchattn_staged.cuh"
#endif

namespace matchattn {

// One lane per head is what a call without knobs gets for these slices only (wider heads are spread over lanes, up to 64
// heads at least): they have the builds without the rare options, which are 4 to 9 % faster.
template <typename T, int CPL>
constexpr bool kPlainBuilds = CPL != 4 && !(sizeof(T) == 4 && CPL == 2);

template <typename T, int R>
static cudaError_t launch_fast_r(const Params &p, int cpl, bool multi, dim3 grid, int threads, cudaStream_t stream)
{
    const bool glue = p.gate != nullptr || p.clamp != 0 || p.kv_shift != 0 || p.out_stride != p.C ||
                      p.attn_stride != p.h * (2 * R + 2) * (2 * R + 2);
    const bool rare = multi || p.guard != nullptr || p.sorted != nullptr || p.debug != nullptr;
    // power-of-two scale: builds that finish two scores per packed instruction
    constexpr bool kCanPack = sizeof(T) == 2;
    const bool pow2 = kCanPack && p.scale_pow2 != 0;
    const auto one_lane = [&](auto chunks) {
        constexpr int CPL = decltype(chunks)::value;
        if constexpr (kPlainBuilds<T, CPL>) {
            if (!rare) {
                if (glue && pow2) launch_chained(fused_forward_kernel<T, R, CPL, false, kGlueOptions, kCanPack>, grid, threads, 0, stream, p);
                else if (glue) launch_chained(fused_forward_kernel<T, R, CPL, false, kGlueOptions>, grid, threads, 0, stream, p);
                else if (pow2) launch_chained(fused_forward_kernel<T, R, CPL, false, kNoOptions, kCanPack>, grid, threads, 0, stream, p);
                else launch_chained(fused_forward_kernel<T, R, CPL, false, kNoOptions>, grid, threads, 0, stream, p);
                return cudaGetLastError();
            }
        }
        launch_chained(fused_forward_kernel<T, R, CPL, false, kAllOptions>, grid, threads, 0, stream, p);
        return cudaGetLastError();
    };
#define MA_CASE(CPL_)                                                                            \
    if (cpl == CPL_) {                                                                           \
        if (!multi) return one_lane(std::integral_constant<int, CPL_>());                        \
        launch_chained(fused_forward_kernel<T, R, CPL_, true, kAllOptions>, grid, threads, 0, stream, p);    \
        return cudaGetLastError();                                                               \
    }
    MA_CASE(1) MA_CASE(2) MA_CASE(3) MA_CASE(4) MA_CASE(5)
#undef MA_CASE
    return cudaErrorInvalidValue;
}

// load: blocks of 256 threads per SM, rounded up.  Calls whose blocks the host has cut in half (fewer than ten per SM) wait for
// their taps more than they fill the chip.  A build for two blocks per SM has the registers to keep more of them on their way,
// and pays where it goes through no more rounds than the one for three, at a load of 1, 2 or 4.  Three blocks / two: float16, 4
// heads x 64, 64x64 tokens 5.9 / 5.8 us, 72x72 (load 3) 6.8 / 7.5, 2 x 64x64 11.7 / 10.7, 104x104 (load 5) 14.1 / 14.3; 4 x 32,
// 104x104 (load 3) 7.3 / 7.9; float32, 8 x 16, 72x72 6.7 / 7.3, 2 x 64x64 12.8 / 10.7.  Two lanes per float32 head gain by the
// registers at higher loads too (8 x 16, 104x208 23.8 / 23.1, a centre per head 30.2 / 29.4); full blocks lose (2 x 192x192, 4 x 64,
// float32 128 / 144).
template <typename T, int R, int CPL, int L, bool RAGGED>
static cudaError_t launch_lanes_one(const Params &p, dim3 grid, int threads, int load, cudaStream_t stream)
{
    if constexpr (lanes_min_blocks<T, R, CPL>() > 2) {
        if (threads < kThreads && ((load + 1) / 2 == (load + 2) / 3 || (sizeof(T) == 4 && L == 2 && load > 4)))
            return launch_chained(lanes_forward_kernel<T, R, CPL, L, RAGGED, 2>, grid, threads, 0, stream, p);
    }
    return launch_chained(lanes_forward_kernel<T, R, CPL, L, RAGGED>, grid, threads, 0, stream, p);
}

// The splits that calls get without knobs (float32 on (2, 2) and (2, 4): from 33 heads on, r = 2); any other runs on the
// kernel above, so do 33 to 64 heads of 128 channels at r = 1.
template <typename T, int R>
static bool launch_lanes_r(const Params &p, int cpl, dim3 grid, int threads, int load, cudaStream_t stream, cudaError_t &err)
{
    const int width = p.hd / 8;      // chunks of a head
#define MA_LANES(CPL_, L_)                                                         \
    if (cpl == CPL_ && p.lph == L_ && width == CPL_ * L_) {                        \
        err = launch_lanes_one<T, R, CPL_, L_, false>(p, grid, threads, load, stream); \
        return true;                                                               \
    }
    MA_LANES(2, 2) MA_LANES(2, 4) MA_LANES(2, 8) MA_LANES(4, 8)
    MA_LANES(3, 2) MA_LANES(3, 4) MA_LANES(5, 2)
    if constexpr (sizeof(T) == 2) {
        if (cpl == 3 && p.lph == 2 && width == 5) {
            err = launch_lanes_one<T, R, 3, 2, true>(p, grid, threads, load, stream);
            return true;
        }
    } else {
        MA_LANES(1, 2) MA_LANES(1, 4) MA_LANES(1, 8)
    }
#undef MA_LANES
    return false;
}

template <>
bool launch_lanes<MATCHATTN_T>(const Params &p, int r, int cpl, dim3 grid, int threads, int load, cudaStream_t stream, cudaError_t &err)
{
    return r == 1 ? launch_lanes_r<MATCHATTN_T, 1>(p, cpl, grid, threads, load, stream, err)
                  : launch_lanes_r<MATCHATTN_T, 2>(p, cpl, grid, threads, load, stream, err);
}

template <>
cudaError_t launch_fast<MATCHATTN_T>(const Params &p, int r, int cpl, bool multi, dim3 grid, int threads, cudaStream_t stream)
{
    if (r == 1) return launch_fast_r<MATCHATTN_T, 1>(p, cpl, multi, grid, threads, stream);
    if (r == 2) return launch_fast_r<MATCHATTN_T, 2>(p, cpl, multi, grid, threads, stream);
    return cudaErrorInvalidValue;
}

#ifdef MATCHATTN_T_IS_16BIT
template <typename T, int CPL>
static cudaError_t launch_mma_cpl(const Params &p, bool sameq, bool pow2, int nch, unsigned blocks, cudaStream_t stream)
{
    if (nch == 1) {
        if (pow2) fused_forward_mma_kernel<T, CPL, false, true, 1><<<blocks, kThreads, 0, stream>>>(p);
        else fused_forward_mma_kernel<T, CPL, false, false, 1><<<blocks, kThreads, 0, stream>>>(p);
    } else if (sameq && pow2) fused_forward_mma_kernel<T, CPL, true, true, 2><<<blocks, kThreads, 0, stream>>>(p);
    else if (sameq) fused_forward_mma_kernel<T, CPL, true, false, 2><<<blocks, kThreads, 0, stream>>>(p);
    else if (pow2) fused_forward_mma_kernel<T, CPL, false, true, 2><<<blocks, kThreads, 0, stream>>>(p);
    else fused_forward_mma_kernel<T, CPL, false, false, 2><<<blocks, kThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

template <>
cudaError_t launch_mma<MATCHATTN_T>(const Params &p, int cpl, bool sameq, bool pow2, int nch, unsigned blocks,
                                    cudaStream_t stream)
{
    switch (cpl) {
    case 1: return launch_mma_cpl<MATCHATTN_T, 1>(p, sameq, pow2, nch, blocks, stream);
    case 2: return launch_mma_cpl<MATCHATTN_T, 2>(p, sameq, pow2, nch, blocks, stream);
    case 3: return launch_mma_cpl<MATCHATTN_T, 3>(p, sameq, pow2, nch, blocks, stream);
    case 4: return launch_mma_cpl<MATCHATTN_T, 4>(p, sameq, pow2, nch, blocks, stream);
    case 5: return launch_mma_cpl<MATCHATTN_T, 5>(p, sameq, pow2, nch, blocks, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <typename T, int CPL, bool SAMEQ>
static cudaError_t launch_binned_one(const BinParams &bp, int grid_blocks, size_t smem_bytes, cudaStream_t stream)
{
    // The opt-in to large dynamic shared memory is a per-device attribute of the kernel: it is set on
    // every launch (cheap, idempotent, safe from any host thread) rather than remembered per process.
    cudaError_t e = cudaFuncSetAttribute(binned_forward_kernel<T, CPL, SAMEQ>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxBinnedSmem));
    if (e != cudaSuccess) return e;
    binned_forward_kernel<T, CPL, SAMEQ><<<grid_blocks, kBinThreads, smem_bytes, stream>>>(bp);
    return cudaGetLastError();
}

template <typename T, int CPL>
static cudaError_t launch_binned_cpl(const BinParams &bp, int grid_blocks, size_t smem_bytes, cudaStream_t stream)
{
    return bp.p.h % 8 == 0 ? launch_binned_one<T, CPL, true>(bp, grid_blocks, smem_bytes, stream)
                           : launch_binned_one<T, CPL, false>(bp, grid_blocks, smem_bytes, stream);
}

template <>
cudaError_t launch_binned<MATCHATTN_T>(const BinParams &bp, int cpl, int grid_blocks, size_t smem_bytes,
                                       cudaStream_t stream)
{
    const Params &p = bp.p;
    const long long total = 1LL * p.B * p.Nq;
    const unsigned qblocks = static_cast<unsigned>((total + 255) / 256);
    bin_count_kernel<MATCHATTN_T, 1><<<qblocks, 256, 0, stream>>>(bp);
    bin_scan_kernel<<<1, 1024, 0, stream>>>(bp);
    bin_scatter_kernel<<<qblocks, 256, 0, stream>>>(bp);
    switch (cpl) {
    case 0: return cudaGetLastError();       // sorting passes only
    case 1: return launch_binned_cpl<MATCHATTN_T, 1>(bp, grid_blocks, smem_bytes, stream);
    case 2: return launch_binned_cpl<MATCHATTN_T, 2>(bp, grid_blocks, smem_bytes, stream);
    case 3: return launch_binned_cpl<MATCHATTN_T, 3>(bp, grid_blocks, smem_bytes, stream);
    case 4: return launch_binned_cpl<MATCHATTN_T, 4>(bp, grid_blocks, smem_bytes, stream);
    case 5: return launch_binned_cpl<MATCHATTN_T, 5>(bp, grid_blocks, smem_bytes, stream);
    default: return cudaErrorInvalidValue;
    }
}
#endif

#ifdef MATCHATTN_T_IS_16BIT
template <typename T, int CPL, bool POW2>
static cudaError_t launch_staged_one(const StagedParams &sp, const CUtensorMap &map_k, const CUtensorMap &map_v, dim3 grid,
                                     size_t smem_bytes, cudaStream_t stream)
{
    // per-device attribute of the kernel: set on every launch (cheap, idempotent, thread-safe)
    cudaError_t e = cudaFuncSetAttribute(staged_forward_kernel<T, CPL, POW2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kStagedRegionBytes + 128));
    if (e != cudaSuccess) return e;
    staged_forward_kernel<T, CPL, POW2><<<grid, kStagedThreads, smem_bytes, stream>>>(sp, map_k, map_v);
    return cudaGetLastError();
}

template <typename T, int CPL, bool POW2>
static cudaError_t launch_persist_one(const PersistParams &sp, const CUtensorMap &map_k, const CUtensorMap &map_v,
                                      int grid_blocks, cudaStream_t stream)
{
    const size_t smem_bytes = 2 * kPersistRegionBytes + 128;
    cudaError_t e = cudaFuncSetAttribute(staged_persistent_kernel<T, CPL, POW2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem_bytes));
    if (e != cudaSuccess) return e;
    staged_persistent_kernel<T, CPL, POW2><<<grid_blocks, kPersistThreads, smem_bytes, stream>>>(sp, map_k, map_v);
    return cudaGetLastError();
}

template <>
cudaError_t launch_staged_persistent<MATCHATTN_T>(const PersistParams &sp, int cpl, const CUtensorMap &map_k,
                                                  const CUtensorMap &map_v, int grid_blocks, cudaStream_t stream)
{
    const bool pow2 = sp.p.scale_pow2 != 0;
    if (cpl == 1) return pow2 ? launch_persist_one<MATCHATTN_T, 1, true>(sp, map_k, map_v, grid_blocks, stream)
                              : launch_persist_one<MATCHATTN_T, 1, false>(sp, map_k, map_v, grid_blocks, stream);
    if (cpl == 2) return pow2 ? launch_persist_one<MATCHATTN_T, 2, true>(sp, map_k, map_v, grid_blocks, stream)
                              : launch_persist_one<MATCHATTN_T, 2, false>(sp, map_k, map_v, grid_blocks, stream);
    return cudaErrorInvalidValue;
}

template <>
cudaError_t launch_staged<MATCHATTN_T>(const StagedParams &sp, int cpl, const CUtensorMap &map_k, const CUtensorMap &map_v,
                                       dim3 grid, size_t smem_bytes, cudaStream_t stream)
{
    const bool pow2 = sp.p.scale_pow2 != 0;
    if (cpl == 1) return pow2 ? launch_staged_one<MATCHATTN_T, 1, true>(sp, map_k, map_v, grid, smem_bytes, stream)
                              : launch_staged_one<MATCHATTN_T, 1, false>(sp, map_k, map_v, grid, smem_bytes, stream);
    if (cpl == 2) return pow2 ? launch_staged_one<MATCHATTN_T, 2, true>(sp, map_k, map_v, grid, smem_bytes, stream)
                              : launch_staged_one<MATCHATTN_T, 2, false>(sp, map_k, map_v, grid, smem_bytes, stream);
    return cudaErrorInvalidValue;
}
#endif

template <>
cudaError_t launch_generic<MATCHATTN_T>(const Params &p, dim3 grid, cudaStream_t stream)
{
    launch_chained(generic_forward_kernel<MATCHATTN_T>, grid, kThreads, 0, stream, p);
    return cudaGetLastError();
}

}  // namespace matchattn
