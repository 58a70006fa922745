// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point
// and the reference interface each one replaces.
#include "adkv_host.h"

#include "adkv_io.cuh"
#include "adkv_narrow.cuh"

namespace adkv {

// =========================================================================================
// Unfused entry points (the reference's two-kernel decode): 2 streams per CTA, one warp each.

// Tokens per tile (see kFusedStages in adkv_fused.cu): the three calls at 512 streams x 1023 tokens 118.7 -> 108.7 us.  Eight query
// heads leave no room for 64, and three tiles of 32 in flight are the faster ones there: 2-bit, 64 streams x 1000 tokens 117 -> 115 us.
template <int G>
constexpr int kQkTok = G > 4 ? kTileTok : 64;
template <int G>
constexpr int kQkStages = G > 4 ? 3 : 2;

template <int BITS, int G, bool EXACT>
__global__ void __launch_bounds__(32 * kStreamsPerCta) forward_qk_kernel(KArgs ka, __half *__restrict__ logits,
                                                                         int n_streams)
{
    __shared__ alignas(128) uint8_t kbuf[kStreamsPerCta][kQkStages<G> * Tile<BITS, kQkTok<G>>::BYTES];
    __shared__ alignas(16) float red[kStreamsPerCta][G * kRedTok<G> * kRedRow];
    __shared__ uint64_t kbar[kStreamsPerCta][kQkStages<G>];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        for (int i = 0; i < kQkStages<G>; ++i) mbar_init(&kbar[warp][i], 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int bh = blockIdx.x * kStreamsPerCta + warp;
    if (bh >= n_streams) return;
    const int b = bh / ka.Hkv, h = bh % ka.Hkv;
    GlobalLogitSink<G, kQkTok<G>> sink;
#pragma unroll
    for (int g = 0; g < G; ++g) sink.row[g] = logits + (size_t(b) * ka.Hq + size_t(h) * G + g) * (ka.T + 1);
    sink.T = ka.T;
    const Seg seg{0, ka.T, true, nullptr, nullptr, 0};
    k_warp<BITS, G, EXACT, GlobalLogitSink<G, kQkTok<G>>, kQkStages<G>, false, false, kRedTok<G>, kQkTok<G>>(ka, seg, b, h, lane, kbuf[warp],
                                                                                                    kbar[warp], red[warp], sink);
}

// Tokens per tile, as for forward_qk: the three calls at 512 streams x 1023 tokens 106.6 -> 99.6 us, 2048 x 2000 530 -> 512 us.
constexpr int kOvTok = 64, kOvStages = 2;

template <int BITS, int G, bool EXACT>
__global__ void __launch_bounds__(32 * kStreamsPerCta) forward_ov_kernel(VArgs va, const __half *__restrict__ attn,
                                                                         int n_streams)
{
    __shared__ alignas(128) uint8_t vbuf[kStreamsPerCta][kOvStages * Tile<BITS, kOvTok>::BYTES];
    __shared__ alignas(16) float2 wts[kStreamsPerCta][G * kOvTok];
    __shared__ uint64_t vbar[kStreamsPerCta][kOvStages];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        for (int i = 0; i < kOvStages; ++i) mbar_init(&vbar[warp][i], 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int bh = blockIdx.x * kStreamsPerCta + warp;
    if (bh >= n_streams) return;
    const int b = bh / va.Hkv, h = bh % va.Hkv;
    GlobalWeightSrc<G, false, kOvTok> src;
#pragma unroll
    for (int g = 0; g < G; ++g) src.row[g] = attn + (size_t(b) * va.Hq + size_t(h) * G + g) * (va.T + 1);
    src.wts = wts[warp];
    src.T = va.T;
    const Seg seg{0, va.T, true, nullptr, nullptr, 0};
    v_warp<BITS, G, EXACT, GlobalWeightSrc<G, false, kOvTok>, kOvStages, false, false, kOvTok>(va, seg, b, h, lane, vbuf[warp], vbar[warp], wts[warp], src);
}

// forward_ov with few streams: two warps per stream, 64 channels each (adkv_narrow.cuh).  Output channels are independent,
// so the two warps have nothing to exchange; what is repeated is the staging of the weights.
template <int BITS, int G, bool EXACT>
__global__ void __launch_bounds__(32 * kNarrowSlices) forward_ov_split_kernel(VArgs va, const __half *__restrict__ attn)
{
    constexpr int S = kNarrowSlices;
    __shared__ alignas(128) uint8_t vbuf[S][kStages * NarrowTile<BITS>::BYTES];
    __shared__ alignas(16) float2 wts[S][G * kTileTok];
    __shared__ uint64_t vbar[S][kStages];
    const int sl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        for (int i = 0; i < kStages; ++i) mbar_init(&vbar[sl][i], 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int bh = blockIdx.x, b = bh / va.Hkv, h = bh % va.Hkv;
    GlobalWeightSrc<G> src;
#pragma unroll
    for (int g = 0; g < G; ++g) src.row[g] = attn + (size_t(b) * va.Hq + size_t(h) * G + g) * (va.T + 1);
    src.wts = wts[sl];
    src.T = va.T;
    const Seg seg{0, va.T, true, nullptr, nullptr, sl};
    v_warp_n<BITS, G, EXACT ? kArithCanon : kArithFma>(va, seg, b, h, lane, vbuf[sl], vbar[sl], wts[sl], src);
}

// forward_ov splits a stream over two warps while each of them has a scheduler to itself: up to 296 streams.  Measured on
// a B200, 1000 tokens, one warp (tiles of 64 tokens, weights fetched ahead) -> two, us, canonical replay where no scale meets a clamp /
// where one channel of every head rests at a bound; contracted replay, the same:
//    256 streams    4-bit 38.0 -> 41.5 / 41.2 -> 53.8; 34.4 -> 39.4 / 38.2 -> 50.9
//                   four heads 55.6 -> 50.0 / 60.7 -> 64.5; 50.2 -> 48.6 / 55.3 -> 60.1
//                   2-bit 51.2 -> 44.5 / 52.1 -> 53.0; 46.1 -> 42.8 / 47.9 -> 52.1
//                   four heads 60.1 -> 58.0 / 65.2 -> 66.2; 55.9 -> 55.9 / 59.1 -> 63.2
//    320 streams    4-bit 38.2 -> 49.7, four heads 55.9 -> 62.1; 2-bit 50.9 -> 54.7, four heads 60.1 -> 71.3 (canonical, no clamp)
// Two warps are the better choice there for several heads and for 2-bit codes away from the bounds; 4-bit codes of one head are the
// exception since one warp takes tiles of 64.
constexpr int kOvSplitMaxStreams = kSchedulers / 2;

}  // namespace adkv

using namespace adkv;

ADKV_HIDDEN int adkv_half_forward_qk(const KArgs &ka, __half *logits, int B, int bits, cudaStream_t s);
ADKV_HIDDEN int adkv_half_forward_ov(const VArgs &va, const __half *attn, int B, int bits, cudaStream_t s);
ADKV_HIDDEN int adkv_wide_forward_qk(const KArgs &ka, __half *logits, int B, int bits, int mode, cudaStream_t s);
ADKV_HIDDEN int adkv_wide_forward_ov(const VArgs &va, const __half *attn, int B, int bits, int mode, cudaStream_t s);

ADKV_DEFINE_TU_STATUS(adkv_tu_status_unfused)

extern "C" {

int adkv_forward_qk(const void *q, void *k_cache, const void *k_new, const adkv_params *p, void *logits, int B,
                    int Hq, int Hkv, int T, int D, int n_super_cap, int bits, float scale_min, float scale_max,
                    unsigned flags, void *stream)
{
    if (!q || !k_cache || !k_new || !logits || !params_ok(p)) return ADKV_E_NULL;
    if (int rc = check_common(B, Hq, Hkv, T, D, n_super_cap, bits, T + 1)) return rc;
    if (!aligned16(k_cache) || !aligned8(q) || !aligned8(k_new) || !params_aligned(p)) return ADKV_E_ALIGN;
    if (B == 0) return 0;
    const KArgs ka{static_cast<const __half *>(q), static_cast<uint8_t *>(k_cache),
                   static_cast<const __half *>(k_new), to_ptrs(p), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D};
    const int n_streams = B * Hkv, grid = (n_streams + kStreamsPerCta - 1) / kStreamsPerCta;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool half = flags & ADKV_FLAG_HALF_STATE, exact = !(flags & ADKV_FLAG_FAST_REPLAY);
    if (D != kD) return adkv_wide_forward_qk(ka, static_cast<__half *>(logits), B, bits, half ? 2 : int(exact), s);
    if (half) return adkv_half_forward_qk(ka, static_cast<__half *>(logits), B, bits, s);
    ADKV_DISPATCH(bits, exact, Hq / Hkv,
                  (forward_qk_kernel<BITS, G, EXACT><<<grid, 32 * kStreamsPerCta, 0, s>>>(
                      ka, static_cast<__half *>(logits), n_streams)))
    return launch_status();
}

int adkv_forward_ov(const void *attn, void *v_cache, const void *v_new, const adkv_params *p, void *out, int B,
                    int Hq, int Hkv, int T, int D, int n_super_cap, int bits, float scale_min, float scale_max,
                    unsigned flags, void *stream)
{
    if (!attn || !v_cache || !v_new || !out || !params_ok(p)) return ADKV_E_NULL;
    if (int rc = check_common(B, Hq, Hkv, T, D, n_super_cap, bits, T + 1)) return rc;
    if (!aligned16(v_cache) || !aligned8(out) || !aligned8(v_new) || !params_aligned(p)) return ADKV_E_ALIGN;
    if (B == 0) return 0;
    const VArgs va{static_cast<uint8_t *>(v_cache), static_cast<const __half *>(v_new), static_cast<__half *>(out),
                   to_ptrs(p), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D};
    const int n_streams = B * Hkv, grid = (n_streams + kStreamsPerCta - 1) / kStreamsPerCta;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool half = flags & ADKV_FLAG_HALF_STATE, exact = !(flags & ADKV_FLAG_FAST_REPLAY);
    if (D != kD) return adkv_wide_forward_ov(va, static_cast<const __half *>(attn), B, bits, half ? 2 : int(exact), s);
    if (half) return adkv_half_forward_ov(va, static_cast<const __half *>(attn), B, bits, s);
    if (n_streams <= kOvSplitMaxStreams) {
        ADKV_DISPATCH(bits, exact, Hq / Hkv,
                      (forward_ov_split_kernel<BITS, G, EXACT><<<n_streams, 32 * kNarrowSlices, 0, s>>>(
                          va, static_cast<const __half *>(attn))))
        return launch_status();
    }
    ADKV_DISPATCH(bits, exact, Hq / Hkv,
                  (forward_ov_kernel<BITS, G, EXACT><<<grid, 32 * kStreamsPerCta, 0, s>>>(
                      va, static_cast<const __half *>(attn), n_streams)))
    return launch_status();
}

}  // extern "C"
