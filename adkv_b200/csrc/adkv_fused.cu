// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point
// and the reference interface each one replaces.
#include "adkv_host.h"

#include "adkv_softmax.cuh"

namespace adkv {

// =========================================================================================
// Fused decode step: one CTA per (batch, kv head); warp 0 scans K, warp 1 scans V.

// Tokens per tile, and tiles in flight per warp.  Every tile costs two waits, the hand-over of its logits, a step of the online
// softmax with its shuffles, and a refill: a few hundred instructions and, for a warp that has its scheduler to itself, about
// a thousand cycles.  Tiles of 32 (three stages) -> 64 (two), device time on a B200: 2-bit, 256 streams of four heads x 32768
// tokens 2359 -> 2183 us, 4-bit x 2000 tokens 162 -> 134 us; 4096 streams x 4096 tokens 1442 -> 1411 us, 256 x 2000 98 -> 91 us,
// 768 x 1531 143 -> 136 us.  Tiles of 128 give 1 % at 2-bit codes and lose 6 % at 200 tokens.  Where the longer tiles are the
// slower ones: see short_tiles.
template <int TOK>
constexpr int kFusedStages = TOK == 64 ? 2 : 3;

// Whether the guarded chunk bodies of this instantiation are function calls (see k_chunk_guarded).  Measured on a
// B200 against the inline form, streams of 32 heads x 128: 4-bit codes with one query head per KV head gain 13 % at
// 128-token contexts and lose nothing elsewhere; 2-bit codes gain 17 % there but lose 7 % in the canonical replay and
// 14 % with 512 streams per launch, so they keep the inline form, as do the instantiations with several query heads.
template <int BITS, int G>
constexpr bool kOutOfLineGuarded = BITS == 4 && G == 1;

// n_rank: number of sequences if the CTAs may take them longest first, 0 if in the order of the batch.
template <int BITS, int G, int ARITH, int TOK>
__global__ void __launch_bounds__(64) decode_attn_kernel(KArgs ka, VArgs va, const float *__restrict__ mask,
                                                         long long mask_stride_b, float scaling,
                                                         const int *__restrict__ seq_lens, int n_rank)
{
    constexpr int ST = kFusedStages<TOK>;
    __shared__ alignas(128) uint8_t kbuf[ST * Tile<BITS, TOK>::BYTES];
    __shared__ alignas(128) uint8_t vbuf[ST * Tile<BITS, TOK>::BYTES];
    __shared__ alignas(16) float red[G * 8 * kRedRow];
    __shared__ alignas(16) float2 wts[G * TOK];
    __shared__ FusedShared<G, 1, TOK> fs;
    __shared__ uint64_t kbar[ST], vbar[ST];

    int b = blockIdx.x / ka.Hkv;
    const int h = blockIdx.x % ka.Hkv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (seq_lens) {
        if (n_rank) b = longest_first<64>(seq_lens, n_rank, b, reinterpret_cast<int *>(red));
        // per-sequence token counts held on the device (ragged batches; also lets a captured launch be
        // replayed while the sequences grow).  The host could not check the capacity, so it is checked here.
        const int T = seq_lens[b];
        if (T < 0 || T / Codec<BITS>::TPW >= ka.n_super_cap) {
            if (threadIdx.x == 0) atomicExch(&g_status, kStatCapacity);
            return;
        }
        ka.T = T;
        va.T = T;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; ++i) { mbar_init(&kbar[i], 1); mbar_init(&vbar[i], 1); }
        fs.init_barriers(1);
        mbar_init_fence();
    }
    __syncthreads();
    const Seg seg{0, ka.T, true, nullptr, nullptr, 0};
    if (warp == 0) {
        RingSink<G, 1, TOK> sink{&fs, 0, 0};
        k_warp<BITS, G, ARITH, RingSink<G, 1, TOK>, ST, false, kOutOfLineGuarded<BITS, G>, 8, TOK>(ka, seg, b, h, lane, kbuf, kbar,
                                                                                                   red, sink);
    } else {
        SoftmaxSrc<G, 1, false, TOK> src;
        src.sh = &fs;
        src.wts = wts;
        src.mask = mask ? mask + size_t(b) * mask_stride_b : nullptr;
        src.scale2 = scaling * 1.4426950408889634f;
        src.n_tiles = (va.T + TOK - 1) / TOK;
        src.t_begin = 0;
        src.init();
        v_warp<BITS, G, ARITH, SoftmaxSrc<G, 1, false, TOK>, ST, false, kOutOfLineGuarded<BITS, G>, TOK>(va, seg, b, h, lane, vbuf,
                                                                                                         vbar, wts, src);
    }
}

}  // namespace adkv

using namespace adkv;

// adkv_decode_attn splits the channels of a head over two warp pairs up to one (batch, kv head) stream per SM, and up to 160
// streams while the set-up counts: a short stream is loaded and appended by more warps, a long one pays the sums, votes and
// rings of twice as many.  Device time on a B200, split / whole head, us (in brackets: one channel of every head at a bound):
//    148 streams, canonical replay    4-bit 100 tokens 10.1 / 11.5, 256 17.0 / 18.6, 2000 100 / 103 (183 / 131); with four heads 142 /
//                                     152 (196 / 159); 2-bit 100 tokens 9.2 / 11.3, 256 20.7 / 18.5, 2000 129 / 108 (179 / 114)
//    148 streams next to tails        4-bit 60 tokens 7.7 / 9.5, 100 9.9 / 10.5; 2-bit, four heads, 100 11.2 / 14.5; longer ones: segments
//    160 streams next to tails        4-bit 100 tokens 10.4 / 10.5, 256 18.2 / 16.6, 2000 110 / 89; 2-bit, four heads, 100 12.9 / 13.8, 256
//                                     24.1 / 24.4, 2000 160 / 140
// Without segments, long 2-bit streams of one head and streams with scales at a bound would be better off whole below 148, too.
constexpr int kSplitChannelsMaxTokens = 256;
constexpr long long kSplitChannelsMaxStreams = 160;

ADKV_HIDDEN int adkv_half_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b,
                                      float scaling, int B, int bits, const int *seq_lens, cudaStream_t s);
ADKV_HIDDEN int adkv_narrow_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b,
                                        float scaling, int B, int bits, bool exact, cudaStream_t s);
ADKV_HIDDEN int adkv_segments_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b,
                                          float scaling, int B, int max_tokens, int bits, const int *seq_lens, cudaStream_t s);
ADKV_HIDDEN int adkv_wide_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b,
                                      float scaling, int B, int bits, int mode, cudaStream_t s);

ADKV_HIDDEN int adkv_tensor_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling,
                                        int B, int bits, const int *seq_lens, int n_rank, const CkptArgs &ck, int n_seg,
                                        float *scratch, cudaStream_t s);

ADKV_DEFINE_TU_STATUS(adkv_tu_status_fused)

// Token segments of a stream side by side (adkv_segments.cu), next to tail states: up to one stream per SM and from 128
// tokens on (max_tokens: the tokens of every sequence, or what the cache can hold of them where the lengths are on the
// device).  The tensor-core kernel goes first, so what comes here is 2-bit caches with one query head and more than kSegmentsAhead
// tokens, and scale bounds that kernel cannot take (tensor_can).  Device time on a B200, segments / tensor cores, 2-bit, one head, 128
// to 148 streams: x 500 tokens 18.9 / 18.2 us, x 700 24.7 / 22.5 us, x 1000 30.0 / 30.7 us, x 12000 256 / 272 us.
// Split head of adkv_narrow.cu / whole head / segments, where no scale meets a clamp and, in brackets, where one channel of every
// head rests at a bound:
//    4-bit                 128 streams x 256 tokens 16.4 / 16.7 / 12.4 us, x 2000 93 / 89 / 49 us (179 / 109 / 80 us)
//    2-bit, four heads     128 streams x 256 tokens 22.0 / 24.4 / 16.0 us, x 2000 141 / 140 / 73 us (185 / 146 / 102 us)
// Measured with tiles of 32 tokens everywhere, split head -> segments: 32 streams x 8000 tokens, 4-bit, 376 -> 176 us (728 -> 322 us);
// 144 x 128, 2-bit, two heads, 12.0 -> 12.0 us (14.8 -> 14.0 us).
// Below 128 tokens set-up and merge are not made up for (2-bit, 128 streams x 96 tokens: 8.4 -> 8.9 us); device-side
// lengths may lie there, and cost a microsecond up to 64 tokens (64 streams x 64 tokens: 8.6 -> 9.3 us, x 96 tokens: 10.0
// -> 9.4 us, x 256 tokens: 17.2 -> 12.3 us).  With more than one stream per SM the extra work has no idle schedulers to go
// to: 256 streams x 8000 tokens with four segments each, 2-bit, 442 -> 378 us / 478 -> 655 us, with eight KV heads 595 ->
// 522 us / 646 -> 788 us.
constexpr long long kSegmentsMaxStreams = kSMs;
constexpr int kSegmentsMinTokens = 128, kSegmentsAhead = 700;

static bool use_segments(const KArgs &ka, int B, int max_tokens, bool exact, unsigned flags)
{
    return ka.tail && !exact && !(flags & (ADKV_FLAG_SPLIT_CHANNELS | ADKV_FLAG_NO_SPLIT_CHANNELS)) &&
           ka.Hq / ka.Hkv <= 4 && (long long)B * ka.Hkv <= kSegmentsMaxStreams && max_tokens >= kSegmentsMinTokens;
}

static bool use_tensor(const KArgs &ka, int B, int bits, int max_tokens, bool device_lengths, bool exact, unsigned flags)
{
    const int G = ka.Hq / ka.Hkv;
    if (bits == 2 && G == 1 && max_tokens > kSegmentsAhead && use_segments(ka, B, max_tokens, exact, flags)) return false;
    return ka.tail && !exact && !(flags & (ADKV_FLAG_SPLIT_CHANNELS | ADKV_FLAG_NO_SPLIT_CHANNELS)) && tensor_can(G, ka.smin, ka.smax) &&
           tensor_pays(bits, G, (long long)B * ka.Hkv, max_tokens, device_lengths);
}

// Whether a launch of whole heads takes tiles of 32 tokens (three stages) instead of 64 (two).  V starts when K is through its
// first tile, so a stream of one or a few tiles is walked by one warp after the other; with few CTAs on an SM nothing fills that
// gap.  With eight query heads 64 tokens also take 38 KB of shared memory (4-bit), so that fewer CTAs fit an SM than its
// registers allow; long streams make up for it.  Device time on a B200, next to tails, 64 -> 32 tokens:
//    up to 64 tokens      256 streams, 2-bit, four heads 12.1 -> 10.7 us; 600 streams, 4-bit 12.4 -> 11.4 us; but 4096 streams, 4-bit,
//                         four heads 60 -> 62 us
//    up to 255 tokens     600 streams x 150, 4-bit 20.7 -> 19.9 us, 2-bit, four heads 31.9 -> 29.6 us; 256 x 200, 2-bit, two heads,
//                         canonical replay 20.0 -> 19.3 us; but 256 x 200, 4-bit, two heads 17.0 -> 17.6 us; 600 x 150, 4-bit, four heads
//                         31.2 -> 32.1 us; 4096 x 200, 2-bit, four heads 141 -> 151 us
//    eight heads          4-bit, 4096 x 150 287 -> 246 us, 4096 x 1000 964 -> 916 us, 600 x 300 72.0 -> 68.6 us, but 1200 x 1000 342 ->
//                         354 us, 150 x 1000 100 -> 103 us;
//                         2-bit, 600 x 200 55.9 -> 51.9 us, 4096 x 150 167 -> 158 us, but 4096 x 300 486 -> 505 us
// Up to one stream per SM only calls with device-side lengths or split_channels = False come here; they keep 64.
// T: the tokens of every sequence, or what the cache can hold of them where the lengths are on the device.
static bool short_tiles(int bits, int G, long long streams, int T)
{
    const bool many = streams > 8 * kSMs;
    if (G == 8) return T < (bits == 4 ? (streams > 16 * kSMs ? 1024 : 512) : (many ? 192 : 256));
    if (many || streams <= kSMs || (bits == 4 && G == 4)) return false;
    if (T <= 64) return true;
    return T < 256 && (bits == 4 ? streams > 2 * kSMs : G > 1);
}

// One CTA per stream.
static int launch_decode(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling, int B,
                         int max_tokens, int bits, bool exact, const int *seq_lens, cudaStream_t s)
{
    const int n_rank = seq_lens && B <= kRankMax && ka.n_super_cap >= kRankMinTokens * bits / 32 ? B : 0;
    if (short_tiles(bits, ka.Hq / ka.Hkv, (long long)B * ka.Hkv, max_tokens)) {
        ADKV_DISPATCH(bits, exact, ka.Hq / ka.Hkv,
                      (decode_attn_kernel<BITS, G, ARITH, 32><<<B * ka.Hkv, 64, 0, s>>>(ka, va, mask, mask_stride_b, scaling,
                                                                                       seq_lens, n_rank)))
        return launch_status();
    }
    ADKV_DISPATCH(bits, exact, ka.Hq / ka.Hkv,
                  (decode_attn_kernel<BITS, G, ARITH, 64><<<B * ka.Hkv, 64, 0, s>>>(ka, va, mask, mask_stride_b, scaling,
                                                                                   seq_lens, n_rank)))
    return launch_status();
}

extern "C" {

int adkv_decode_attn(const void *q, void *k_cache, void *v_cache, const void *k_new, const void *v_new,
                     const adkv_params *kp, const adkv_params *vp, void *k_tail, void *v_tail, const void *mask,
                     long long mask_stride_b,
                     void *out, int B, int Hq, int Hkv, int T, int D, int n_super_cap, int bits, float scaling,
                     float scale_min, float scale_max, unsigned flags, void *stream)
{
    if (!q || !k_cache || !v_cache || !k_new || !v_new || !out || !params_ok(kp) || !params_ok(vp))
        return ADKV_E_NULL;
    if (int rc = check_common(B, Hq, Hkv, T, D, n_super_cap, bits, T + 1)) return rc;
    if (int rc = check_tails(k_tail, v_tail, flags)) return rc;
    if (!aligned16(k_cache) || !aligned16(v_cache) || !aligned8(q) || !aligned8(out) || !aligned8(k_new) ||
        !aligned8(v_new) || !params_aligned(kp) || !params_aligned(vp))
        return ADKV_E_ALIGN;
    if (B == 0) return 0;
    const bool keep = flags & ADKV_FLAG_TAIL_KEEP;
    const KArgs ka{static_cast<const __half *>(q), static_cast<uint8_t *>(k_cache),
                   static_cast<const __half *>(k_new), to_ptrs(kp), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D,
                   static_cast<float *>(k_tail), keep};
    const VArgs va{static_cast<uint8_t *>(v_cache), static_cast<const __half *>(v_new), static_cast<__half *>(out),
                   to_ptrs(vp), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D, static_cast<float *>(v_tail), keep};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool half = flags & ADKV_FLAG_HALF_STATE, exact = !(flags & ADKV_FLAG_FAST_REPLAY);
    if (D != kD)
        return adkv_wide_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, bits,
                                     half ? 2 : int(exact), s);
    if (half)
        return adkv_half_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, bits, nullptr, s);
    if (use_tensor(ka, B, bits, T, false, exact, flags))
        return adkv_tensor_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, bits, nullptr, 0, CkptArgs{}, 1, nullptr, s);
    if (use_segments(ka, B, T, exact, flags))
        return adkv_segments_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, T, bits, nullptr, s);
    // Very few streams: split every head over two warp pairs (adkv_narrow.cu).
    const bool split = (flags & ADKV_FLAG_SPLIT_CHANNELS) ||
                       (!(flags & ADKV_FLAG_NO_SPLIT_CHANNELS) &&
                        ((long long)B * Hkv <= kSMs || ((long long)B * Hkv <= kSplitChannelsMaxStreams && T < kSplitChannelsMaxTokens)));
    if (split)
        return adkv_narrow_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, bits, exact, s);
    return launch_decode(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, T, bits, exact, nullptr, s);
}

int adkv_decode_attn_varlen(const void *q, void *k_cache, void *v_cache, const void *k_new, const void *v_new,
                            const adkv_params *kp, const adkv_params *vp, void *k_tail, void *v_tail,
                            const void *seq_lens, void *out, int B, int Hq, int Hkv, int D, int n_super_cap, int bits,
                            float scaling, float scale_min, float scale_max, unsigned flags, void *stream)
{
    if (!q || !k_cache || !v_cache || !k_new || !v_new || !out || !seq_lens || !params_ok(kp) || !params_ok(vp))
        return ADKV_E_NULL;
    if (D != kD) return ADKV_E_HEAD_DIM;   // device-side lengths: 128-wide heads only
    if (int rc = check_common(B, Hq, Hkv, 0, D, n_super_cap, bits, 1)) return rc;
    if (int rc = check_tails(k_tail, v_tail, flags)) return rc;
    if (!aligned16(k_cache) || !aligned16(v_cache) || !aligned8(q) || !aligned8(out) || !aligned8(k_new) ||
        !aligned8(v_new) || !params_aligned(kp) || !params_aligned(vp) || (reinterpret_cast<uintptr_t>(seq_lens) & 3u))
        return ADKV_E_ALIGN;
    if (B == 0) return 0;
    const bool keep = flags & ADKV_FLAG_TAIL_KEEP;
    const KArgs ka{static_cast<const __half *>(q), static_cast<uint8_t *>(k_cache),
                   static_cast<const __half *>(k_new), to_ptrs(kp), Hq, Hkv, 0, n_super_cap, scale_min, scale_max, D,
                   static_cast<float *>(k_tail), keep};
    const VArgs va{static_cast<uint8_t *>(v_cache), static_cast<const __half *>(v_new), static_cast<__half *>(out),
                   to_ptrs(vp), Hq, Hkv, 0, n_super_cap, scale_min, scale_max, D, static_cast<float *>(v_tail), keep};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (flags & ADKV_FLAG_HALF_STATE)
        return adkv_half_decode_attn(ka, va, nullptr, 0, scaling, B, bits, static_cast<const int *>(seq_lens), s);
    const bool exact = !(flags & ADKV_FLAG_FAST_REPLAY);
    const int room = min(n_super_cap, 1 << 20) * (32 / bits) - 1;
    if (use_tensor(ka, B, bits, room, true, exact, flags))
        return adkv_tensor_decode_attn(ka, va, nullptr, 0, scaling, B, bits, static_cast<const int *>(seq_lens),
                                       B <= kRankMax && n_super_cap >= kRankMinTokens * bits / 32 ? B : 0, CkptArgs{}, 1, nullptr, s);
    if (use_segments(ka, B, room, exact, flags))
        return adkv_segments_decode_attn(ka, va, nullptr, 0, scaling, B, room, bits, static_cast<const int *>(seq_lens), s);
    return launch_decode(ka, va, nullptr, 0, scaling, B, room, bits, exact, static_cast<const int *>(seq_lens), s);
}

}  // extern "C"
