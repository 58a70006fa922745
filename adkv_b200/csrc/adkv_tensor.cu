// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point.
//
// Fused decode step next to tail states with the sums over channels (K) and over tokens (V) on the tensor cores, one CTA per (batch,
// KV head) stream or checkpoint segment.  Reached through adkv_decode_attn, adkv_decode_attn_varlen and adkv_decode_attn_ckpt.
//
// In the scans of adkv_decode.cuh a token costs, besides the recurrence, a multiply-add per channel and query head for K and for V, the
// zero points, and sums over the lanes; and a stream is two warps that wait for their own results.  Here a thread owns ONE channel,
// 128 threads scan K and 128 scan V, and all that they form is code times scale, x = q * s, written as a sum of two fp16 numbers
// (22 bits).  The rest are products of matrices, 64 tokens at a time, with fp32 accumulators in tensor memory:
//
//  K   [tokens x channels] x [channels x (q, alpha * q)]: a logit is sum_c q_c x_c plus what the zero points add, and the zero points'
//      share advances by sum_c alpha_c q_c x_c a token, so one running sum per head takes the place of 128 zero points.  q is an
//      fp16 number already; alpha * q takes two.  The rounded parts and the remainders of x are the two halves of one M = 128 product.
//  V   [channels x tokens] x [tokens x (p, P)] for the weights p and the sums P of the weights behind each token in its tile: with zp
//      the zero point at the start of a tile its share of the result is  zp * sum(p) + sum_t (p_t + alpha * P_t) x_t, and a column of
//      ones advances zp.  x lies in tensor memory, p and P are pairs of fp16 numbers again.
//
// So a value costs the scanning threads about nine instructions whatever the number of query heads, and one stream keeps eight warps
// busy instead of two.  Four more warps move the sums of K out of tensor memory, form the weights (online softmax, warp e for head
// e) and add the sums of V to the result; two issue the products and the copies of packed words.  All meet at mbarriers, two tiles
// in flight.  What bounds it: issue and register reads of the scans, 10 cycles a value and scheduler with four warps, 13 with two
// (measured alone; a third of it the split into fp16 parts), so with one query head and many streams the packed scans of
// adkv_decode.cuh stay ahead (12 cycles with everything); with one CTA on an SM the warps that move the sums, weigh and add, one after
// the other, 2600 cycles a tile.  The lines are in tensor_pays (adkv_host.h).  Against 64 bits the error of a logit is 0.85 to 0.98
// times that of one scan with fp32 sums (eight sets of 2000 tokens pooled, 192 logits each, for either code width and every number of
// query heads; three sets of 16000: 0.88 to 0.97; single sets 0.7 to 1.25), with one channel of a head at a bound 0.85 to 1.00, with every
// scale of a 4-bit cache at the lower bound 1.01 to 1.02.  A whole result, before it is rounded to fp16: 0.8 to 1.2, 0.90 where
// the weights are flat.  Carrying what the scale loses in guarded windows, too, would leave 0.87 at the lower bound and cost
// 5 to 10 % of such steps and up to 4 % of all.
//
// Only the appended token needs the encoder's exact state, and that comes from the tail.
#include "adkv_host.h"

#include "adkv_softmax.cuh"
#include "adkv_tensor.cuh"

namespace adkv {

constexpr int kTcTok = 64;         // tokens per tile
constexpr int kTcWarps = 14;       // 0-3: K, 4-7: V (a channel a thread), 8-11: softmax and results, 12: K products, 13: V products
constexpr int kTcThreads = 32 * kTcWarps;
constexpr float kTcP = 4096.f, kTcS = 256.f;   // weights and their suffix sums are scaled by these before they become fp16 pairs

template <int BITS, int G>
struct TensorShared {
    static constexpr int KN = (3 * G + 15) / 16 * 16;      // K product, columns per head: q, alpha * q (rounded), its remainder
    static constexpr int VN = (4 * G + 1 + 15) / 16 * 16;  // V product, columns per head: p, suffix sum, their remainders; then ones
    // groups of eight columns that are stored; a product of more columns than that reads the first group again, or what lies behind
    static constexpr int KG = (3 * G + 7) / 8, VG = (4 * G + 1 + 7) / 8;
    static constexpr int ST = 3;                           // tiles of packed words in flight per tensor
    static constexpr int NB = 2;                           // buffers: the products read one tile while the next is scanned
    alignas(128) __half a[NB][2][kTcTok / 8][kD][8];       // K values of a tile, rounded and remainder: [buffer][part][token / 8][channel][token % 8]
    alignas(128) uint32_t words[2][ST][kTcTok * BITS / 32][kD];   // packed tiles of K and V
    alignas(128) __half kb[KG][kD][8];                 // [column / 8][channel][column % 8]
    alignas(128) __half vb[NB][VG][kTcTok][8];         // [buffer][column / 8][token][column % 8]
    alignas(16) float lbuf[NB][2][G][2][kTcTok];            // K: sums over the channels of a tile: [buffer][part][head][with q, with alpha * q]
    float2 fac[4][G];                                      // of a tile: factor of the sums so far, sum of the weights
    alignas(16) float self_x[kD];                          // dequantised appended V
    float back[G][2];                                      // undo the scaling of the columns of kb
    float self_logit[G], m[G], l[G];
    float z0[4][G];                                        // sum of q * zp at the start, per K warp
    uint32_t top[4][2 * G];                                // largest |q|, |alpha * q| per K warp (bit patterns)
    uint32_t tmem;
    int dead;                                              // a bounded wait gave up
    // barriers of tile i, slot i % NB (loaded: i % ST): words are there; K values are there, K sums are there, and
    // have been read; sums are in lbuf, and have been read; V values, weights, V sums are there, V sums have been read
    uint64_t loaded[2][ST], kfull[NB], kdone[NB], kread, lfull[NB], lread[NB], vfull[NB], wfull[NB], vdone[NB], vread[NB];
};

// two fp16 numbers
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// the halves of h minus a and b, as fp16: the remainders with the sign turned (the products of this part subtract)
__device__ __forceinline__ uint32_t pack_remainder(uint32_t h, float a, float b)
{
    float d0, d1;
    asm("{.reg .b16 x, y;\n\tmov.b32 {x, y}, %1;\n\tsub.rn.f32.f16 %0, x, %2;\n\t}" : "=f"(d0) : "r"(h), "f"(a));
    asm("{.reg .b16 x, y;\n\tmov.b32 {x, y}, %1;\n\tsub.rn.f32.f16 %0, y, %2;\n\t}" : "=f"(d1) : "r"(h), "f"(b));
    return pack_half2(d0, d1);
}

// What one thread keeps of its channel.  The scale is held in units of a power of two below the upper bound, so that the fp16 parts
// of the dequantised values have their bits where they are needed; scaling by it rounds nothing.
struct TensorChan {
    float s, beta, tc, lo, hi;   // scale, constants of its update, interval in which eight updates cannot meet a bound
    float inv;                   // one over the unit
    float lost = 0.f;            // what the last rounding of the scale took away
    __device__ __forceinline__ bool safe() const { return __all_sync(kFull, s >= lo && s <= hi); }
};
struct Window {
    float x[8], s;
};
template <int BITS>
__device__ __noinline__ Window guarded_window(uint32_t w, float s, float beta, float tc, float smin, float smax, float eps)
{
    Window r;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float q = code_f_rt<BITS>(w, j);
        r.x[j] = __fmul_rn(q, fmaxf(s, eps));
        s = fminf(fmaxf(s * fmaf(beta, fabsf(q), tc), smin), smax);
    }
    r.s = s;
    return r;
}
// Code times scale of eight tokens (fields 0..7 of w); advances the scale, without guards.  What every fourth product of the scale
// loses in rounding goes into the next: two multiply-adds more in eight tokens than without, and logits end 6 to 12 % nearer to 64
// bits than with every eighth, 256 streams x 8192 tokens 334 -> 337 us.
template <int BITS>
__device__ __forceinline__ void scale_window(uint32_t w, const FieldConsts<BITS> &fc, TensorChan &c, float (&x)[8])
{
    static_for<8>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        const float q = fc.template code<j % 4>(j < 4 ? w : w >> (4 * BITS));
        x[j] = __fmul_rn(q, c.s);
        const float f = fmaf(c.beta, fabsf(q), c.tc), s = c.s;
        c.s = j % 4 == 0 ? fmaf(s, f, c.lost * f) : s * f;
        if (j % 4 == 3) c.lost = fmaf(s, f, -c.s);
    });
}
// The same with them, by a call.
template <int BITS>
__device__ __forceinline__ void scale_window_guarded(uint32_t w, TensorChan &c, float smin, float smax, float (&x)[8])
{
    const Window r = guarded_window<BITS>(w, c.s, c.beta, c.tc, smin * c.inv, smax * c.inv, kEps * c.inv);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = r.x[j];
    c.s = r.s;
    c.lost = 0.f;
}
// Sixteen tokens.  safe: no channel of the warp can meet a bound in the next eight.  The second eight run on that they cannot
// either, and are done again where the scale between the two says otherwise: one vote for sixteen tokens instead of two, each of
// which costs a warp with one other on its scheduler 22 cycles.
template <int BITS>
__device__ __forceinline__ void scale_windows(uint32_t wa, uint32_t wb, const FieldConsts<BITS> &fc, TensorChan &c, float smin, float smax,
                                              float (&xa)[8], float (&xb)[8], bool &safe)
{
    if (safe) {
        scale_window<BITS>(wa, fc, c, xa);
        const float between = c.s;
        scale_window<BITS>(wb, fc, c, xb);
        const bool held = between >= c.lo && between <= c.hi;
        safe = __all_sync(kFull, held && c.s >= c.lo && c.s <= c.hi);
        if (!safe) {
            if (!__all_sync(kFull, held)) {
                c.s = between;
                scale_window_guarded<BITS>(wb, c, smin, smax, xb);
            }
            safe = c.safe();
        }
    } else {
        scale_window_guarded<BITS>(wa, c, smin, smax, xa);
        scale_window_guarded<BITS>(wb, c, smin, smax, xb);
        safe = c.safe();
    }
}

// The code of the first token of a channel.
template <int BITS>
__device__ __noinline__ float first_code(const uint8_t *cache, size_t at)
{
    return code_f_rt<BITS>(reinterpret_cast<const uint32_t *>(cache)[at], 0);
}

__device__ __forceinline__ float redux_max(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float pow2_bits(int exponent_field) { return __uint_as_float(uint32_t(exponent_field) << 23); }
__device__ __forceinline__ int exponent_field(float v) { return int(__float_as_uint(v) >> 23 & 0xff); }
__device__ __forceinline__ void arrive_warp(uint64_t *bar, int lane)
{
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

template <int BITS, int G, bool PART>
__global__ void __launch_bounds__(kTcThreads, 2)
    decode_attn_tensor_kernel(KArgs ka, VArgs va, const float *__restrict__ mask, long long mask_stride_b, float scaling,
                              const int *__restrict__ seq_lens, int n_rank, CkptArgs ck, float *__restrict__ scratch)
{
    extern __shared__ __align__(128) uint8_t smem_raw[];
    using Shared = TensorShared<BITS, G>;
    Shared &sh = *reinterpret_cast<Shared *>(smem_raw);
    constexpr int kSums = G == 4 ? 2 : 4;    // see the products of K
    constexpr int TPW = Codec<BITS>::TPW, KN = Shared::KN, VN = Shared::VN, KG = Shared::KG, VG = Shared::VG, NB = Shared::NB, ST = Shared::ST;
    constexpr int ROWS = kTcTok / TPW;       // word rows of a tile
    // columns of tensor memory: V values (rounded, then remainders) and sums of V, NB buffers each; sums of K
    constexpr uint32_t kVPart = kTcTok / 2, kVBuf = kTcTok, kDV = NB * kTcTok, kDK = kDV + NB * VN, kColumns = 256;
    static_assert(KN <= 16 && VN <= 32 && kDK + kSums * KN <= kColumns, "columns of tensor memory");

    int b = blockIdx.x / ka.Hkv;
    const int h = blockIdx.x % ka.Hkv;
    const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // uniform: products want uniform registers
    if (seq_lens) {   // as in decode_attn_kernel
        if (n_rank) b = longest_first<kTcThreads>(seq_lens, n_rank, b, reinterpret_cast<int *>(&sh.lbuf[0][0][0][0][0]));
        const int T = seq_lens[b];
        if (T < 0 || T / TPW >= ka.n_super_cap) {
            if (threadIdx.x == 0) atomicExch(&g_status, kStatCapacity);
            return;
        }
        ka.T = T;
        va.T = T;
    }
    const int bh = b * ka.Hkv + h, T = ka.T;
    const int seg = PART ? blockIdx.y : 0, n_seg = PART ? gridDim.y : 1;
    const int t_begin = PART ? seg * ck.interval : 0, t_end = PART ? min(T, t_begin + ck.interval) : T;
    const bool mute_k = PART && ck.mute_k;   // self-test: K is not scanned, and every wait behind that runs out
    const bool append = seg == n_seg - 1 && !mute_k;
    const int ntok = t_end - t_begin, n_tiles = (ntok + kTcTok - 1) / kTcTok;
    const int n_rows = (ntok + TPW - 1) / TPW;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) {
            mbar_init(&sh.kfull[i], 4);
            mbar_init(&sh.kdone[i], 2);
            mbar_init(&sh.vfull[i], 4);
            mbar_init(&sh.wfull[i], G);
            mbar_init(&sh.vdone[i], 2);
            mbar_init(&sh.vread[i], 4);
            mbar_init(&sh.lfull[i], 4);
            mbar_init(&sh.lread[i], G);
        }
        for (int i = 0; i < 2; ++i) {
            for (int k = 0; k < ST; ++k) mbar_init(&sh.loaded[i][k], 1);
        }
        mbar_init(&sh.kread, 4);
        sh.dead = 0;
        mbar_init_fence();
    }
    if (warp == 12) tmem_alloc(&sh.tmem, kColumns);

    // the channel of a K, V or result thread
    const bool is_k = warp < 4;
    const int c = threadIdx.x & (kD - 1);
    TensorChan ch;
    FieldConsts<BITS> fc;
    float zp, alpha, unit;
    if (warp < 12) {
        if (warp < 8) fc.init();
        const ParamPtrs &p = is_k ? ka.p : va.p;
        const size_t po = size_t(h) * kD + c;
        alpha = __half2float(p.alpha[po]);
        const float beta = __half2float(p.beta[po]), target = __half2float(p.target[po]);
        float s;
        if (PART && seg > 0) {
            const float *init = (is_k ? ck.k_ckpt : ck.v_ckpt) + (size_t(bh) * ck.n_ckpt_cap + seg - 1) * 2 * kD;
            zp = init[c];
            s = init[kD + c];
        } else {
            zp = __half2float(p.zp_init[po]);
            s = __half2float(p.scale_init[po]);
        }
        // The unit goes by the upper bound: eight times that stays in the range of fp16, and a lower bound no further away than
        // tensor_can allows leaves every value its 22 bits, wherever the scale moves.  Only scale_init may lie above the bound, and
        // counts where its code is not zero (the values of this channel then start that large, too).  One branch for the warp and a
        // call: a branch for each thread, or the word read in any case, costs long streams 1 % and a step of 300 tokens 0.25 us.
        int e = max(exponent_field(s), exponent_field(ka.smax)) - 11;
        if ((!PART || seg == 0) && __any_sync(kFull, e > exponent_field(ka.smax) - 11)) {
            if (first_code<BITS>(is_k ? ka.cache : va.cache, size_t(bh) * ka.n_super_cap * kD + c) == 0.f) e = exponent_field(ka.smax) - 11;
        }
        e = min(max(e, 127 - 40), 127 + 40);
        const float inv = pow2_bits(254 - e);
        unit = pow2_bits(e);
        ch.s = s * inv;
        ch.beta = beta;
        ch.tc = fmaf(-beta, target, 1.0f);
        ch.inv = inv;
        SafeRange safe{0.f, INFINITY};
        const float be[1] = {beta}, tg[1] = {target};
        safe.template init<BITS, 1>(be, tg, fmaxf(ka.smin, kEps) * inv, ka.smax * inv);
        ch.lo = safe.lo;
        ch.hi = safe.hi;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    const float scale2 = scaling * 1.4426950408889634f;
    const float *mask_row = mask ? mask + size_t(b) * mask_stride_b : nullptr;
    bool ok = true;

    // packed tiles of tensor `which` (0: K, 1: V), by one lane
    const auto load_tile = [&](int which, int i) {
        const uint32_t bytes = min(ROWS, n_rows - i * ROWS) * kD * 4;
        uint64_t *bar = &sh.loaded[which][i % ST];
        mbar_expect_tx(bar, bytes);
        bulk_load(&sh.words[which][i % ST][0][0],
                  (which ? va.cache : ka.cache) + (size_t(bh) * ka.n_super_cap + t_begin / TPW + size_t(i) * ROWS) * kD * 4, bytes, bar);
    };
    // the new token, quantised from its tail; xh: this lane's four channels, dequantised
    const auto append_token = [&](bool v, float (&xh)[4]) {
        const int n = bh;
        float *tail = v ? va.tail : ka.tail, *ckpt = v ? ck.v_ckpt : ck.k_ckpt;
        append_from_tail<BITS>(v ? va.p : ka.p, size_t(h) * kD + 4 * lane, tail + size_t(n) * 2 * kD, ka.tail_keep,
                               (v ? va.x_new : ka.x_new) + size_t(n) * kD + 4 * lane,
                               reinterpret_cast<uint4 *>((v ? va.cache : ka.cache) + (size_t(n) * ka.n_super_cap + T / TPW) * kD * 4) + lane, T,
                               ka.smin, ka.smax,
                               PART && (T + 1) % ck.interval == 0 ? ckpt + (size_t(n) * ck.n_ckpt_cap + (T + 1) / ck.interval - 1) * 2 * kD : nullptr,
                               4 * lane, xh);
    };

    if (warp < 8) {
        // ------------------------------------------------------------------------------ K and V
        // One loop for both: two that run at the same time would take turns in the instruction cache of a scheduler.
        if (is_k) {
            float q[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                q[g] = __half2float(ka.q[(size_t(b) * ka.Hq + size_t(h) * G + g) * kD + c]);
                const float z = warp_sum(q[g] * zp);
                const uint32_t ta = __reduce_max_sync(kFull, __float_as_uint(fabsf(q[g] * unit)));
                const uint32_t tb = __reduce_max_sync(kFull, __float_as_uint(fabsf(alpha * q[g] * unit)));
                if (lane == 0) {
                    sh.z0[warp][g] = z;
                    sh.top[warp][2 * g] = ta;
                    sh.top[warp][2 * g + 1] = tb;
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            __half col[8 * KG];
#pragma unroll
            for (int i = 0; i < 8 * KG; ++i) col[i] = __float2half_rn(0.f);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float up[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t top = max(max(sh.top[0][2 * g + i], sh.top[1][2 * g + i]), max(sh.top[2][2 * g + i], sh.top[3][2 * g + i]));
                    const int e = max(int(top >> 23), 15);
                    up[i] = pow2_bits(268 - e);
                    if (c == 0) sh.back[g][i] = pow2_bits(e - 14);
                }
                const float qa = alpha * q[g] * unit * up[1];
                col[3 * g] = __float2half_rn(q[g] * unit * up[0]);
                col[3 * g + 1] = __float2half_rn(qa);
                col[3 * g + 2] = __float2half_rn(qa - __half2float(col[3 * g + 1]));
            }
#pragma unroll
            for (int i = 0; i < KG; ++i) *reinterpret_cast<uint4 *>(&sh.kb[i][c][0]) = *reinterpret_cast<const uint4 *>(&col[8 * i]);
        }
        const int which = warp >> 2;
        uint64_t *loaded = sh.loaded[which], *freed = is_k ? sh.kdone : sh.vdone, *full = is_k ? sh.kfull : sh.vfull;
        const uint32_t lanes = tmem + (uint32_t(32 * (warp & 3)) << 16);
        bool safe = ch.safe();
        if (mute_k && is_k) ok = false;
#pragma unroll 1
        for (int i = mute_k && is_k ? n_tiles : 0; i < n_tiles; ++i) {
            const int buf = i % NB, st = i % ST;
            const int rounds = (min(ROWS, n_rows - i * ROWS) + 16 / TPW - 1) / (16 / TPW);   // of 16 tokens, as the products of V take
            // the words have come, and the products that read this buffer before are done
            if (!(ok = mbar_wait_both(&loaded[st], i / ST & 1, i >= NB ? &freed[buf] : nullptr, (i / NB & 1) ^ 1, kStatKWait))) break;
            tc_fence_after();
            const uint32_t *row = &sh.words[which][st][0][c];
            uint8_t *k_dst = reinterpret_cast<uint8_t *>(&sh.a[buf][0][0][c][0]);
            uint32_t v_dst = lanes + kVBuf * buf, wa = row[0], wb = BITS == 4 ? row[kD] : wa >> 16;
            const auto store = [&](const float (&x)[8]) {
                uint4 hi, lo;
                hi.x = pack_half2(x[0], x[1]); lo.x = pack_remainder(hi.x, x[0], x[1]);
                hi.y = pack_half2(x[2], x[3]); lo.y = pack_remainder(hi.y, x[2], x[3]);
                hi.z = pack_half2(x[4], x[5]); lo.z = pack_remainder(hi.z, x[4], x[5]);
                hi.w = pack_half2(x[6], x[7]); lo.w = pack_remainder(hi.w, x[6], x[7]);
                if (is_k) {
                    *reinterpret_cast<uint4 *>(k_dst) = hi;
                    *reinterpret_cast<uint4 *>(k_dst + sizeof(sh.a[0][0])) = lo;
                } else {
                    tmem_st4(v_dst, hi.x, hi.y, hi.z, hi.w);
                    tmem_st4(v_dst + kVPart, lo.x, lo.y, lo.z, lo.w);
                }
                k_dst += kD * 16;
                v_dst += 4;
            };
#pragma unroll 1
            for (int n = 0; n < rounds; ++n) {
                row += 16 / TPW * kD;
                const uint32_t next_a = row[0], next_b = BITS == 4 ? row[kD] : next_a >> 16;   // behind a tile: whatever lies there, not used
                float xa[8], xb[8];
                scale_windows<BITS>(wa, wb, fc, ch, ka.smin, ka.smax, xa, xb, safe);
                store(xa);
                store(xb);
                wa = next_a;
                wb = next_b;
            }
            if (is_k) {
                fence_async_shared();
            } else {
                tmem_wait_st();
                tc_fence_before();
            }
            arrive_warp(&full[buf], lane);
        }
        // every thread of this tensor has read the word that the new code goes into
        if (is_k) asm volatile("bar.sync 1, 128;" ::: "memory");
        else asm volatile("bar.sync 2, 128;" ::: "memory");
        if (ok && append && (warp & 3) == 0) {
            float xh[4];
            append_token(!is_k, xh);
            if (is_k) {
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    float qv[4], x = 0.f;
                    load_half4(qv, ka.q + (size_t(b) * ka.Hq + size_t(h) * G + g) * kD + 4 * lane);
#pragma unroll
                    for (int n = 0; n < 4; ++n) x = fmaf(qv[n], xh[n], x);
                    x = warp_sum(x);
                    if (lane == 0) sh.self_logit[g] = x;
                }
            } else {
                *reinterpret_cast<float4 *>(&sh.self_x[4 * lane]) = make_float4(xh[0], xh[1], xh[2], xh[3]);
            }
        }
        if (!ok && lane == 0) sh.dead = 1;
        __syncthreads();
    } else if (warp < 12) {
        // ------------------------------------------------------------------------------ softmax and results
        // All four warps move the K sums of a tile to shared memory and add its V sums to the result; the weights of head e are
        // formed by warp e.
        const int e = warp & 3;
        const uint32_t lanes = tmem + (uint32_t(32 * e) << 16);
        float m = -INFINITY, l = 0.f, z = 0.f;   // of head e: maximum, this lane's share of the denominator, sum of q * zp before the next tile
        float acc[G];
#pragma unroll
        for (int g = 0; g < G; ++g) acc[g] = 0.f;
        // column of ones behind those of the heads
        for (int i = c; i < NB * kTcTok; i += kD)
            *reinterpret_cast<uint4 *>(&sh.vb[i / kTcTok][4 * G / 8][i % kTcTok][0]) =
                G == 1 ? make_uint4(0u, 0u, 0x00003c00u, 0u) : make_uint4(0x00003c00u, 0u, 0u, 0u);
        fence_async_shared();
        const auto move_sums = [&](int i) {   // K sums of tile i to lbuf.  Rows 0-63: rounded parts of tokens 0-63, rows 64-127: remainders.
            const int buf = i % NB;
            if (!mbar_wait(&sh.kdone[buf], i / NB & 1, kStatLFullWait)) return false;
            tc_fence_after();
            constexpr int C = G == 1 ? 4 : G == 2 ? 8 : 16, AT = G == 4 ? 2 : 4;   // columns to read, loads in flight
            float sum[3 * G];
#pragma unroll
            for (int n = 0; n < kSums; n += AT) {
                uint32_t r[AT][C];
#pragma unroll
                for (int m = 0; m < AT; ++m) tmem_ld(r[m], lanes + kDK + KN * (n + m));
#pragma unroll
                for (int m = 0; m < AT; ++m) tmem_wait_ld(r[m]);
#pragma unroll
                for (int k = 0; k < 3 * G; ++k) {
                    float part = __uint_as_float(r[0][k]);
#pragma unroll
                    for (int m = 1; m < AT; ++m) part += __uint_as_float(r[m][k]);
                    sum[k] = n ? sum[k] + part : part;
                }
            }
            tc_fence_before();
            arrive_warp(&sh.kread, lane);
            if (i >= NB && !mbar_wait(&sh.lread[buf], (i / NB & 1) ^ 1, kStatLEmptyWait)) return false;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                sh.lbuf[buf][e >> 1][g][0][32 * (e & 1) + lane] = sum[3 * g];
                sh.lbuf[buf][e >> 1][g][1][32 * (e & 1) + lane] = sum[3 * g + 1] + sum[3 * g + 2];
            }
            arrive_warp(&sh.lfull[buf], lane);
            return true;
        };
        const auto weigh = [&](int i) {   // weights of tile i, the heads that fall to this warp
            const int buf = i % NB, t0 = i * kTcTok + 2 * lane;
            if (e >= G) return true;
            const int g = e;
            const bool in0 = t0 < ntok, in1 = t0 + 1 < ntok;
            const float mk0 = mask_row && in0 ? mask_row[t_begin + t0] * 1.4426950408889634f : 0.f;
            const float mk1 = mask_row && in1 ? mask_row[t_begin + t0 + 1] * 1.4426950408889634f : 0.f;
            if (!mbar_wait(&sh.lfull[buf], i / NB & 1, kStatLFullWait)) return false;
            // the products that read this buffer of weights before are done: add_sums(i - 2) has waited for them
            const float ba = sh.back[g][0], bb = sh.back[g][1];
            const float2 a_hi = *reinterpret_cast<const float2 *>(&sh.lbuf[buf][0][g][0][2 * lane]);
            const float2 a_lo = *reinterpret_cast<const float2 *>(&sh.lbuf[buf][1][g][0][2 * lane]);
            const float2 b_hi = *reinterpret_cast<const float2 *>(&sh.lbuf[buf][0][g][1][2 * lane]);
            const float2 b_lo = *reinterpret_cast<const float2 *>(&sh.lbuf[buf][1][g][1][2 * lane]);
            const float2 A = make_float2((a_hi.x - a_lo.x) * ba, (a_hi.y - a_lo.y) * ba);   // remainders have their sign turned
            const float2 Z = make_float2((b_hi.x - b_lo.x) * bb, (b_hi.y - b_lo.y) * bb);
            float run = Z.x + Z.y;   // zero points: running sum of the alpha * q sums
#pragma unroll
            for (int o = 1; o < 32; o *= 2) {
                const float up = __shfl_up_sync(kFull, run, o);
                if (lane >= o) run += up;
            }
            const float before = __shfl_up_sync(kFull, run, 1);
            if (i == 0) z = (sh.z0[0][g] + sh.z0[1][g]) + (sh.z0[2][g] + sh.z0[3][g]);
            const float z0 = lane ? z + before : z, z1 = z0 + Z.x;
            z += __shfl_sync(kFull, run, 31);
            const float v0 = in0 ? fmaf(A.x + z0, scale2, mk0) : -INFINITY;
            const float v1 = in1 ? fmaf(A.y + z1, scale2, mk1) : -INFINITY;
            const float top = fmaxf(m, redux_max(fmaxf(v0, v1)));
            const bool none = top == -INFINITY;
            const float corr = none ? 1.f : exp2f(m - top), p0 = none ? 0.f : exp2f(v0 - top), p1 = none ? 0.f : exp2f(v1 - top);
            m = top;
            l = fmaf(l, corr, p0 + p1);
            float sfx = p0 + p1;   // weights of the tokens from this lane on
#pragma unroll
            for (int o = 1; o < 32; o *= 2) {
                const float down = __shfl_down_sync(kFull, sfx, o);
                if (lane + o < 32) sfx += down;
            }
            const float after = __shfl_down_sync(kFull, sfx, 1);
            const float s1 = lane < 31 ? after : 0.f, s0 = s1 + p1;
            if (lane == 0) sh.fac[i & 3][g] = make_float2(corr, sfx);
            const uint32_t h0 = pack_half2(p0 * kTcP, s0 * kTcS), h1 = pack_half2(p1 * kTcP, s1 * kTcS);
            const uint32_t r0 = pack_remainder(h0, p0 * kTcP, s0 * kTcS) ^ 0x80008000u, r1 = pack_remainder(h1, p1 * kTcP, s1 * kTcS) ^ 0x80008000u;
            *reinterpret_cast<uint2 *>(&sh.vb[buf][g / 2][2 * lane][g % 2 * 4]) = make_uint2(h0, r0);
            *reinterpret_cast<uint2 *>(&sh.vb[buf][g / 2][2 * lane + 1][g % 2 * 4]) = make_uint2(h1, r1);
            fence_async_shared();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sh.lread[buf]);
                mbar_arrive(&sh.wfull[buf]);
            }
            return true;
        };
        const auto add_sums = [&](int i) {   // V sums of tile i join those before
            const int buf = i % NB;
            if (!mbar_wait(&sh.vdone[buf], i / NB & 1, kStatVWait)) return false;
            tc_fence_after();
            constexpr int N = G == 1 ? 8 : 16;
            uint32_t r[N], last[1];
            tmem_ld(r, lanes + kDV + VN * buf);
            if constexpr (G == 4) tmem_ld(last, lanes + kDV + VN * buf + 4 * G);
            else last[0] = 0u;
            tmem_wait_ld(r);
            if constexpr (G == 4) tmem_wait_ld(last);
            const float ones = __uint_as_float(G == 4 ? last[0] : r[4 * G % N]), a = alpha * unit;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float2 f = sh.fac[i & 3][g];
                const float p = __uint_as_float(r[4 * g]) + __uint_as_float(r[4 * g + 2]);
                const float sfx = __uint_as_float(r[4 * g + 1]) + __uint_as_float(r[4 * g + 3]);
                acc[g] = fmaf(acc[g], f.x, fmaf(zp, f.y, fmaf(a * (1.f / kTcS), sfx, unit * (1.f / kTcP) * p)));
            }
            zp = fmaf(a, ones, zp);
            tc_fence_before();
            arrive_warp(&sh.vread[buf], lane);   // of fac, too
            return true;
        };
#pragma unroll 1
        for (int i = 0; i < n_tiles; ++i) {
            if (!(ok = move_sums(i))) break;
            if (!(ok = weigh(i))) break;
            if (i > 0 && !(ok = add_sums(i - 1))) break;
        }
        if (ok && n_tiles > 0) ok = add_sums(n_tiles - 1);
        if (e < G) {
            const float sum = warp_sum(l);
            if (lane == 0) {
                sh.m[e] = m;
                sh.l[e] = sum;
            }
        }
        if (!ok && lane == 0) sh.dead = 1;
        __syncthreads();
        // sums so far and the appended token
        const bool dead = sh.dead != 0;
        const float mk = append && mask_row ? mask_row[T] * 1.4426950408889634f : 0.f;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float mx = sh.m[g], den = sh.l[g], o = acc[g];
            if (append) {
                const float v = fmaf(sh.self_logit[g], scale2, mk), top = fmaxf(mx, v);
                const bool none = top == -INFINITY;
                const float corr = none ? 1.f : exp2f(mx - top), w = none ? 0.f : exp2f(v - top);
                den = fmaf(den, corr, w);
                o = fmaf(o, corr, w * sh.self_x[c]);
                mx = top;
            }
            if (PART) {
                float *part = scratch + ((size_t(bh) * n_seg + seg) * G + g) * kPartStride;
                if (c == 0) {
                    part[0] = dead ? -INFINITY : mx;
                    part[1] = dead ? __int_as_float(0x7fc00000) : den;
                }
                part[4 + c] = dead ? 0.f : o;
            } else if (!dead) {
                va.out[(size_t(b) * va.Hq + size_t(h) * G + g) * kD + c] = __float2half_rn(o / den);
            }
        }
    } else {
        // ------------------------------------------------------------------------------ copies and products of one tensor
        constexpr uint32_t k_desc = mma_desc(128, KN, true, false), v_hi = mma_desc(128, VN, false, false), v_lo = mma_desc(128, VN, false, true);
        const int which = warp - 12;
        if (elect_one())
            for (int i = 0; i < min(ST, n_tiles); ++i) load_tile(which, i);
        int i = 0;
#pragma unroll 1
        for (; i < n_tiles; ++i) {
            const int buf = i % NB;
            const uint32_t phase = i / NB & 1;
            if (which == 0) {
                if (i > 0 && !(ok = mbar_wait(&sh.kread, (i & 1) ^ 1, kStatKWait))) break;
                if (!(ok = mbar_wait(&sh.kfull[buf], phase, kStatKWait))) break;
                tc_fence_after();
                if (elect_one()) {
                    // Accumulation rounds towards zero.  One running sum over the eight steps puts logits 1 to 5 % further from 64 bits
                    // than several that are added up in fp32; more sums are more to read: four heads, 4-bit, 256 streams x 4096
                    // tokens, four sums 159 us, two 155 us, one 156 us; one and two heads the same with six, four and two.
                    const uint64_t a = mn_major_desc(&sh.a[buf][0][0][0][0], 128, kD * 16), bd = mn_major_desc(&sh.kb[0][0][0], 128, KG == 1 ? 0 : kD * 16);
#pragma unroll
                    for (int n = 0; n < kD / 16; ++n) mma_smem(tmem + kDK + KN * (n % kSums), a + 16 * n, bd + 16 * n, k_desc, n >= kSums);
                    mbar_arrive(&sh.kdone[buf]);   // and this thread has seen back and z0 written: the commit is for the products alone
                    mma_commit(&sh.kdone[buf]);
                }
            } else {
                if (i >= NB && !(ok = mbar_wait(&sh.vread[buf], phase ^ 1, kStatVWait))) break;
                if (!(ok = mbar_wait(&sh.vfull[buf], phase, kStatVWait))) break;
                if (!(ok = mbar_wait(&sh.wfull[buf], phase, kStatVWait))) break;
                tc_fence_after();
                if (elect_one()) {
                    const int steps = (min(kTcTok, ntok - i * kTcTok) + 15) / 16;
                    const uint32_t d = tmem + kDV + VN * buf, a = tmem + kVBuf * buf;
                    const uint64_t bd = mn_major_desc(&sh.vb[buf][0][0][0], 128, VG == 1 ? 0 : kTcTok * 16);
#pragma unroll
                    for (int n = 0; n < kTcTok / 16; ++n)
                        if (n < steps) {
                            mma_tmem(d, a + 8 * n, bd + 16 * n, v_hi, n > 0);
                            mma_tmem(d, a + kVPart + 8 * n, bd + 16 * n, v_lo, true);
                        }
                    mbar_arrive(&sh.vdone[buf]);   // and this thread has seen the weights written, and with them fac
                    mma_commit(&sh.vdone[buf]);
                }
            }
            if (elect_one() && i + ST < n_tiles) load_tile(which, i + ST);   // the threads of this tensor have read the tile
            __syncwarp();
        }
        if (!ok && lane == 0) sh.dead = 1;
        __syncthreads();
        if (sh.dead) {   // products and copies in flight
            uint64_t *done = which ? sh.vdone : sh.kdone;
            for (int k = max(i - NB, 0); k < i; ++k) mbar_wait(&done[k % NB], k / NB & 1, kStatDrain);
            for (int k = i; k < min(i + ST, n_tiles); ++k) mbar_wait(&sh.loaded[which][k % ST], k / ST & 1, kStatDrain);
        }
    }
    __syncthreads();
    if (warp == 12) tmem_free(tmem, kColumns);
}

}  // namespace adkv

using namespace adkv;

ADKV_DEFINE_TU_STATUS(adkv_tu_status_tensor)

template <int BITS, int G, bool PART>
static int launch_tensor(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling, dim3 grid,
                         const int *seq_lens, int n_rank, const CkptArgs &ck, float *scratch, cudaStream_t s)
{
    // no more CTAs on an SM than its tensor memory serves: a third would wait inside its allocation
    constexpr int size = int(sizeof(TensorShared<BITS, G>)), bytes = size > 78 * 1024 ? size : 78 * 1024;
    static_assert(2 * (bytes + 1024) <= 228 * 1024, "shared memory of an SM");
    const auto kernel = decode_attn_tensor_kernel<BITS, G, PART>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return launch_status();
    kernel<<<grid, kTcThreads, bytes, s>>>(ka, va, mask, mask_stride_b, scaling, seq_lens, n_rank, ck, scratch);
    return launch_status();
}

// Arguments checked by the caller (head dim 128, fp32 arithmetic, contracted, tail states present, Hq / Hkv at most 4).
// scratch: partial results of the checkpointed step (adkv_split.cu), or nullptr.
ADKV_HIDDEN int adkv_tensor_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling,
                                        int B, int bits, const int *seq_lens, int n_rank, const CkptArgs &ck, int n_seg,
                                        float *scratch, cudaStream_t s)
{
    const dim3 grid(B * ka.Hkv, n_seg);
    switch (bits * 16 + ka.Hq / ka.Hkv) {
#define ADKV_TC_CASE(BITS_, G_)                                                                                                        \
    case BITS_ * 16 + G_:                                                                                                              \
        return scratch ? launch_tensor<BITS_, G_, true>(ka, va, mask, mask_stride_b, scaling, grid, seq_lens, n_rank, ck, scratch, s)  \
                       : launch_tensor<BITS_, G_, false>(ka, va, mask, mask_stride_b, scaling, grid, seq_lens, n_rank, ck, scratch, s);
        ADKV_TC_CASE(4, 1) ADKV_TC_CASE(4, 2) ADKV_TC_CASE(4, 4)
        ADKV_TC_CASE(2, 1) ADKV_TC_CASE(2, 2) ADKV_TC_CASE(2, 4)
#undef ADKV_TC_CASE
    default: return ADKV_E_SHAPE;
    }
}
