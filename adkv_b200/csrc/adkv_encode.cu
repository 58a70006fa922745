// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point
// and the reference interface each one replaces.
#include "adkv_host.h"

#include <algorithm>
using std::min;

namespace adkv {

// =========================================================================================
// Prefill quantise + pack (canonical arithmetic).  One 64-thread CTA per (batch, head); a thread
// owns two adjacent channels: per token the warp reads 128 contiguous bytes of the fp16 row
// (half2 per lane) and per supergroup it writes 256 contiguous bytes (uint2 per lane).  The next
// word's tokens are fetched while the current word is quantised.
constexpr int kEncThreads = kD / 2;
constexpr int kEncStages = 2;   // 32-token (8 KB) tiles of fp16 input in flight per CTA.  16 KB per CTA lets 14 CTAs share an SM,
                                // which is what a launch over several layers needs (8 layers: 0.645 ms per layer with 2
                                // stages, 0.688 ms with 3); K and V of one layer are 6.9 CTAs per SM either way (0.86 ms)

// A clamped quotient within 4e-6 of a rounding boundary: cannot tell which way the exact one rounds.
constexpr float kClear = 0.5f - 4e-6f;

// Eight tokens for the two channels of a thread,
// speculative quantiser (see quantize_spec) on the channel pair with packed fp32 arithmetic: half the
// issue slots for the adds and multiplies, every element rounded exactly as by the scalar instruction.
// Min/max, the reciprocal and the compare have no packed form and stay scalar.  Returns true when some
// code is in doubt and the group must be redone with the exactly rounded division.
// A word is assembled by shifting: every new code enters at the top (one funnel shift takes the low BITS bits of
// its source) and pushes the earlier tokens down, so after TPW tokens token 0 sits in the lowest field.
template <int BITS, bool GUARDED>
__device__ __forceinline__ bool encode_group(const __half2 *xin /* 8 rows of kD/2 */, Chan (&ch)[2],
                                             uint32_t (&word)[2], float smin, float smax, f32x2 one)
{
    using C = Codec<BITS>;
    constexpr float M = 12582912.f + float(C::BIAS);   // 1.5 * 2^23 + BIAS: the low bits of (v + M) are code + BIAS
    bool doubt = !(ch[0].s < 1e29f) || !(ch[1].s < 1e29f);   // reciprocal would flush to zero
    float worst = 0.f;   // largest distance of a clamped quotient from its code
    f32x2 zp = pk2(ch[0].zp, ch[1].zp), s = pk2(ch[0].s, ch[1].s);
    const f32x2 alpha = pk2(ch[0].alpha, ch[1].alpha), beta = pk2(ch[0].beta, ch[1].beta);
    const f32x2 neg_t = pk2(-ch[0].tc, -ch[1].tc), m2 = pk2(M, M);
    static_for<8>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        const float2 xf = __half22float2(xin[j * (kD / 2)]);
        float s0, s1;
        upk2(s, s0, s1);
        if (GUARDED) {
            s0 = fmaxf(s0, kEps);
            s1 = fmaxf(s1, kEps);
        }
        const f32x2 ss = GUARDED ? pk2(s0, s1) : s;
        float i0, i1;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(i0) : "f"(s0));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(i1) : "f"(s1));
        const f32x2 v = mul2(sub2(pk2(xf.x, xf.y), zp), pk2(i0, i1));
        float v0, v1;
        upk2(v, v0, v1);
        const f32x2 vc = pk2(fminf(fmaxf(v0, C::qlo()), C::qhi()), fminf(fmaxf(v1, C::qlo()), C::qhi()));
        const f32x2 t = add2(vc, m2);
        const f32x2 q = sub2(t, m2);
        float d0, d1;
        upk2(sub2(vc, q), d0, d1);
        if (BITS == 4) worst = fmaxf(fmaxf(worst, fabsf(d0)), fabsf(d1));   // one three-input instruction; not faster for 2 bits
        else doubt |= !(fabsf(d0) < kClear) || !(fabsf(d1) < kClear);
        const f32x2 rh = mul2(q, ss);
        uint32_t t0, t1;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(t0), "=r"(t1) : "l"(t));
        word[0] = __funnelshift_r(word[0], t0, BITS);
        word[1] = __funnelshift_r(word[1], t1, BITS);
        // state update, canonical order (products are added as fma(x, 1, y): see add_product2)
        zp = add_product2(mul2(alpha, rh), one, zp);
        const f32x2 s_new = add_product2(mul2(mul2(s, beta), add2(abs2(q), neg_t)), one, s);
        if (GUARDED) {
            float n0, n1;
            upk2(s_new, n0, n1);
            s = pk2(fminf(fmaxf(n0, smin), smax), fminf(fmaxf(n1, smin), smax));
        } else {
            s = s_new;
        }
    });
    upk2(zp, ch[0].zp, ch[1].zp);
    upk2(s, ch[0].s, ch[1].s);
    return doubt || !(worst < kClear);
}

// Eight tokens of one 2-bit channel, without a quotient.  clamp(rint(r / s), -2, 1) asks on which side of -1.5, -0.5 and 0.5
// the correctly rounded quotient lies, and comparisons answer that exactly:
//    r / s rounds to more than 0.5           <=>  r >  h = s / 2           (the floats next to h are more than half an ulp of
//    r / s rounds to -0.5 or more            <=>  r >= -h                   the quotient away; s / 2 is exact)
//    r / s rounds to -1.5 or less (ties of   <=>  r <= -(1.5 - 2^-24) * s  <=>  r <= -thr, the product rounded up to a float
//    the rounding go to the even 1.5)
// A NaN fails all three and gets -2, as from the minimum and maximum of quantize().  A code can then only move the state to
// four zero points and three scales, each formed as the canonical step forms it (q * s and alpha * q * s are exact multiples of
// s and of alpha * s rounded once), and all of them are on hand before the code is known: what is left from token to token is
// a subtraction, a comparison and two selections, instead of the reciprocal, clamps, roundings and products in a row.
// One B200, K and V of 32 heads, device time with the quotient -> this: 1 x 777 tokens 50.0 -> 38.6 us, 2 x 2000 tokens 123 -> 94
// us, 4 x 2000 tokens 131 -> 113 us, 1 x 60 tokens 8.2 -> 6.1 us.
// Returns true where that does not hold: scales near overflow, which the range of the unguarded form leaves out even without an
// upper bound, alpha that is not finite, a zero point of -0.
template <bool GUARDED>
__device__ __forceinline__ bool encode_group_compare(const __half *xin, Chan &c, uint32_t &word, float smin, float smax)
{
    const bool odd = !(c.s < 1e29f) || !(fabsf(c.alpha) < INFINITY) || __float_as_uint(c.zp) == 0x80000000u;
    const float err0 = __fsub_rn(0.f, c.tc), err1 = __fsub_rn(1.f, c.tc), err2 = __fsub_rn(2.f, c.tc);
    float top = c.s;
    static_for<8>([&](auto jc) {
        const float x = __half2float(xin[decltype(jc)::value * kD]);
        const float ss = GUARDED ? fmaxf(c.s, kEps) : c.s;
        const float h = __fmul_rn(ss, 0.5f), thr = __fmaf_ru(ss, 0.5f - 0x1p-24f, ss);
        const float as = __fmul_rn(c.alpha, ss), sb = __fmul_rn(c.s, c.beta);
        const float z1 = __fadd_rn(c.zp, as), zm1 = __fsub_rn(c.zp, as), zm2 = __fmaf_rn(-2.f, as, c.zp);
        const float s0 = __fadd_rn(c.s, __fmul_rn(sb, err0)), s1 = __fadd_rn(c.s, __fmul_rn(sb, err1)),
                    s2 = __fadd_rn(c.s, __fmul_rn(sb, err2));
        const float r = __fsub_rn(x, c.zp);
        const bool is1 = r > h, ge0 = r >= -h, gem1 = r > -thr;
        const uint32_t field = gem1 ? (is1 ? 3u : ge0 ? 2u : 1u) : 0u;
        c.zp = gem1 ? (is1 ? z1 : ge0 ? c.zp : zm1) : zm2;
        const float s_new = gem1 ? (ge0 && !is1 ? s0 : s1) : s2;
        c.s = GUARDED ? fminf(fmaxf(s_new, smin), smax) : s_new;
        if (GUARDED) top = fmaxf(top, c.s);
        word = __funnelshift_r(word, field, 2);
    });
    return odd || (GUARDED && !(top < 1e29f));
}

// The same for the one channel of a thread (launches with few streams, see launch_encode): every operation rounded as in
// encode_group.  xin: 8 rows of kD.
template <int BITS, bool GUARDED>
__device__ __forceinline__ bool encode_group(const __half *xin, Chan (&ch)[1], uint32_t (&word)[1], float smin, float smax, f32x2)
{
    using C = Codec<BITS>;
    constexpr float M = 12582912.f + float(C::BIAS);
    Chan &c = ch[0];
    if constexpr (BITS == 2) return encode_group_compare<GUARDED>(xin, c, word[0], smin, smax);
    const bool doubt = !(c.s < 1e29f);
    float worst = 0.f;
    static_for<8>([&](auto jc) {
        const float x = __half2float(xin[decltype(jc)::value * kD]);
        const float ss = GUARDED ? fmaxf(c.s, kEps) : c.s;
        float inv;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(ss));
        const float v = fminf(fmaxf(__fmul_rn(__fsub_rn(x, c.zp), inv), C::qlo()), C::qhi());
        const float t = __fadd_rn(v, M), q = __fsub_rn(t, M);
        worst = fmaxf(worst, fabsf(__fsub_rn(v, q)));
        advance_canonical_g<GUARDED>(q, __fmul_rn(q, ss), c, smin, smax);
        word[0] = __funnelshift_r(word[0], __float_as_uint(t), BITS);
    });
    return doubt || !(worst < kClear);
}

// One tensor (K or V) of a launch, which takes several, so that K and V of a layer are quantised side by side.
struct EncTensor {
    uint32_t *cache;
    const __half *x;
    ParamPtrs p;
    float *tail;
    float *ckpt;   // state checkpoints [B*H][n_ckpt_cap][2][D] or nullptr; entry k = state before token (k+1)*interval
};
struct CkptSpec {
    int interval;     // tokens between checkpoints (multiple of 32), 0 = none
    int n_ckpt_cap;
    int D;            // head dim (128, 256 or 512); a CTA handles one 128-channel slice of one stream
};
constexpr int kEncMaxTensors = 16;   // tensors per launch: K and V of up to 8 layers (the struct is a kernel parameter)
struct EncBatch {
    EncTensor t[kEncMaxTensors];
};

// WIDE = false: head dim 128, all strides are compile-time constants.  CPT: channels per thread, 2 or 1.
template <int CPT>
struct EncIo;    // a thread's channels of a row: half inputs, packed words, float states
template <>
struct EncIo<2> {
    using Half = __half2;
    using Word = uint2;
    using Float = float2;
    __device__ static void get(float2 v, float (&o)[2]) { o[0] = v.x; o[1] = v.y; }
    __device__ static void get(__half2 v, float (&o)[2]) { get(__half22float2(v), o); }
    __device__ static void get(uint2 v, uint32_t (&o)[2]) { o[0] = v.x; o[1] = v.y; }
    __device__ static uint2 word(const uint32_t (&w)[2]) { return make_uint2(w[0], w[1]); }
    __device__ static float2 zp(const Chan (&c)[2]) { return make_float2(c[0].zp, c[1].zp); }
    __device__ static float2 scale(const Chan (&c)[2]) { return make_float2(c[0].s, c[1].s); }
};
template <>
struct EncIo<1> {
    using Half = __half;
    using Word = uint32_t;
    using Float = float;
    __device__ static void get(float v, float (&o)[1]) { o[0] = v; }
    __device__ static void get(__half v, float (&o)[1]) { o[0] = __half2float(v); }
    __device__ static void get(uint32_t v, uint32_t (&o)[1]) { o[0] = v; }
    __device__ static uint32_t word(const uint32_t (&w)[1]) { return w[0]; }
    __device__ static float zp(const Chan (&c)[1]) { return c[0].zp; }
    __device__ static float scale(const Chan (&c)[1]) { return c[0].s; }
};

// A CTA takes one 128-channel slice (blockIdx.x) of one stream of one tensor (blockIdx.y).  PART: the launch is one of two that run side
// by side (see launch_encode) and takes the slices from `first` on, n_slices per tensor.
constexpr int kAlone = 0, kFirstPart = 1, kSecondPart = 2;
template <int BITS, bool WIDE, int CPT, int PART = kAlone>
__global__ void __launch_bounds__(kD / CPT) encode_kernel(EncBatch batch, CkptSpec cs, int first, int n_slices, int H, int T,
                                                             int n_super_cap, int t_start, float smin, float smax)
{
    if (PART == kFirstPart) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // the work that follows on the stream waits for the second part, so that one ends after the first
    const auto leave = [] {
        if (PART == kSecondPart) asm volatile("griddepcontrol.wait;" ::: "memory");
    };
    const int number = first + blockIdx.x, slice = PART == kAlone ? blockIdx.x : number % n_slices;
    using C = Codec<BITS>;
    using Io = EncIo<CPT>;
    using Half = typename Io::Half;
    using Word = typename Io::Word;
    using Float = typename Io::Float;
    const EncTensor &et = batch.t[PART == kAlone ? blockIdx.y : number / n_slices];
    uint32_t *__restrict__ cache = et.cache;
    const __half *__restrict__ x = et.x;
    const ParamPtrs p = et.p;
    float *__restrict__ tail = et.tail;
    const int D = WIDE ? cs.D : kD, S = WIDE ? D / kD : 1;
    const int bh = slice / S, h = bh % H, c0 = kD * (slice % S) + CPT * threadIdx.x;   // c0: channel in the head
    const size_t po = size_t(h) * D + c0;
    Chan ch[CPT];
    float beta[CPT], target[CPT];
    {
        float al[CPT], zp[CPT], sc[CPT];
        Io::get(*reinterpret_cast<const Half *>(p.alpha + po), al);
        Io::get(*reinterpret_cast<const Half *>(p.beta + po), beta);
        Io::get(*reinterpret_cast<const Half *>(p.target + po), target);
        if (t_start > 0) {
            Io::get(*reinterpret_cast<const Float *>(tail + size_t(bh) * 2 * D + c0), zp);
            Io::get(*reinterpret_cast<const Float *>(tail + size_t(bh) * 2 * D + D + c0), sc);
        } else {
            Io::get(*reinterpret_cast<const Half *>(p.zp_init + po), zp);
            Io::get(*reinterpret_cast<const Half *>(p.scale_init + po), sc);
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) ch[c] = Chan{zp[c], sc[c], al[c], beta[c], target[c]};
    }
    SafeRange safe;
    safe.template init<BITS, CPT>(beta, target, smin, fminf(smax, 1e29f));   // 1e29: see encode_group_compare
    const f32x2 one = opaque_ones2();

    __shared__ alignas(128) __half buf[kEncStages][32 * kD];
    __shared__ uint64_t bar[kEncStages];
    if (threadIdx.x == 0) {
        for (int i = 0; i < kEncStages; ++i) mbar_init(&bar[i], 1);
        mbar_init_fence();
    }
    __syncthreads();

    Word *w = reinterpret_cast<Word *>(cache + size_t(bh) * n_super_cap * D + c0);   // stride RS per word row
    const Half *xs = reinterpret_cast<const Half *>(x + size_t(bh) * T * D + c0);    // stride RS per token
    const int RS = D / CPT;          // row stride in global memory (words / inputs of a thread)
    constexpr int SRS = kD / CPT;    // row stride of the staged slice in shared memory

    // one token with a run-time field position, exactly rounded division (partial words, redone groups)
    // (the word is shifted, not indexed: see encode_group)
    auto exact_token = [&](int t, uint32_t(&word)[CPT]) {
        float xa[CPT];
        Io::get(xs[size_t(t - t_start) * RS], xa);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            float rh;
            const float q = quantize<BITS>(xa[c], ch[c], rh);
            word[c] = __funnelshift_r(word[c], uint32_t(int(q) + C::BIAS), BITS);
            advance_canonical(q, rh, ch[c], smin, smax);
        }
    };

    // checkpoint k is written when the state before token (k+1)*interval is reached
    float *ckpt = (et.ckpt && cs.interval > 0) ? et.ckpt + size_t(bh) * cs.n_ckpt_cap * 2 * D + c0 : nullptr;
    int next_ckpt = ckpt ? (t_start / cs.interval + 1) * cs.interval : 0x7fffffff;
    auto checkpoint = [&](int t_reached) {
        if (t_reached == next_ckpt) {
            const int k = next_ckpt / cs.interval - 1;
            if (k < cs.n_ckpt_cap) {
                *reinterpret_cast<Float *>(ckpt + size_t(k) * 2 * D) = Io::zp(ch);
                *reinterpret_cast<Float *>(ckpt + size_t(k) * 2 * D + D) = Io::scale(ch);
            }
            next_ckpt += cs.interval;
        }
    };

    const int t_end = t_start + T;
    int t = t_start;
    uint32_t word[CPT] = {};
    auto flush = [&](int at) {   // a word is complete
        w[size_t(at / C::TPW) * RS] = Io::word(word);
#pragma unroll
        for (int c = 0; c < CPT; ++c) word[c] = 0u;
    };
    // a chunk that starts inside a word keeps the fields already there (moved to the top, where the shifting
    // assembly expects the tokens seen so far)
    if (t % C::TPW != 0 && t < t_end) {
        Io::get(w[size_t(t / C::TPW) * RS], word);
        const int up = BITS * (C::TPW - t % C::TPW);
#pragma unroll
        for (int c = 0; c < CPT; ++c) word[c] <<= up;
    }
    // tokens up to the next multiple of 8
    for (; t < t_end && t % 8 != 0; ++t) {
        exact_token(t, word);
        checkpoint(t + 1);
        if ((t + 1) % C::TPW == 0) flush(t);
    }
    // Groups of 8 tokens.  The fp16 rows of the stream are contiguous, so they are staged through a
    // ring of 32-token tiles filled by bulk copies (1-D TMA, issued by thread 0) that run ahead of
    // the quantiser by kEncStages - 1 tiles.
    const int n_groups = (t_end - t) / 8;
    const int n_tiles = (n_groups + 3) / 4;
    const __half *src = x + (size_t(bh) * T + (t - t_start)) * D + kD * (slice % S);
    auto issue = [&](int i) {
        const int rows = min(4, n_groups - 4 * i) * 8;
        const uint32_t bytes = uint32_t(rows) * kD * 2;
        mbar_expect_tx(&bar[i % kEncStages], bytes);
        if (S == 1) {
            bulk_load(&buf[i % kEncStages][0], src + size_t(i) * 32 * kD, bytes, &bar[i % kEncStages]);
        } else {   // the slice's 256-byte rows are strided in global memory: one copy per token row
            for (int r = 0; r < rows; ++r)
                bulk_load(&buf[i % kEncStages][r * kD], src + (size_t(i) * 32 + r) * D, kD * 2, &bar[i % kEncStages]);
        }
    };
    if (threadIdx.x == 0)
        for (int i = 0; i < min(kEncStages, n_tiles); ++i) issue(i);
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
        const bool landed = mbar_wait_bounded(&bar[i % kEncStages], (i / kEncStages) & 1, kStatKWait);
        if (!__syncthreads_and(landed)) {
            // give up as one CTA; let copies already in flight land (bounded) before the memory is released
            for (int k = i; k < min(n_tiles, i + kEncStages); ++k)
                if (!mbar_wait_bounded(&bar[k % kEncStages], (k / kEncStages) & 1, kStatDrain)) break;
            leave();
            return;
        }
        const int ng = min(4, n_groups - 4 * i);
#pragma unroll 1
        for (int g = 0; g < ng; ++g, t += 8) {
            const Half *rows = reinterpret_cast<const Half *>(&buf[i % kEncStages][0]) + g * 8 * SRS + threadIdx.x;
            Chan saved[CPT];
            uint32_t word_in[CPT];
#pragma unroll
            for (int c = 0; c < CPT; ++c) { saved[c] = ch[c]; word_in[c] = word[c]; }
            const bool doubt = safe.holds(ch) ? encode_group<BITS, false>(rows, ch, word, smin, smax, one)
                                              : encode_group<BITS, true>(rows, ch, word, smin, smax, one);
            if (doubt) {   // rare, per thread: redo the group from the saved state with the exact quantiser
#pragma unroll
                for (int c = 0; c < CPT; ++c) { ch[c] = saved[c]; word[c] = word_in[c]; }
                for (int j = 0; j < 8; ++j) exact_token(t + j, word);
            }
            checkpoint(t + 8);
            if ((t + 8) % C::TPW == 0) flush(t);
        }
        __syncthreads();   // every thread is done with this stage
        if (threadIdx.x == 0 && i + kEncStages < n_tiles) issue(i + kEncStages);
    }
    // trailing tokens; unused fields of the last word stay zero
    for (; t < t_end; ++t) {
        exact_token(t, word);
        checkpoint(t + 1);
    }
    if (t % C::TPW != 0) {   // bring the tokens of the last, partial word down; its unused fields are zero
        const int down = BITS * (C::TPW - t % C::TPW);
#pragma unroll
        for (int c = 0; c < CPT; ++c) word[c] >>= down;
        w[size_t(t / C::TPW) * RS] = Io::word(word);
    }
    if (tail) {
        *reinterpret_cast<Float *>(tail + size_t(bh) * 2 * D + c0) = Io::zp(ch);
        *reinterpret_cast<Float *>(tail + size_t(bh) * 2 * D + D + c0) = Io::scale(ch);
    }
    leave();
}

// Tensors of one append launch over several layers: K and V of up to 32 (4.6 KB of kernel parameters).
constexpr int kAppendMaxTensors = 64;
struct AppendBatch {
    EncTensor t[kAppendMaxTensors];
};

// Single-token append from the persisted tail state, a channel pair per thread and two 128-channel slices per CTA.
// A step moves 26 bytes a channel, so it is bound by the latency of one round of loads and by how many threads the chip
// takes in at once: half the threads and twice the bytes per load of one channel per thread (append_kernel).  All
// tensors of 32 layers in one launch instead of four: 41 us -> 21.5 us a call at 32 layers x batch 16 x 32 heads, 2-bit,
// one B200 (109 MB of tails, words and tokens that cannot be left out: 17 us at the measured copy bandwidth).
// Wider accesses need the alignment that append_aligned checks; what fails it takes append_kernel.
template <int BITS, class Batch>
__global__ void __launch_bounds__(kD) append_pair_kernel(const __grid_constant__ Batch batch, CkptSpec cs, int H, int n_slices,
                                                         int T, int n_super_cap, float smin, float smax)
{
    using C = Codec<BITS>;
    const EncTensor &et = batch.t[blockIdx.y];
    const int D = cs.D, S = D / kD;
    const int slice = blockIdx.x * 2 + (threadIdx.x >> 6);
    if (slice >= n_slices) return;
    const int bh = slice / S, h = bh % H, c = kD * (slice % S) + 2 * (threadIdx.x & 63);
    const size_t po = size_t(h) * D + c;
    uint2 *slot = reinterpret_cast<uint2 *>(et.cache + (size_t(bh) * n_super_cap + T / C::TPW) * D + c);
    float2 *zp_at = reinterpret_cast<float2 *>(et.tail + size_t(bh) * 2 * D + c), *s_at = zp_at + D / 2;
    const float2 al = __half22float2(*reinterpret_cast<const __half2 *>(et.p.alpha + po));
    const float2 be = __half22float2(*reinterpret_cast<const __half2 *>(et.p.beta + po));
    const float2 tg = __half22float2(*reinterpret_cast<const __half2 *>(et.p.target + po));
    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(et.x + size_t(bh) * D + c));
    const float2 zp = *zp_at, sc = *s_at;
    const uint2 old = *slot;
    Chan ch[2] = {Chan{zp.x, sc.x, al.x, be.x, tg.x}, Chan{zp.y, sc.y, al.y, be.y, tg.y}};
    const float xv[2] = {x.x, x.y};
    uint32_t word[2] = {old.x, old.y};
    const int sh = BITS * (T % C::TPW);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float rh;
        const float q = quantize<BITS>(xv[i], ch[i], rh);
        word[i] = (word[i] & ~(C::FIELD << sh)) | (uint32_t(int(q) + C::BIAS) << sh);
        advance_canonical(q, rh, ch[i], smin, smax);
    }
    *slot = make_uint2(word[0], word[1]);
    *zp_at = make_float2(ch[0].zp, ch[1].zp);
    *s_at = make_float2(ch[0].s, ch[1].s);
    if (et.ckpt && cs.interval > 0 && (T + 1) % cs.interval == 0) {
        const int k = (T + 1) / cs.interval - 1;
        if (k < cs.n_ckpt_cap) {
            float *dst = et.ckpt + (size_t(bh) * cs.n_ckpt_cap + k) * 2 * D + c;
            *reinterpret_cast<float2 *>(dst) = make_float2(ch[0].zp, ch[1].zp);
            *reinterpret_cast<float2 *>(dst + D) = make_float2(ch[0].s, ch[1].s);
        }
    }
}

// The same, one channel per thread: for pointers that are only aligned to their own type.
template <int BITS>
__global__ void __launch_bounds__(kD) append_kernel(EncBatch batch, CkptSpec cs, int H, int T, int n_super_cap,
                                                    float smin, float smax)
{
    using C = Codec<BITS>;
    const EncTensor &et = batch.t[blockIdx.y];
    uint32_t *__restrict__ cache = et.cache;
    const __half *__restrict__ x_new = et.x;
    const ParamPtrs p = et.p;
    float *__restrict__ tail = et.tail;
    const int D = cs.D, S = D / kD;
    const int bh = blockIdx.x / S, h = bh % H, c = kD * (blockIdx.x % S) + threadIdx.x;
    const size_t po = size_t(h) * D + c;
    Chan ch;
    ch.alpha = __half2float(p.alpha[po]);
    ch.beta = __half2float(p.beta[po]);
    ch.tc = __half2float(p.target[po]);
    ch.zp = tail[size_t(bh) * 2 * D + c];
    ch.s = tail[size_t(bh) * 2 * D + D + c];
    float rh;
    const float q = quantize<BITS>(__half2float(x_new[size_t(bh) * D + c]), ch, rh);
    uint32_t *slot = cache + (size_t(bh) * n_super_cap + T / C::TPW) * D + c;
    const int sh = BITS * (T % C::TPW);
    *slot = (*slot & ~(C::FIELD << sh)) | (uint32_t(int(q) + C::BIAS) << sh);
    advance_canonical(q, rh, ch, smin, smax);
    tail[size_t(bh) * 2 * D + c] = ch.zp;
    tail[size_t(bh) * 2 * D + D + c] = ch.s;
    if (et.ckpt && cs.interval > 0 && (T + 1) % cs.interval == 0) {
        const int k = (T + 1) / cs.interval - 1;
        if (k < cs.n_ckpt_cap) {
            float *dst = et.ckpt + (size_t(bh) * cs.n_ckpt_cap + k) * 2 * D;
            dst[c] = ch.zp;
            dst[D + c] = ch.s;
        }
    }
}

}  // namespace adkv

using namespace adkv;

ADKV_DEFINE_TU_STATUS(adkv_tu_status_encode)

static int encode_check(const void *cache, const void *x, const adkv_params *p, const void *tail, int T, int t_start)
{
    if (!cache || (!x && T > 0) || !params_ok(p)) return ADKV_E_NULL;
    if (t_start > 0 && !tail) return ADKV_E_START;
    if ((reinterpret_cast<uintptr_t>(cache) & 7u) || (reinterpret_cast<uintptr_t>(x) & 15u) ||
        (reinterpret_cast<uintptr_t>(tail) & 7u) || (reinterpret_cast<uintptr_t>(p->zp_init) & 3u) ||
        (reinterpret_cast<uintptr_t>(p->scale_init) & 3u) || (reinterpret_cast<uintptr_t>(p->alpha) & 3u) ||
        (reinterpret_cast<uintptr_t>(p->beta) & 3u) || (reinterpret_cast<uintptr_t>(p->target) & 3u))
        return ADKV_E_ALIGN;
    return 0;
}

static EncTensor enc_tensor(void *cache, const void *x, const adkv_params *p, void *tail, void *ckpt = nullptr)
{
    return EncTensor{static_cast<uint32_t *>(cache), static_cast<const __half *>(x), to_ptrs(p),
                     static_cast<float *>(tail), static_cast<float *>(ckpt)};
}

static int ckpt_check(const void *k_ckpt, const void *v_ckpt, int interval, int n_ckpt_cap, int t_last_plus_1)
{
    if (interval <= 0 || interval % 32 != 0 || n_ckpt_cap < 0) return ADKV_E_SHAPE;
    if (!k_ckpt || !v_ckpt) return ADKV_E_NULL;
    if ((reinterpret_cast<uintptr_t>(k_ckpt) & 15u) || (reinterpret_cast<uintptr_t>(v_ckpt) & 15u)) return ADKV_E_ALIGN;
    if (t_last_plus_1 / interval > n_ckpt_cap) return ADKV_E_CAPACITY;
    return 0;
}

// An odd number of two-warp CTAs on an SM leaves two of its schedulers a warp more than the other two, and all wait for those.  Then
// the CTAs beyond the even number come as four warps of one channel a thread, one for each scheduler: two launches side by side
// (the second is a programmatic dependent that starts as soon as the first is in place).  Device time on a B200, K and V of 32 heads, 4-bit,
// one launch -> two: 16 x 8192 tokens (6.9 CTAs an SM) 856 -> 796 us, 15 x 4000 426 -> 392 us, 11 x 4000 (4.8) 346 -> 323 us, 19 x 2000 (8.2)
// 262 -> 243 us, 1628 slices (11) x 1024 162 -> 148 us, 612 (4.1) x 256 25.7 -> 25.4 us; 2-bit 16 x 8192 852 -> 818 us, 14 x 2000 (6.1) 216 -> 206
// us, 1628 x 1024 157 -> 152 us.  Short 2-bit prefills of few CTAs an SM do not gain: 612 x 256 24.9 -> 27.2 us, x 768 66.2 -> 68.3 us, x 2048 173.1 ->
// 171.2 us; 908 (6.1) x 256 29.3 -> 30.1 us, x 384 42.7 -> 41.9 us; 1204 (8.1) x 256 34.5 -> 34.3 us.  With more than one left over for an SM
// the two do not come out even; twelve CTAs an SM would gain as eleven do.  Returns the size of the first, 0 for one launch.
static int side_by_side(long long grid, int T, int bits)
{
    const long long even = grid / (2 * kSMs) * (2 * kSMs), rest = grid - even;
    const int from = bits == 4 || even > 6 * kSMs ? 256 : even > 4 * kSMs ? 384 : 2048;
    return even >= 4 * kSMs && even <= 10 * kSMs && rest > 0 && rest <= kSMs && T >= from ? int(even) : 0;
}

static int launch_encode(const EncBatch &b, int n, int B, int H, int T, int D, int n_super_cap, int bits,
                         int t_start, float smin, float smax, void *stream, CkptSpec cs = CkptSpec{0, 0, 0})
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cs.D = D;
    const int n_slices = B * H * (D / kD);
    const long long grid = (long long)n_slices * n;
    // One channel per thread while that leaves a warp scheduler at most three warps: a warp then has its scheduler (nearly)
    // to itself and takes as long as its own instructions, of which one channel needs about half as many as a pair.
    // Measured on a B200, K and V of 32 heads: 1 x 4000 tokens 251 -> 231 us, 2 x 2000 tokens 131 -> 121 us, 4 x 2000 tokens
    // 137 -> 133 us, 6 x 3000 tokens 213 -> 199 us (2-bit 224 -> 212 us), but 8 x 2000 tokens 148 -> 155 us.  With more streams the
    // schedulers are busy and the packed pair needs fewer issue slots per channel.
    const bool few = grid * (kD / 32) <= 3 * kSchedulers;
    const auto kernel = D == kD ? (bits == 4 ? (few ? encode_kernel<4, false, 1> : encode_kernel<4, false, 2>)
                                             : (few ? encode_kernel<2, false, 1> : encode_kernel<2, false, 2>))
                                : (bits == 4 ? encode_kernel<4, true, 2> : encode_kernel<2, true, 2>);
    const int split = D == kD && !few ? side_by_side(grid, T, bits) : 0;
    if (split) {
        const auto first = bits == 4 ? encode_kernel<4, false, 2, kFirstPart> : encode_kernel<2, false, 2, kFirstPart>;
        const auto second = bits == 4 ? encode_kernel<4, false, 1, kSecondPart> : encode_kernel<2, false, 1, kSecondPart>;
        // A refusal must not leave half of the prefill written: the second kernel is loaded (asking for its attributes does that) before
        // the first runs, and where it may not run beside the first it follows as an ordinary launch.
        cudaFuncAttributes unused;
        if (cudaFuncGetAttributes(&unused, second) != cudaSuccess) return launch_status();
        first<<<split, kEncThreads, 0, s>>>(b, cs, 0, n_slices, H, T, n_super_cap, t_start, smin, smax);
        if (int rc = launch_status()) return rc;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(int(grid) - split);
        cfg.blockDim = dim3(kD);
        cfg.stream = s;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, second, b, cs, split, n_slices, H, T, n_super_cap, t_start, smin, smax) != cudaSuccess) {
            cudaGetLastError();
            second<<<cfg.gridDim, cfg.blockDim, 0, s>>>(b, cs, split, n_slices, H, T, n_super_cap, t_start, smin, smax);
        }
        return launch_status();
    }
    kernel<<<dim3(n_slices, n), D == kD && few ? kD : kEncThreads, 0, s>>>(b, cs, 0, n_slices, H, T, n_super_cap, t_start, smin, smax);
    return launch_status();
}

static bool append_aligned(const EncTensor &t)
{
    const auto at = [](const void *p, unsigned n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; };
    return at(t.cache, 8) && at(t.x, 4) && at(t.tail, 8) && at(t.ckpt, 8) && at(t.p.alpha, 4) && at(t.p.beta, 4) &&
           at(t.p.target, 4);
}

// Batch: EncBatch, or AppendBatch for the layered call.
template <class Batch>
static int launch_append(const Batch &b, int n, int B, int H, int T, int D, int n_super_cap, int bits,
                         float smin, float smax, void *stream, CkptSpec cs = CkptSpec{0, 0, 0})
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cs.D = D;
    const int n_slices = B * H * (D / kD);
    bool aligned = true;
    for (int i = 0; i < n; ++i) aligned = aligned && append_aligned(b.t[i]);
    if (aligned) {
        const dim3 grid((n_slices + 1) / 2, n);
        if (bits == 4) append_pair_kernel<4><<<grid, kD, 0, s>>>(b, cs, H, n_slices, T, n_super_cap, smin, smax);
        else append_pair_kernel<2><<<grid, kD, 0, s>>>(b, cs, H, n_slices, T, n_super_cap, smin, smax);
        return launch_status();
    }
    for (int i = 0; i < n; i += kEncMaxTensors) {
        EncBatch part{};
        const int m = min(kEncMaxTensors, n - i);
        for (int j = 0; j < m; ++j) part.t[j] = b.t[i + j];
        const dim3 grid(n_slices, m);
        if (bits == 4) append_kernel<4><<<grid, kD, 0, s>>>(part, cs, H, T, n_super_cap, smin, smax);
        else append_kernel<2><<<grid, kD, 0, s>>>(part, cs, H, T, n_super_cap, smin, smax);
        if (int rc = launch_status()) return rc;
    }
    return 0;
}

ADKV_HIDDEN int adkv_half_encode(void *k_cache, const void *k, const adkv_params *kp, void *k_tail, void *k_ckpt,
                                 void *v_cache, const void *v, const adkv_params *vp, void *v_tail, void *v_ckpt,
                                 int interval, int n_ckpt_cap, int n, int B, int H, int T, int D, int n_super_cap,
                                 int bits, int t_start, cudaStream_t s);
ADKV_HIDDEN int adkv_half_append(void *k_cache, const void *k_new, const adkv_params *kp, void *k_tail, void *k_ckpt,
                                 void *v_cache, const void *v_new, const adkv_params *vp, void *v_tail, void *v_ckpt,
                                 int interval, int n_ckpt_cap, int n, int B, int H, int T, int D, int n_super_cap,
                                 int bits, cudaStream_t s);

extern "C" {

int adkv_encode_kv_flags(void *k_cache, const void *k, const adkv_params *kp, void *k_tail, void *k_ckpt,
                         void *v_cache, const void *v, const adkv_params *vp, void *v_tail, void *v_ckpt,
                         int interval, int n_ckpt_cap, int B, int H, int T, int D, int n_super_cap, int bits,
                         int t_start, float scale_min, float scale_max, unsigned flags, void *stream)
{
    const bool pair = v_cache != nullptr;
    if (interval < 0 || (interval > 0 && !pair)) return ADKV_E_SHAPE;   // checkpoints are kept for K and V together
    if (!(flags & ADKV_FLAG_HALF_STATE)) {
        if (interval > 0)
            return adkv_encode_kv_ckpt(k_cache, k, kp, k_tail, k_ckpt, v_cache, v, vp, v_tail, v_ckpt, interval, n_ckpt_cap,
                                       B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max, stream);
        return pair ? adkv_encode_kv(k_cache, k, kp, k_tail, v_cache, v, vp, v_tail, B, H, T, D, n_super_cap, bits,
                                     t_start, scale_min, scale_max, stream)
                    : adkv_encode(k_cache, k, kp, k_tail, B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max,
                                  stream);
    }
    if (t_start < 0) return ADKV_E_SHAPE;
    if (int rc = encode_check(k_cache, k, kp, k_tail, T, t_start)) return rc;
    if (pair)
        if (int rc = encode_check(v_cache, v, vp, v_tail, T, t_start)) return rc;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, t_start + T)) return rc;
    if (interval > 0)
        if (int rc = ckpt_check(k_ckpt, v_ckpt, interval, n_ckpt_cap, t_start + T)) return rc;
    if (B * H == 0 || (T == 0 && !((k_tail || v_tail) && t_start == 0))) return 0;
    return adkv_half_encode(k_cache, k, kp, k_tail, k_ckpt, v_cache, v, vp, v_tail, v_ckpt, interval, n_ckpt_cap,
                            pair ? 2 : 1, B, H, T, D, n_super_cap, bits, t_start, static_cast<cudaStream_t>(stream));
}

int adkv_append_kv_flags(void *k_cache, const void *k_new, const adkv_params *kp, void *k_tail, void *k_ckpt,
                         void *v_cache, const void *v_new, const adkv_params *vp, void *v_tail, void *v_ckpt,
                         int interval, int n_ckpt_cap, int B, int H, int T, int D, int n_super_cap, int bits,
                         float scale_min, float scale_max, unsigned flags, void *stream)
{
    const bool pair = v_cache != nullptr;
    if (interval < 0 || (interval > 0 && !pair)) return ADKV_E_SHAPE;
    if (!(flags & ADKV_FLAG_HALF_STATE)) {
        if (interval > 0)
            return adkv_append_kv_ckpt(k_cache, k_new, kp, k_tail, k_ckpt, v_cache, v_new, vp, v_tail, v_ckpt, interval,
                                       n_ckpt_cap, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream);
        return pair ? adkv_append_kv(k_cache, k_new, kp, k_tail, v_cache, v_new, vp, v_tail, B, H, T, D, n_super_cap,
                                     bits, scale_min, scale_max, stream)
                    : adkv_append(k_cache, k_new, kp, k_tail, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream);
    }
    if (!k_cache || !k_new || !k_tail || !params_ok(kp)) return ADKV_E_NULL;
    if (pair && (!v_new || !v_tail || !params_ok(vp))) return ADKV_E_NULL;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, T + 1)) return rc;
    if (interval > 0)
        if (int rc = ckpt_check(k_ckpt, v_ckpt, interval, n_ckpt_cap, T + 1)) return rc;
    if (B * H == 0) return 0;
    return adkv_half_append(k_cache, k_new, kp, k_tail, k_ckpt, v_cache, v_new, vp, v_tail, v_ckpt, interval, n_ckpt_cap,
                            pair ? 2 : 1, B, H, T, D, n_super_cap, bits, static_cast<cudaStream_t>(stream));
}

int adkv_encode(void *cache, const void *x, const adkv_params *p, void *tail, int B, int H, int T, int D,
                int n_super_cap, int bits, int t_start, float scale_min, float scale_max, void *stream)
{
    if (t_start < 0) return ADKV_E_SHAPE;
    if (int rc = encode_check(cache, x, p, tail, T, t_start)) return rc;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, t_start + T)) return rc;
    if (B * H == 0 || (T == 0 && !(tail && t_start == 0))) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(cache, x, p, tail);
    return launch_encode(b, 1, B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max, stream);
}

int adkv_encode_kv(void *k_cache, const void *k, const adkv_params *kp, void *k_tail, void *v_cache, const void *v,
                   const adkv_params *vp, void *v_tail, int B, int H, int T, int D, int n_super_cap, int bits,
                   int t_start, float scale_min, float scale_max, void *stream)
{
    if (t_start < 0) return ADKV_E_SHAPE;
    if (int rc = encode_check(k_cache, k, kp, k_tail, T, t_start)) return rc;
    if (int rc = encode_check(v_cache, v, vp, v_tail, T, t_start)) return rc;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, t_start + T)) return rc;
    if (B * H == 0 || (T == 0 && !((k_tail || v_tail) && t_start == 0))) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(k_cache, k, kp, k_tail);
    b.t[1] = enc_tensor(v_cache, v, vp, v_tail);
    return launch_encode(b, 2, B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max, stream);
}

int adkv_append(void *cache, const void *x_new, const adkv_params *p, void *tail, int B, int H, int T, int D,
                int n_super_cap, int bits, float scale_min, float scale_max, void *stream)
{
    if (!cache || !x_new || !tail || !params_ok(p)) return ADKV_E_NULL;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, T + 1)) return rc;
    if (B * H == 0) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(cache, x_new, p, tail);
    return launch_append(b, 1, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream);
}

int adkv_append_kv(void *k_cache, const void *k_new, const adkv_params *kp, void *k_tail, void *v_cache,
                   const void *v_new, const adkv_params *vp, void *v_tail, int B, int H, int T, int D,
                   int n_super_cap, int bits, float scale_min, float scale_max, void *stream)
{
    if (!k_cache || !k_new || !k_tail || !params_ok(kp) || !v_cache || !v_new || !v_tail || !params_ok(vp))
        return ADKV_E_NULL;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, T + 1)) return rc;
    if (B * H == 0) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(k_cache, k_new, kp, k_tail);
    b.t[1] = enc_tensor(v_cache, v_new, vp, v_tail);
    return launch_append(b, 2, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream);
}

int adkv_encode_kv_layers(const adkv_layer_kv *layers, int n_layers, int B, int H, int T, int D, int n_super_cap,
                          int bits, int t_start, float scale_min, float scale_max, void *stream)
{
    if (!layers) return ADKV_E_NULL;
    if (n_layers < 0 || t_start < 0) return ADKV_E_SHAPE;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, t_start + T)) return rc;
    for (int l = 0; l < n_layers; ++l) {
        if (int rc = encode_check(layers[l].k_cache, layers[l].k, &layers[l].kp, layers[l].k_tail, T, t_start)) return rc;
        if (int rc = encode_check(layers[l].v_cache, layers[l].v, &layers[l].vp, layers[l].v_tail, T, t_start)) return rc;
    }
    if (B * H == 0 || T == 0) return 0;
    for (int l0 = 0; l0 < n_layers; l0 += kEncMaxTensors / 2) {
        const int n = min(kEncMaxTensors / 2, n_layers - l0);
        EncBatch b{};
        for (int l = 0; l < n; ++l) {
            const adkv_layer_kv &L = layers[l0 + l];
            b.t[2 * l] = enc_tensor(L.k_cache, L.k, &L.kp, L.k_tail);
            b.t[2 * l + 1] = enc_tensor(L.v_cache, L.v, &L.vp, L.v_tail);
        }
        if (int rc = launch_encode(b, 2 * n, B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max, stream)) return rc;
    }
    return 0;
}

int adkv_append_kv_layers(const adkv_layer_kv *layers, int n_layers, int B, int H, int T, int D, int n_super_cap,
                          int bits, float scale_min, float scale_max, void *stream)
{
    if (!layers) return ADKV_E_NULL;
    if (n_layers < 0) return ADKV_E_SHAPE;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, T + 1)) return rc;
    for (int l = 0; l < n_layers; ++l) {
        const adkv_layer_kv &L = layers[l];
        if (!L.k_cache || !L.k || !L.k_tail || !params_ok(&L.kp) || !L.v_cache || !L.v || !L.v_tail || !params_ok(&L.vp))
            return ADKV_E_NULL;
    }
    if (B * H == 0) return 0;
    for (int l0 = 0; l0 < n_layers; l0 += kAppendMaxTensors / 2) {
        const int n = min(kAppendMaxTensors / 2, n_layers - l0);
        AppendBatch b{};
        for (int l = 0; l < n; ++l) {
            const adkv_layer_kv &L = layers[l0 + l];
            b.t[2 * l] = enc_tensor(L.k_cache, L.k, &L.kp, L.k_tail);
            b.t[2 * l + 1] = enc_tensor(L.v_cache, L.v, &L.vp, L.v_tail);
        }
        if (int rc = launch_append(b, 2 * n, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream)) return rc;
    }
    return 0;
}

int adkv_encode_kv_ckpt(void *k_cache, const void *k, const adkv_params *kp, void *k_tail, void *k_ckpt,
                        void *v_cache, const void *v, const adkv_params *vp, void *v_tail, void *v_ckpt,
                        int interval, int n_ckpt_cap, int B, int H, int T, int D, int n_super_cap, int bits,
                        int t_start, float scale_min, float scale_max, void *stream)
{
    if (t_start < 0) return ADKV_E_SHAPE;
    if (int rc = encode_check(k_cache, k, kp, k_tail, T, t_start)) return rc;
    if (int rc = encode_check(v_cache, v, vp, v_tail, T, t_start)) return rc;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, t_start + T)) return rc;
    if (int rc = ckpt_check(k_ckpt, v_ckpt, interval, n_ckpt_cap, t_start + T)) return rc;
    if (B * H == 0 || (T == 0 && !((k_tail || v_tail) && t_start == 0))) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(k_cache, k, kp, k_tail, k_ckpt);
    b.t[1] = enc_tensor(v_cache, v, vp, v_tail, v_ckpt);
    return launch_encode(b, 2, B, H, T, D, n_super_cap, bits, t_start, scale_min, scale_max, stream,
                         CkptSpec{interval, n_ckpt_cap, D});
}

int adkv_append_kv_ckpt(void *k_cache, const void *k_new, const adkv_params *kp, void *k_tail, void *k_ckpt,
                        void *v_cache, const void *v_new, const adkv_params *vp, void *v_tail, void *v_ckpt,
                        int interval, int n_ckpt_cap, int B, int H, int T, int D, int n_super_cap, int bits,
                        float scale_min, float scale_max, void *stream)
{
    if (!k_cache || !k_new || !k_tail || !params_ok(kp) || !v_cache || !v_new || !v_tail || !params_ok(vp))
        return ADKV_E_NULL;
    if (int rc = check_common(B, H, H, T, D, n_super_cap, bits, T + 1)) return rc;
    if (int rc = ckpt_check(k_ckpt, v_ckpt, interval, n_ckpt_cap, T + 1)) return rc;
    if (B * H == 0) return 0;
    EncBatch b{};
    b.t[0] = enc_tensor(k_cache, k_new, kp, k_tail, k_ckpt);
    b.t[1] = enc_tensor(v_cache, v_new, vp, v_tail, v_ckpt);
    return launch_append(b, 2, B, H, T, D, n_super_cap, bits, scale_min, scale_max, stream,
                         CkptSpec{interval, n_ckpt_cap, D});
}

}  // extern "C"
