// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point.
//
// Fused decode step for launches with few (batch, kv head) streams, next to tail states: the token axis of every stream
// is cut into eight segments that run side by side in ONE CTA, a K and a V warp each.  Reached through
// adkv_decode_attn and adkv_decode_attn_varlen.
//
// What bounds a step with few streams is one warp's dependent instruction stream: a K/V pair walks its stream at about
// 100 cycles a token whatever the rest of the SM does, and splitting the channels of a head over more warps repeats the
// per-token overhead in each.  The token axis looks serial, but the scale recurrence s' = clamp(s * (tc + beta*|q|)) is a
// running product of factors that depend on the codes alone, and the zero point a running sum, so:
//
//  1. every warp forms the product F of the factors of its segment and the extremes of its running product (about half
//     the arithmetic of a scan, no clamps);
//  2. the states at the segment starts follow from the products of the segments before.  If some segment, from the state
//     it really starts with, may have met a clamp (the extremes, widened by the worst case of four tokens, reach a
//     bound), what becomes of the two bounds is formed for all segments of that tensor as well (scale_map), still side by
//     side;
//  3. the scans run as in adkv_decode.cuh, with zero points relative to the segment start.  For K that shifts every logit
//     of a segment by one number, sum_c q_c * zp_c(start), for V it leaves out (sum of weights) * zp(start): both are put
//     back
//  4. when the partial softmax results of the segments are merged in shared memory.
//
// Only the appended token needs the encoder's exact state, and that comes from the tail.  Against 64 bits a logit is off
// by 0.75 to 0.83 times what it is off after one scan over the whole stream (root mean square of 3840 to 9600 logits each,
// 1500 to 4096 tokens, 4 and 2 bits), because the segments start from less rounding.
//
// Steps 1 and 2 add a third to the work, two thirds where a clamp is met, so this pays only while a stream per warp pair
// leaves schedulers idle, and where the tensor-core kernel (adkv_tensor.cu) is no faster: see use_segments in adkv_fused.cu.
#include "adkv_host.h"

#include "adkv_softmax.cuh"

namespace adkv {

constexpr int NS = 8;             // segments per stream
constexpr int kSegStages = 2;     // bulk-copy ring depth per warp
// Tokens per tile (TOK), 64 as in adkv_fused.cu, but 32 where 64 tokens of 16 warps do not fit the shared memory, and for segments
// of one such tile, where V would wait until K is through: 300 tokens, device time on a B200, 64 -> 32: 4-bit, two heads, 8
// streams 16.6 -> 15.5 us, 2-bit, 64 streams, two heads 16.8 -> 15.8 us, four heads 19.2 -> 18.7 us.  Segments have 64 tokens
// from 257 to 512 tokens of a stream; with four heads 500 tokens are back where 64 is no slower (2-bit, 128 streams 24.1 -> 25.1 us).
template <int BITS, int G>
constexpr bool kSegLongTiles = !(BITS == 4 && G == 4);
template <int G>
constexpr int kSegShortTokens = G == 4 ? 384 : 512;
constexpr int kPartFloats = 4 + kD;   // per (segment, head): maximum (log2 units), denominator, 2 pad, kD sums

template <int BITS, int G, int TOK>
struct SegShared {
    alignas(128) uint8_t buf[2][NS][kSegStages * Tile<BITS, TOK>::BYTES];
    alignas(16) float red[NS][G * 8 * kRedRow];
    alignas(16) float2 wts[NS][G * TOK];
    union {
        alignas(16) float comp[2][NS][3][kD];     // steps 1 and 2: product, smallest and largest running product
        alignas(16) float part[NS][G][kPartFloats];   // steps 3 and 4
    };
    alignas(16) float init[2][NS][2][kD];         // zero point (relative) and scale at the segment starts
    alignas(16) float zp_end[NS][kD];             // V: zero points after the segment, relative to its start
    alignas(16) float self_x[kD];                        // V: dequantised appended token
    float z_end[NS][G];                           // K: sum_c q_c * zp_c after the segment, relative
    float self_logit[G];
    int clamps[2];                                       // step 2: a segment of K / of V may have met a clamp
    FusedShared<G, 1, TOK> fs[NS];
    uint64_t bar[2][NS][kSegStages];
};

template <int G, int TOK>
struct SegSink : RingSink<G, 1, TOK> {
    float *z_end;
    bool done;
    __device__ __forceinline__ void end_state(const Chan (&ch)[4], const float (&qv)[G][4], int lane)
    {
        done = true;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float z = warp_sum(fmaf(qv[g][3], ch[3].zp, fmaf(qv[g][2], ch[2].zp, fmaf(qv[g][1], ch[1].zp, qv[g][0] * ch[0].zp))));
            if (lane == 0) z_end[g] = z;
        }
    }
};

template <int G, int TOK>
struct SegSrc : SoftmaxSrc<G, 1, false, TOK> {
    float *part;       // [G][kPartFloats] of this segment
    float *zp_end;
    bool done;
    __device__ __forceinline__ void end_state(const Chan (&ch)[4], int c0)
    {
        done = true;
        *reinterpret_cast<float4 *>(zp_end + c0) = make_float4(ch[0].zp, ch[1].zp, ch[2].zp, ch[3].zp);
    }
    __device__ __forceinline__ void put(int c0, int g, float m, float l, float4 acc) const
    {
        if (c0 == 0) {
            part[g * kPartFloats] = m;
            part[g * kPartFloats + 1] = l;
        }
        *reinterpret_cast<float4 *>(part + g * kPartFloats + 4 + c0) = acc;
    }
    __device__ __forceinline__ void store(const VArgs &, int, int, int c0, const float (&acc)[G][4]) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g)
            put(c0, g, this->m[g], this->denominator(g), make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]));
    }
    // a bounded wait gave up: the merged output of these heads becomes NaN
    __device__ __forceinline__ void give_up(int c0) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) put(c0, g, -INFINITY, __int_as_float(0x7fc00000), make_float4(0.f, 0.f, 0.f, 0.f));
    }
};

// Scales of four channels and what advances them (contracted constants: ch[].tc = 1 - beta * target).
struct ScaleConst {
    f32x2 beta[2], tc[2];
};

// Interval that the scales at every fourth token (start and end included) have to lie in for the unclamped trajectory
// between them to stay inside the bounds, for all four channels of a lane: at most four updates after one of them and at
// most four before the next, whichever says more (for 2-bit codes the latter: a scale falls by 2.5 % a token at most but
// grows by 7.5 %, so the upper bound is 0.90 * smax instead of 0.75 * smax).
__device__ __forceinline__ SafeRange block_range(const float (&beta)[4], const float (&target)[4], int bias, float smin, float smax)
{
    SafeRange r{0.f, INFINITY};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float g0 = 1.f - beta[c] * target[c], g1 = g0 + beta[c] * float(bias);
        const float gmn = fminf(fminf(g0, g1), 1.f), gmx = fmaxf(fmaxf(g0, g1), 1.f);
        const float pmn = gmn * gmn * gmn * gmn, pmx = gmx * gmx * gmx * gmx;
        r.lo = fmaxf(r.lo, gmn > 0.f ? fmaxf(smin, kEps) * fminf(__fdividef(1.f, pmn), pmx) * (1.f + 2e-5f) : INFINITY);
        r.hi = fminf(r.hi, smax * fmaxf(__fdividef(1.f, pmx), pmn) * (1.f - 2e-5f));
    }
    if (!(r.lo <= r.hi)) { r.lo = INFINITY; r.hi = 0.f; }
    return r;
}

// Step 1: product of the factors of `n_words` words of a stream and the extremes of the running product at every
// fourth token (1 at the start included).  src: this lane's vector of the first word.
//
// The state that a segment starts with must not carry more rounding than a scan from the start of the stream would have
// brought to it, so two factors at a time are multiplied without rounding, as a sum of two numbers, and the running
// product is rounded every second token.  (A rounded product of factors will not do: factors take a handful of values, so
// its rounding repeats and adds up, 7e-5 over 8192 tokens instead of 8e-6.)
template <int BITS>
__device__ __forceinline__ void scale_product(const uint4 *src, int n_words, const ScaleConst &sc, float (&F)[4],
                                              float (&mn)[4], float (&mx)[4])
{
    constexpr int kAhead = 4;
    FieldConsts<BITS> fc;
    fc.init();
    const f32x2 minus = pk2(-1.f, -1.f);
    f32x2 f2[2] = {pk2(1.f, 1.f), pk2(1.f, 1.f)};
#pragma unroll
    for (int c = 0; c < 4; ++c) mn[c] = mx[c] = 1.f;
    uint4 w[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) w[i] = src[min(i, n_words - 1) * (kD / 4)];
#pragma unroll 1
    for (int wd = 0; wd < n_words; wd += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            uint32_t grp[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
            w[i] = src[min(wd + kAhead + i, n_words - 1) * (kD / 4)];
            if (wd + i < n_words) {
#pragma unroll 1
                for (int blk = 0; blk < Codec<BITS>::TPW / 4; ++blk) {
                    static_for<2>([&](auto hc) {
                        constexpr int k = 2 * decltype(hc)::value;
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const f32x2 a = fma2(sc.beta[p], abs2(fc.template code2<k>(grp[2 * p], grp[2 * p + 1])), sc.tc[p]);
                            const f32x2 b = fma2(sc.beta[p], abs2(fc.template code2<k + 1>(grp[2 * p], grp[2 * p + 1])), sc.tc[p]);
                            const f32x2 ab = mul2(a, b), rest = fma2(a, b, mul2(ab, minus));   // a * b == ab + rest
                            f2[p] = fma2(f2[p], ab, mul2(f2[p], rest));
                        }
                    });
                    upk2(f2[0], F[0], F[1]);
                    upk2(f2[1], F[2], F[3]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        mn[c] = fminf(mn[c], F[c]);
                        mx[c] = fmaxf(mx[c], F[c]);
                        grp[c] >>= 4 * BITS;
                    }
                }
            }
        }
    }
    upk2(f2[0], F[0], F[1]);
    upk2(f2[1], F[2], F[3]);
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (F[c] != F[c]) F[c] = mx[c] = INFINITY;   // past the range of fp32 the sum above is infinity minus infinity
}

// Step 2 where a clamp may have acted.  The composition of the clamped steps is again a clamped scaling: a state x inside
// the bounds ends as clamp(F * x, lo, hi), where F is the product of the factors (step 1) and lo and hi are what the two
// bounds themselves end as.  (A factor below zero sends every state to the same bound: then lo == hi.)  lo, hi: in the
// states to start from -- the bounds, or twice the state itself where it is known and may lie outside them.  ends: [2].
template <int BITS>
__device__ __noinline__ void scale_map(const uint4 *src, int n_words, const ScaleConst &sc, float smin, float smax, float4 lo4,
                                       float4 hi4, float4 *ends)
{
    FieldConsts<BITS> fc;
    fc.init();
    f32x2 lo[2] = {pk2(lo4.x, lo4.y), pk2(lo4.z, lo4.w)}, hi[2] = {pk2(hi4.x, hi4.y), pk2(hi4.z, hi4.w)};
    const auto clamped = [&](f32x2 v) {
        float a, b;
        upk2(v, a, b);
        return pk2(fminf(fmaxf(a, smin), smax), fminf(fmaxf(b, smin), smax));
    };
    uint4 w = *src;
#pragma unroll 1
    for (int wd = 0; wd < n_words; ++wd) {
        const uint4 next = src[min(wd + 1, n_words - 1) * (kD / 4)];
        uint32_t grp[4] = {w.x, w.y, w.z, w.w};
#pragma unroll 1
        for (int blk = 0; blk < Codec<BITS>::TPW / 4; ++blk) {
            static_for<4>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const f32x2 f = fma2(sc.beta[p], abs2(fc.template code2<k>(grp[2 * p], grp[2 * p + 1])), sc.tc[p]);
                    lo[p] = clamped(mul2(lo[p], f));
                    hi[p] = clamped(mul2(hi[p], f));
                }
            });
#pragma unroll
            for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
        }
        w = next;
    }
    *reinterpret_cast<ulonglong2 *>(ends) = make_ulonglong2(lo[0], lo[1]);
    *reinterpret_cast<ulonglong2 *>(ends + kD / 4) = make_ulonglong2(hi[0], hi[1]);
}

template <int BITS, int G, int TOK>
__global__ void __launch_bounds__(64 * NS)
    decode_attn_segments_kernel(KArgs ka, VArgs va, const float *__restrict__ mask, long long mask_stride_b, float scaling,
                                const int *__restrict__ seq_lens)
{
    extern __shared__ uint8_t smem_raw[];
    SegShared<BITS, G, TOK> &sh = *reinterpret_cast<SegShared<BITS, G, TOK> *>(smem_raw);
    using C = Codec<BITS>;
    const int bh = blockIdx.x, b = bh / ka.Hkv, h = bh % ka.Hkv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Warps go to the four schedulers round robin: a pair of warps is the K and the V warp of one segment, and the order
    // flips with every other pair so that each scheduler holds as many K as V warps.
    const int seg = warp >> 1, role = (warp ^ (warp >> 2)) & 1;
    if (seq_lens) {   // as in decode_attn_kernel
        const int T = seq_lens[b];
        if (T < 0 || T / C::TPW >= ka.n_super_cap) {
            if (threadIdx.x == 0) atomicExch(&g_status, kStatCapacity);
            return;
        }
        ka.T = T;
        va.T = T;
    }
    if (threadIdx.x < 2) sh.clamps[threadIdx.x] = 0;
    if (threadIdx.x < NS) {
        for (int r = 0; r < 2; ++r)
            for (int i = 0; i < kSegStages; ++i) mbar_init(&sh.bar[r][threadIdx.x][i], 1);
        sh.fs[threadIdx.x].init_barriers(1);
        for (int g = 0; g < G; ++g) sh.z_end[threadIdx.x][g] = 0.f;
        mbar_init_fence();
    }
    const int T = ka.T, n_tiles = (T + kTileTok - 1) / kTileTok;
    const int per_seg = (n_tiles + NS - 1) / NS * kTileTok;
    const int t_begin = min(seg * per_seg, T), t_end = min(t_begin + per_seg, T);
    const ParamPtrs &p = role ? va.p : ka.p;
    const int c0 = 4 * lane;
    const size_t poff = size_t(h) * kD + c0;
    const uint4 *words = reinterpret_cast<const uint4 *>((role ? va.cache : ka.cache) +
                                                         (size_t(bh) * ka.n_super_cap + t_begin / C::TPW) * kD * 4) + lane;

    // 1. products of all segments that another one follows (those are whole tiles)
    ScaleConst sc;
    SafeRange range;
    float s[4] = {};
    const bool followed = t_end < T;
    if (per_seg < T) {
        Chan ch[4];
        load_chan4<BITS, true>(ch, range, p, poff, ka.smin, ka.smax);
        float be[4], tg[4], tc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            be[c] = ch[c].beta;
            tg[c] = ch[c].tc;
            tc[c] = fmaf(-be[c], tg[c], 1.0f);
            s[c] = ch[c].s;
        }
        range = block_range(be, tg, C::BIAS, ka.smin, ka.smax);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            sc.beta[q] = pk2(be[2 * q], be[2 * q + 1]);
            sc.tc[q] = pk2(tc[2 * q], tc[2 * q + 1]);
        }
    }
    if (followed) {
        float F[4], mn[4], mx[4];
        scale_product<BITS>(words, per_seg / C::TPW, sc, F, mn, mx);
        *reinterpret_cast<float4 *>(&sh.comp[role][seg][0][c0]) = make_float4(F[0], F[1], F[2], F[3]);
        *reinterpret_cast<float4 *>(&sh.comp[role][seg][1][c0]) = make_float4(mn[0], mn[1], mn[2], mn[3]);
        *reinterpret_cast<float4 *>(&sh.comp[role][seg][2][c0]) = make_float4(mx[0], mx[1], mx[2], mx[3]);
    }
    __syncthreads();

    // 2. scale at the start of this warp's segment
    const float4 start = make_float4(s[0], s[1], s[2], s[3]);
    const bool empty = seg > 0 && t_begin >= T;
    bool proven = true;      // no segment up to this one can have met a clamp, in any channel of the warp
    for (int i = 0; i < seg && proven && !empty; ++i) {
        const float4 F = *reinterpret_cast<const float4 *>(&sh.comp[role][i][0][c0]);
        const float4 mn = *reinterpret_cast<const float4 *>(&sh.comp[role][i][1][c0]);
        const float4 mx = *reinterpret_cast<const float4 *>(&sh.comp[role][i][2][c0]);
        const bool ok = s[0] * mn.x >= range.lo && s[1] * mn.y >= range.lo && s[2] * mn.z >= range.lo && s[3] * mn.w >= range.lo &&
                        s[0] * mx.x <= range.hi && s[1] * mx.y <= range.hi && s[2] * mx.z <= range.hi && s[3] * mx.w <= range.hi;
        proven = __all_sync(kFull, ok);
        s[0] *= F.x; s[1] *= F.y; s[2] *= F.z; s[3] *= F.w;
    }
    if (!proven && lane == 0) sh.clamps[role] = 1;
    __syncthreads();
    if (sh.clamps[0] | sh.clamps[1]) {
        const bool redo = sh.clamps[role] != 0;
        const float4 lo = seg ? make_float4(ka.smin, ka.smin, ka.smin, ka.smin) : start;
        const float4 hi = seg ? make_float4(ka.smax, ka.smax, ka.smax, ka.smax) : start;
        if (followed && redo)
            scale_map<BITS>(words, per_seg / C::TPW, sc, ka.smin, ka.smax, lo, hi,
                            reinterpret_cast<float4 *>(&sh.comp[role][seg][1][c0]));
        __syncthreads();
        if (redo) { s[0] = start.x; s[1] = start.y; s[2] = start.z; s[3] = start.w; }
        for (int i = 0; i < seg && redo && !empty; ++i) {
            const float4 F = *reinterpret_cast<const float4 *>(&sh.comp[role][i][0][c0]);
            const float4 l = *reinterpret_cast<const float4 *>(&sh.comp[role][i][1][c0]);
            const float4 u = *reinterpret_cast<const float4 *>(&sh.comp[role][i][2][c0]);
            s[0] = fminf(fmaxf(F.x * s[0], l.x), u.x);
            s[1] = fminf(fmaxf(F.y * s[1], l.y), u.y);
            s[2] = fminf(fmaxf(F.z * s[2], l.z), u.z);
            s[3] = fminf(fmaxf(F.w * s[3], l.w), u.w);
        }
        __syncthreads();
    }

    // 3. the scans; a lane reads back only the state that it wrote itself
    *reinterpret_cast<float4 *>(&sh.init[role][seg][0][c0]) = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4 *>(&sh.init[role][seg][1][c0]) = make_float4(s[0], s[1], s[2], s[3]);
    const Seg sg{t_begin, t_end, false, seg ? &sh.init[role][seg][0][0] : nullptr, nullptr, 0};
    const float *mask_row = mask ? mask + size_t(b) * mask_stride_b : nullptr;
    const float scale2 = scaling * 1.4426950408889634f;
    const auto append = [&](const ParamPtrs &pp, float *tail, bool keep, const __half *x_new, uint8_t *cache, float (&xh)[4]) {
        append_from_tail<BITS>(pp, poff, tail + size_t(bh) * 2 * kD, keep, x_new + size_t(bh) * kD + c0,
                               reinterpret_cast<uint4 *>(cache + (size_t(bh) * ka.n_super_cap + T / C::TPW) * kD * 4) + lane,
                               T, ka.smin, ka.smax, nullptr, c0, xh);
    };
    // The appended token goes into the word behind the last cached one: only the warps that read that word may write it.
    const bool last = t_end == T && (seg == 0 || t_begin < T);
    if (role == 0) {
        SegSink<G, TOK> sink;
        sink.sh = &sh.fs[seg];
        sink.slot = 0;
        sink.sl = 0;
        sink.z_end = sh.z_end[seg];
        sink.done = false;
        k_warp<BITS, G, kArithFma, SegSink<G, TOK>, kSegStages, false, false, 8, TOK>(ka, sg, b, h, lane, sh.buf[0][seg], sh.bar[0][seg], sh.red[seg], sink);
        if (last && sink.done) {
            float xh[4];
            append(ka.p, ka.tail, ka.tail_keep, ka.x_new, ka.cache, xh);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float qv[4], x = 0.f;
                load_half4(qv, ka.q + (size_t(b) * ka.Hq + size_t(h) * G + g) * kD + c0);
#pragma unroll
                for (int c = 0; c < 4; ++c) x = fmaf(qv[c], xh[c], x);
                x = warp_sum(x);
                if (lane == 0) sh.self_logit[g] = x;
            }
        }
    } else {
        SegSrc<G, TOK> src;
        src.sh = &sh.fs[seg];
        src.wts = sh.wts[seg];
        src.mask = mask_row;
        src.scale2 = scale2;
        src.n_tiles = (t_end - t_begin + TOK - 1) / TOK;
        src.t_begin = t_begin;
        src.part = &sh.part[seg][0][0];
        src.zp_end = sh.zp_end[seg];
        src.done = false;
        src.init();
        v_warp<BITS, G, kArithFma, SegSrc<G, TOK>, kSegStages, false, false, TOK>(va, sg, b, h, lane, sh.buf[1][seg], sh.bar[1][seg], sh.wts[seg], src);
        if (last && src.done) {
            float xh[4];
            append(va.p, va.tail, va.tail_keep, va.x_new, va.cache, xh);
            *reinterpret_cast<float4 *>(&sh.self_x[c0]) = make_float4(xh[0], xh[1], xh[2], xh[3]);
        }
    }
    __syncthreads();

    // 4. merge: segment maxima shifted by the zero points K left out, sums completed with those V left out
    const float mk = mask_row ? mask_row[T] * 1.4426950408889634f : 0.f;
    for (int i = threadIdx.x; i < G * kD; i += 64 * NS) {
        const int g = i / kD, c = i % kD;
        float m[NS], z = 0.f;
        const float v = fmaf(sh.self_logit[g], scale2, mk);
        float M = v;
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            m[j] = sh.part[j][g][0];
            if (m[j] != -INFINITY) m[j] = fmaf(z, scale2, m[j]);
            z += sh.z_end[j][g];
            M = fmaxf(M, m[j]);
        }
        const bool dead = M == -INFINITY;
        const float w_self = dead ? 0.f : exp2f(v - M);
        float L = w_self, A = w_self * sh.self_x[c], zp = 0.f;
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            const float w = m[j] == -INFINITY ? 0.f : exp2f(m[j] - M);
            const float l = sh.part[j][g][1];
            L = fmaf(l, w, L);
            A = fmaf(fmaf(l, zp, sh.part[j][g][4 + c]), w, A);
            zp += sh.zp_end[j][c];
        }
        va.out[(size_t(b) * ka.Hq + size_t(h) * G + g) * kD + c] = __float2half_rn(A / L);
    }
}

}  // namespace adkv

using namespace adkv;

ADKV_DEFINE_TU_STATUS(adkv_tu_status_segments)

template <int BITS, int G, int TOK>
static int launch_segments(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling, int B,
                           const int *seq_lens, cudaStream_t s)
{
    constexpr int bytes = int(sizeof(SegShared<BITS, G, TOK>));
    static_assert(bytes <= 227 * 1024, "shared memory of one CTA");
    // per device and process: cheap enough (a host-side call) to be made before every launch
    if (cudaFuncSetAttribute(decode_attn_segments_kernel<BITS, G, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
        return launch_status();
    decode_attn_segments_kernel<BITS, G, TOK><<<B * ka.Hkv, 64 * NS, bytes, s>>>(ka, va, mask, mask_stride_b, scaling, seq_lens);
    return launch_status();
}

// Arguments checked by the caller (head dim 128, fp32 arithmetic, contracted, tail states present, Hq / Hkv at most 4).
// max_tokens: as in use_segments (adkv_fused.cu).
ADKV_HIDDEN int adkv_segments_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b,
                                          float scaling, int B, int max_tokens, int bits, const int *seq_lens, cudaStream_t s)
{
    switch (bits * 16 + ka.Hq / ka.Hkv) {
#define ADKV_SEG_CASE(BITS_, G_)                                                                                            \
    case BITS_ * 16 + G_:                                                                                                   \
        if constexpr (kSegLongTiles<BITS_, G_>)                                                                             \
            if (max_tokens > kSegShortTokens<G_>)                                                                           \
                return launch_segments<BITS_, G_, 64>(ka, va, mask, mask_stride_b, scaling, B, seq_lens, s);                \
        return launch_segments<BITS_, G_, 32>(ka, va, mask, mask_stride_b, scaling, B, seq_lens, s);
        ADKV_SEG_CASE(4, 1) ADKV_SEG_CASE(4, 2) ADKV_SEG_CASE(4, 4)
        ADKV_SEG_CASE(2, 1) ADKV_SEG_CASE(2, 2) ADKV_SEG_CASE(2, 4)
#undef ADKV_SEG_CASE
    default: return ADKV_E_SHAPE;
    }
}
