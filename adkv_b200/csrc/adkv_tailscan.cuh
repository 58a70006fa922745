// K scan of the decode step next to a persisted tail state (contracted arithmetic, head dim 128, one query head per KV
// head).
//
// The tail supplies the state the appended token is quantised with, so a replay only has to feed the two attention
// sums.  What bounds it is instruction issue: a packed fp32 instruction holds the issue port for two cycles, and the
// contracted recurrence as written (adkv_decode.cuh) needs seven of them per channel pair and token.  Two identities
// leave 5.25:
//
//  * Scale.  s' = s * (tc + beta*|q|) with tc = 1 - beta*target.  With s = tc^k * u inside a block of four tokens
//    (k = 0..3), u' = u + (beta/tc) * |q*u|: one multiply-add on the product q*u that the value needs anyway.  The
//    powers tc^k are folded into the query; once per block u is scaled
//    back by tc^4.
//  * K.  The logit needs the zero points only as z_t = sum_c q_c * zp_c(t), a running sum over tokens like zp itself:
//    each lane carries its share of z in ONE register pair instead of a zero point per channel.
//
// Clamp and eps guard are left out where eight worst-case updates cannot reach a bound, else where four cannot (on the
// benchmark data the eight-token test fails for 7 % of the 4-bit chunks and 16 % of the 2-bit ones, the four-token test
// for none); only what is left runs guarded.
//
// Used inside the segments of adkv_segments.cu, where it is as exact against 64 bits as the recurrence as written.  Over a
// whole stream it is not (2.66e-4 instead of 2.47e-4 at 8192 tokens, 2-bit), so launches with one warp pair per stream
// keep decode_attn_kernel although this scan would take 1.33 ms instead of 1.47 ms at batch 128 x 4096 tokens.
#pragma once
#include "adkv_softmax.cuh"

namespace adkv {

constexpr int kTailStages = 4;                        // bulk-copy ring depth per warp
constexpr int kDriftTiles = 4;                        // tiles between two corrections of the scales (TailChan::drift)
constexpr int kRedUnits = 8;                          // (head, block of 4 tokens) pairs reduced per pass
constexpr int kRedFloats = kRedUnits * 32 * 4;        // per K warp

// ------------------------------------------------------------------------------------------ constants of a lane

// FieldConsts with the subtrahends kept as packed pairs.
template <int BITS>
struct PairFields {
    uint32_t e[4];
    f32x2 negc[4];
    __device__ __forceinline__ void init()
    {
        FieldConsts<BITS> f;
        f.init();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            e[k] = f.e[k];
            asm volatile("mov.b64 %0, {%1, %1};" : "=l"(negc[k]) : "r"(f.negc[k]));
        }
    }
    template <int K>
    __device__ __forceinline__ f32x2 code2(uint32_t ga, uint32_t gb) const
    {
        uint32_t a, b;
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(a) : "r"(ga), "n"(Codec<BITS>::FIELD << (BITS * K)), "r"(e[K]));
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(b) : "r"(gb), "n"(Codec<BITS>::FIELD << (BITS * K)), "r"(e[K]));
        f32x2 f;
        asm("mov.b64 %0, {%1, %2};" : "=l"(f) : "r"(a), "r"(b));
        return add2(f, negc[K]);
    }
};

// What a scan holds on its lane's four consecutive channels, as two pairs.
struct TailChan {
    f32x2 s[2], zp[2];       // state
    f32x2 alpha[2];
    f32x2 bp[2];             // beta / tc
    f32x2 e[4][2];           // tc^1 .. tc^4
    uint32_t drift[2];       // relative correction of the scale per kDriftTiles tiles, two bfloat16 per pair
    SafeRange safe, safe4;   // intervals for the next 8 and the next 4 tokens
};

// The factors are formed in double and rounded once.  The rounding of tc^4 and of beta / tc is an error that every
// block would repeat -- up to 3e-8 a block, 2.4e-4 after 32768 tokens --, so what it amounts to over kDriftTiles tiles
// (for beta / tc: at the mean code magnitude, which the recurrence keeps at `target`) is put right at that distance.
// slow: [2][32] float4 of this warp, offset by the lane: beta and tc for the guarded bodies.
template <int BITS>
__device__ __forceinline__ void load_tail_chan(TailChan &t, const ParamPtrs &p, size_t off, const float *init, int c0,
                                               float smin, float smax, float4 *slow)
{
    Chan ch[4];
    load_chan4<BITS, true>(ch, t.safe, p, off, smin, smax);   // canonical constants: ch[].tc is the target
    load_init_state(ch, init, c0, kD);
    float e[4][4], bp[4], drift[4], be[4], tg[4];
    bool usable = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        be[i] = ch[i].beta;
        tg[i] = ch[i].tc;
        const double t1 = 1.0 - double(be[i]) * double(tg[i]), t2 = t1 * t1;
        e[0][i] = float(t1);
        e[1][i] = float(t2);
        e[2][i] = float(t2 * t1);
        e[3][i] = float(t2 * t2);
        // outside this interval (also NaN) the four-token form is not used: every chunk takes the guarded body
        const bool in = e[0][i] >= 0.125f && e[0][i] <= 8.f;
        usable = usable && in;
        bp[i] = in ? __fdiv_rn(be[i], e[0][i]) : 0.f;
        drift[i] = in ? float(kDriftTiles * kTileTok / 4) * __fdividef(float(t2 * t2 - double(e[3][i])), e[3][i]) +
                            float(kDriftTiles * kTileTok) * tg[i] * float(double(be[i]) - double(bp[i]) * t1)
                      : 0.f;
    }
    t.safe4.template init<BITS, 4, 4>(be, tg, smin, smax);
    if (!usable) { t.safe.lo = t.safe4.lo = INFINITY; t.safe.hi = t.safe4.hi = 0.f; }
    slow[0] = make_float4(be[0], be[1], be[2], be[3]);
    slow[32] = make_float4(fmaf(-be[0], tg[0], 1.0f), fmaf(-be[1], tg[1], 1.0f), fmaf(-be[2], tg[2], 1.0f),
                           fmaf(-be[3], tg[3], 1.0f));
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        t.s[q] = pk2(ch[2 * q].s, ch[2 * q + 1].s);
        t.zp[q] = pk2(ch[2 * q].zp, ch[2 * q + 1].zp);
        t.alpha[q] = pk2(ch[2 * q].alpha, ch[2 * q + 1].alpha);
        t.bp[q] = pk2(bp[2 * q], bp[2 * q + 1]);
        t.drift[q] = __byte_perm(__float_as_uint(drift[2 * q]), __float_as_uint(drift[2 * q + 1]), 0x7632);
#pragma unroll
        for (int k = 0; k < 4; ++k) t.e[k][q] = pk2(e[k][2 * q], e[k][2 * q + 1]);
    }
}

__device__ __forceinline__ void correct_drift(f32x2 (&s)[2], const uint32_t (&drift)[2])
{
#pragma unroll
    for (int p = 0; p < 2; ++p)
        s[p] = fma2(s[p], pk2(__uint_as_float(drift[p] << 16), __uint_as_float(drift[p] & 0xffff0000u)), s[p]);
}

// warp-uniform: the next updates of any scale of the warp meet neither clamp nor guard
__device__ __forceinline__ bool tail_safe(const SafeRange &r, const f32x2 (&s)[2])
{
    float a, b, c, d;
    upk2(s[0], a, b);
    upk2(s[1], c, d);
    const float mn = fminf(fminf(fminf(a, b), c), d), mx = fmaxf(fmaxf(fmaxf(a, b), c), d);
    return __all_sync(kFull, mn >= r.lo && mx <= r.hi);
}

__device__ __forceinline__ void load_slow_consts(const float4 *slow, float (&be)[4], float (&tc)[4])
{
    const float4 a = slow[0], b = slow[32];
    be[0] = a.x; be[1] = a.y; be[2] = a.z; be[3] = a.w;
    tc[0] = b.x; tc[1] = b.y; tc[2] = b.z; tc[3] = b.w;
}

// One guarded step of a channel: returns q * max(s, eps) and advances s.
__device__ __forceinline__ float guarded_scale_step(float q, float &s, float be, float tc, float smin, float smax)
{
    const float rh = q * fmaxf(s, kEps);
    s = fminf(fmaxf(s * fmaf(be, fabsf(q), tc), smin), smax);
    return rh;
}

// Quantise the new token of this lane's channels from the tail (see append_new_token).
template <int BITS>
__device__ __forceinline__ void append_from_tail(const ParamPtrs &p, size_t poff, float *tail, bool tail_keep,
                                                 const __half *x_new, uint4 *slot, int T, float smin, float smax,
                                                 int c0, float (&xh)[4])
{
    Chan ch[4];
    SafeRange unused;
    load_chan4<BITS, true>(ch, unused, p, poff, smin, smax);
    append_new_token<BITS, kArithCanon>(ch, p, poff, tail, tail_keep, x_new, slot, T, smin, smax, nullptr, c0, kD, xh);
}

// ------------------------------------------------------------------------------------------ walking a tile

__device__ __forceinline__ void shift_words(uint4 &w, int n)
{
    w.x >>= n; w.y >>= n; w.z >>= n; w.w >>= n;
}

// Calls chunk(word, first token) for every eight tokens of a full tile, two chunks per trip: half the loop's instructions,
// and the bodies still stay in the instruction cache.
template <int BITS, class Chunk>
__device__ __forceinline__ void walk_full_tile(const uint4 *tile, Chunk &&chunk)
{
#pragma unroll 1
    for (int tok = 0; tok < kTileTok; tok += 16) {
        uint4 w = *tile, w2;
        tile += kD / 4;
        if (BITS == 4) {
            w2 = *tile;
            tile += kD / 4;
        }
        chunk(w, tok);
        if (BITS == 2) {
            w2 = w;
            shift_words(w2, 16);
        }
        chunk(w2, tok + 8);
    }
}

// Any tile: body(word, first token, valid tokens) per eight tokens.
template <int BITS, class Body>
__device__ __forceinline__ void walk_tile(const uint4 *tile, int ntok, Body &&body)
{
#pragma unroll 1
    for (int tok = 0; tok < ntok; tok += 8) {
        uint4 w = tile[(tok / Codec<BITS>::TPW) * (kD / 4)];
        if (BITS == 2 && (tok & 8)) shift_words(w, 16);
        body(w, tok, ntok - tok);
    }
}

// ------------------------------------------------------------------------------------------ logits of a K warp

// Sum eight units of per-lane partials over the 32 lanes.  red: [unit][lane] float4, the four tokens of a unit.
// Lane l adds the partials of source lanes 8*(l&3) .. +7 of unit l>>2 (in an order that keeps every 16-byte phase free
// of bank conflicts), then the four lanes of a unit exchange: lane l returns the sum of token l&3 of unit l>>2.
// 8 loads, 16 packed adds and 3 shuffles per 32 sums; the transpose of adkv_decode.cuh takes 8 loads, 36 adds and
// 8 shuffles, and one 4-byte store per sum and lane instead of a 16-byte store per four.
__device__ __forceinline__ float reduce_units(const float *red, int lane)
{
    __syncwarp();
    const int sub = lane & 3;
    const float4 *src = reinterpret_cast<const float4 *>(red) + (lane >> 2) * 32 + sub * 8;
    const int rot = sub + (lane & 4);
    f32x2 lo = 0ull, hi = 0ull;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(src + (i ^ rot));
        lo = i ? add2(lo, x.x) : x.x;
        hi = i ? add2(hi, x.y) : x.y;
    }
    float t0, t1, t2, t3;
    upk2(lo, t0, t1);
    upk2(hi, t2, t3);
    const bool up = sub & 2, odd = sub & 1;
    float k0 = up ? t2 : t0, k1 = up ? t3 : t1;
    k0 += __shfl_xor_sync(kFull, up ? t0 : t2, 2);
    k1 += __shfl_xor_sync(kFull, up ? t1 : t3, 2);
    const float r = (odd ? k1 : k0) + __shfl_xor_sync(kFull, odd ? k0 : k1, 1);
    __syncwarp();
    return r;
}

// ------------------------------------------------------------------------------------------ K side

struct KTailState {
    f32x2 s[2];
    f32x2 z;       // this lane's share of sum_c q_c * zp_c, over the two halves of its pairs
};

// Four tokens (fields 0..3 of grp) without guards.  Q[k] = q * tc^k, A[k] = alpha * Q[k].
template <int BITS>
__device__ __forceinline__ void k_tail_block(const uint32_t (&grp)[4], const PairFields<BITS> &fc, KTailState &st,
                                             const f32x2 (&bp)[2], const f32x2 (&e4)[2], const f32x2 (&Q)[4][2],
                                             const f32x2 (&A)[4][2], float4 *red)
{
    float v[4];
    static_for<4>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        f32x2 part = st.z;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const f32x2 r = mul2(fc.template code2<k>(grp[2 * p], grp[2 * p + 1]), st.s[p]);
            part = fma2(Q[k][p], r, part);
            st.z = fma2(A[k][p], r, st.z);
            st.s[p] = fma2(bp[p], abs2(r), st.s[p]);
        }
        float lo, hi;
        upk2(part, lo, hi);
        v[k] = lo + hi;
    });
    *red = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
    for (int p = 0; p < 2; ++p) st.s[p] = mul2(st.s[p], e4[p]);
}

// Up to eight tokens, `count` of them valid, as a function call (see k_chunk_guarded): chunks that fail the eight-token
// test and the ragged end of a stream.  q, qa: query and alpha * query.
template <int BITS>
__device__ __noinline__ KTailState k_tail_slow(uint4 w, KTailState st, float4 q, float4 qa, const float4 *slow, float4 *red,
                                               int count, SafeRange safe4, float smin, float smax)
{
    float be[4], tc[4];
    load_slow_consts(slow, be, tc);
    PairFields<BITS> fc;
    fc.init();
    const float qv[4] = {q.x, q.y, q.z, q.w}, qav[4] = {qa.x, qa.y, qa.z, qa.w};
#pragma unroll 1
    for (int half = 0; half < 2; ++half, count -= 4, red += 32) {
        const uint32_t grp[4] = {w.x, w.y, w.z, w.w};
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (count >= 4 && tail_safe(safe4, st.s)) {
            static_for<4>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                f32x2 part = st.z;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const f32x2 q2 = fc.template code2<k>(grp[2 * p], grp[2 * p + 1]);
                    const f32x2 r = mul2(q2, st.s[p]);
                    part = fma2(pk2(qv[2 * p], qv[2 * p + 1]), r, part);
                    st.z = fma2(pk2(qav[2 * p], qav[2 * p + 1]), r, st.z);
                    st.s[p] = mul2(st.s[p], fma2(pk2(be[2 * p], be[2 * p + 1]), abs2(q2), pk2(tc[2 * p], tc[2 * p + 1])));
                }
                float lo, hi;
                upk2(part, lo, hi);
                v[k] = lo + hi;
            });
        } else {
            float s[4], z, z1;
            upk2(st.s[0], s[0], s[1]);
            upk2(st.s[1], s[2], s[3]);
            upk2(st.z, z, z1);
            z += z1;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k < count) {
                    v[k] = z;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float rh = guarded_scale_step(code_f_rt<BITS>(grp[c], k), s[c], be[c], tc[c], smin, smax);
                        v[k] = fmaf(qv[c], rh, v[k]);
                        z = fmaf(qav[c], rh, z);
                    }
                }
            }
            st.s[0] = pk2(s[0], s[1]);
            st.s[1] = pk2(s[2], s[3]);
            st.z = pk2(z, 0.f);
        }
        *red = make_float4(v[0], v[1], v[2], v[3]);
        shift_words(w, 4 * BITS);
    }
    return st;
}

// ------------------------------------------------------------------------------------------ K warp

// Sink: RingSink<1> (begin_tile_short, put, end_tile, put_self, finish); without APPEND (a scan that does not reach the
// end of its stream) also end_share(this lane's share of sum_c q_c * zp_c after the last token, lane).
// red: kRedFloats floats, 16-byte aligned; slow: 64 float4.
template <int BITS, int STAGES, bool APPEND, class Sink>
__device__ __forceinline__ void k_tail_warp(const KArgs &a, const Seg &seg, int b, int h, int lane, uint8_t *ring_buf,
                                            uint64_t *ring_bar, float *red, float4 *slow, Sink &sink)
{
    using C = Codec<BITS>;
    const int bh = b * a.Hkv + h, c0 = 4 * lane;
    const size_t poff = size_t(h) * kD + c0;
    uint8_t *stream = a.cache + size_t(bh) * a.n_super_cap * kD * 4;
    const int n_tok = seg.t_end - seg.t_begin;
    StreamRing<BITS, STAGES> ring{ring_buf, ring_bar, stream + size_t(seg.t_begin / C::TPW) * (kD * 4),
                                  (n_tok + kTileTok - 1) / kTileTok, n_tok, kStatKWait, kD * 4};
    ring.prologue(lane);   // first: the copies of the first tiles fly while the parameters below are loaded
    PairFields<BITS> fc;
    fc.init();
    float4 *red4 = reinterpret_cast<float4 *>(red) + lane;
    slow += lane;
    TailChan t;
    load_tail_chan<BITS>(t, a.p, poff, seg.init, c0, a.smin, a.smax, slow);
    float qv[4], al[4];
    load_half4(qv, a.q + (size_t(b) * a.Hq + h) * kD + c0);
    upk2(t.alpha[0], al[0], al[1]);
    upk2(t.alpha[1], al[2], al[3]);
    const float4 qf = make_float4(qv[0], qv[1], qv[2], qv[3]);
    const float4 qaf = make_float4(qv[0] * al[0], qv[1] * al[1], qv[2] * al[2], qv[3] * al[3]);
    f32x2 Q[4][2], A[4][2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        Q[0][p] = p ? pk2(qf.z, qf.w) : pk2(qf.x, qf.y);
        A[0][p] = p ? pk2(qaf.z, qaf.w) : pk2(qaf.x, qaf.y);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            Q[k][p] = mul2(Q[0][p], t.e[k - 1][p]);
            A[k][p] = mul2(A[0][p], t.e[k - 1][p]);
        }
    }
    KTailState st;
    st.s[0] = t.s[0];
    st.s[1] = t.s[1];
    st.z = fma2(Q[0][1], t.zp[1], mul2(Q[0][0], t.zp[0]));
    const auto slow_chunk = [&](const uint4 &w, int tok, int count) {
        st = k_tail_slow<BITS>(w, st, qf, qaf, slow, red4 + (tok >> 2) * 32, count, t.safe4, a.smin, a.smax);
    };
    const auto chunk = [&](const uint4 &w, int tok) {
        if (tail_safe(t.safe, st.s)) {
            float4 *dst = red4 + (tok >> 2) * 32;
            uint32_t grp[4] = {w.x, w.y, w.z, w.w};
            k_tail_block<BITS>(grp, fc, st, t.bp, t.e[3], Q, A, dst);
#pragma unroll
            for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
            k_tail_block<BITS>(grp, fc, st, t.bp, t.e[3], Q, A, dst + 32);
        } else {
            slow_chunk(w, tok, 8);
        }
    };
    bool ok = true;
    int i = 0;
    for (; i < ring.n_tiles; ++i) {
        if (!(ok = ring.wait_short(i))) break;
        if (!(ok = sink.begin_tile_short(i))) break;
        const uint4 *tile = ring.tile(i, lane);
        const int ntok = min(kTileTok, n_tok - i * kTileTok);
        if (ntok == kTileTok) walk_full_tile<BITS>(tile, chunk);
        else walk_tile<BITS>(tile, ntok, slow_chunk);
        if ((i + 1) % kDriftTiles == 0) correct_drift(st.s, t.drift);
        sink.put(0, lane, reduce_units(red, lane));
        sink.end_tile(i, lane);
        ring.release_and_refill(i, lane);
    }
    if (!ok) {
        ring.drain(i);
        return;
    }
    if constexpr (APPEND) {
        // Append k_new as token T from the tail, then its own logit from the dequantised value.
        float xh[4];
        append_from_tail<BITS>(a.p, poff, a.tail + size_t(bh) * 2 * kD, a.tail_keep, a.x_new + size_t(bh) * kD + c0,
                               reinterpret_cast<uint4 *>(stream + size_t(a.T / C::TPW) * (kD * 4)) + lane, a.T, a.smin,
                               a.smax, c0, xh);
        if (!sink.begin_tile_short(ring.n_tiles)) return;
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) s = fmaf(qv[c], xh[c], s);
        s = warp_sum(s);
        if (lane == 0) sink.put_self(0, s);
        sink.finish(lane);
    } else {
        float lo, hi;
        upk2(st.z, lo, hi);
        sink.end_share(lo + hi, lane);
    }
}

}  // namespace adkv
