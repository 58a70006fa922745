// Scans of the decode step next to a persisted tail state (contracted arithmetic, head dim 128).
//
// The tail supplies the state the appended token is quantised with, so a replay only has to feed the two attention
// sums.  What bounds it is instruction issue: a packed fp32 instruction holds the issue port for two cycles, and the
// contracted recurrence as written (adkv_decode.cuh) needs 6 + G of them per channel pair and token with G query heads.
//
//  * Scale.  s' = s * (tc + beta*|q|) with tc = 1 - beta*target.  With s = tc^k * u inside a block of four tokens
//    (k = 0..3), u' = u + (beta/tc) * |q*u|: one multiply-add on the product q*u that the value needs anyway.  The
//    powers tc^k are folded into constants; once per block u is scaled back by tc^4.  5.25 + G instructions.
//  * K, one head.  The logit needs the zero points only as z_t = sum_c q_c * zp_c(t), a running sum over tokens like zp
//    itself: each lane carries its share of z in ONE register pair instead of a zero point per channel.  5.25.
//  * V, one head, whole stream.  zp_t = zp_T - alpha * sum_{u >= t} q_u*s_u, and zp_T is known before the scan: it is the
//    tail.  Hence sum_t w_t*zp_t = zp_T * W - alpha * sum_u P_u*q_u*s_u with the running sums P_u = w_0 + .. + w_u, which
//    the online softmax forms anyway (its denominator): no zero point is replayed, and tc^k goes into one accumulator
//    per position.  5.25.
//
// Clamp and eps guard are left out where eight worst-case updates cannot reach a bound, else where four cannot (on the
// benchmark data the eight-token test fails for 7 % of the 4-bit chunks and 16 % of the 2-bit ones, the four-token test
// for none); only what is left runs guarded.
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
                                                 float *ckpt_out, int c0, float (&xh)[4])
{
    Chan ch[4];
    SafeRange unused;
    load_chan4<BITS, true>(ch, unused, p, poff, smin, smax);
    append_new_token<BITS, kArithCanon>(ch, p, poff, tail, tail_keep, x_new, slot, T, smin, smax, ckpt_out, c0, kD, xh);
}

// Optional members of sinks and stores: what a scan without append ends in.
template <class S, int G>
__device__ __forceinline__ auto sink_end_shares(S &s, const float (&z)[G], int lane, int)
    -> decltype(s.end_shares(z, lane), void()) { s.end_shares(z, lane); }
template <class S, int G>
__device__ __forceinline__ void sink_end_shares(S &, const float (&)[G], int, long) {}
template <class S>
__device__ __forceinline__ auto store_end_zp(S &s, const f32x2 (&zp)[2], int c0, int) -> decltype(s.end_zp(zp, c0), void())
{
    s.end_zp(zp, c0);
}
template <class S>
__device__ __forceinline__ void store_end_zp(S &, const f32x2 (&)[2], int, long) {}

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

// ------------------------------------------------------------------------------------------ K side, one head

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

// ------------------------------------------------------------------------------------------ value form (both sides)

// Replays four tokens; value(k, xh) takes the dequantised values of position k as two pairs.  aE[k] = alpha * tc^k.
template <int BITS, class Value>
__device__ __forceinline__ void x_tail_block(const uint32_t (&grp)[4], const PairFields<BITS> &fc, f32x2 (&s)[2], f32x2 (&zp)[2],
                                             const TailChan &t, const f32x2 (&aE)[4][2], Value &&value)
{
    static_for<4>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        f32x2 xh[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const f32x2 r = mul2(fc.template code2<k>(grp[2 * p], grp[2 * p + 1]), s[p]);
            xh[p] = k == 0 ? add2(r, zp[p]) : fma2(t.e[k ? k - 1 : 0][p], r, zp[p]);
            zp[p] = fma2(aE[k][p], r, zp[p]);
            s[p] = fma2(t.bp[p], abs2(r), s[p]);
        }
        value(kc, xh);
    });
#pragma unroll
    for (int p = 0; p < 2; ++p) s[p] = mul2(s[p], t.e[3][p]);
}

// The same with guards and clamp for one token (inline: with several heads the operands of a call would not fit the
// registers of the calling convention).
template <int BITS>
__device__ __forceinline__ void x_tail_guarded(const uint32_t (&grp)[4], int j, f32x2 (&s2)[2], f32x2 (&zp2)[2],
                                               const f32x2 (&alpha)[2], const float4 *slow, float smin, float smax, f32x2 (&xh)[2])
{
    float be[4], tc[4], s[4];
    load_slow_consts(slow, be, tc);
    upk2(s2[0], s[0], s[1]);
    upk2(s2[1], s[2], s[3]);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float a = guarded_scale_step(code_f_rt<BITS>(grp[2 * p], j), s[2 * p], be[2 * p], tc[2 * p], smin, smax);
        const float b = guarded_scale_step(code_f_rt<BITS>(grp[2 * p + 1], j), s[2 * p + 1], be[2 * p + 1], tc[2 * p + 1], smin, smax);
        const f32x2 r = pk2(a, b);
        xh[p] = add2(r, zp2[p]);
        zp2[p] = fma2(alpha[p], r, zp2[p]);
        s2[p] = pk2(s[2 * p], s[2 * p + 1]);
    }
}

__device__ __forceinline__ void scaled_alpha(const TailChan &t, f32x2 (&aE)[4][2])
{
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        aE[0][p] = t.alpha[p];
#pragma unroll
        for (int k = 1; k < 4; ++k) aE[k][p] = mul2(t.alpha[p], t.e[k - 1][p]);
    }
}

// ------------------------------------------------------------------------------------------ K warp

// Sink: RingSink<G> (begin_tile, put, end_tile, put_self, finish) or one with end_state(share of sum_c q_c * zp_c per
// lane and head, lane) for a scan without append.  red: kRedFloats floats, 16-byte aligned.
template <int BITS, int G, int STAGES, class Sink>
__device__ __forceinline__ void k_tail_warp(const KArgs &a, const Seg &seg, int b, int h, int lane, uint8_t *ring_buf,
                                            uint64_t *ring_bar, float *red, float4 *slow, Sink &sink)
{
    using C = Codec<BITS>;
    constexpr int kBlocks = kRedUnits / G;            // blocks of 4 tokens per reduction pass
    const int bh = b * a.Hkv + h, c0 = 4 * lane;
    const size_t poff = size_t(h) * kD + c0;
    const __half *q = a.q + (size_t(b) * a.Hq + size_t(h) * G) * kD + c0;
    uint8_t *stream = a.cache + size_t(bh) * a.n_super_cap * kD * 4;
    const int n_tok = seg.t_end - seg.t_begin;
    StreamRing<BITS, STAGES> ring{ring_buf, ring_bar, stream + size_t(seg.t_begin / C::TPW) * (kD * 4),
                                  (n_tok + kTileTok - 1) / kTileTok, n_tok, kStatKWait, kD * 4};
    ring.prologue(lane);   // first: the copies of the first tiles fly while the parameters below are loaded
    PairFields<BITS> fc;
    fc.init();
    float4 *red4 = reinterpret_cast<float4 *>(red) + lane;
    slow += lane;
    bool ok = true;
    int i = 0;
    float z_lane[G];

    // Walks the tiles; tile_body(words, valid tokens) replays one.
    const auto scan = [&](auto &&tile_body, f32x2 (&scale)[2], const uint32_t (&drift)[2]) {
        for (; i < ring.n_tiles; ++i) {
            if (!(ok = ring.wait_short(i))) break;
            if (!(ok = sink.begin_tile_short(i))) break;
            tile_body(ring.tile(i, lane), min(kTileTok, n_tok - i * kTileTok));
            if ((i + 1) % kDriftTiles == 0) correct_drift(scale, drift);
            if constexpr (G == 1) sink.put(0, lane, reduce_units(red, lane));
            sink.end_tile(i, lane);
            ring.release_and_refill(i, lane);
        }
    };

    TailChan t;
    load_tail_chan<BITS>(t, a.p, poff, seg.init, c0, a.smin, a.smax, slow);
    if constexpr (G == 1) {
        float qv[4], al[4];
        load_half4(qv, q);
        upk2(t.alpha[0], al[0], al[1]);
        upk2(t.alpha[1], al[2], al[3]);
        const float4 qf = make_float4(qv[0], qv[1], qv[2], qv[3]);
        const float4 qaf = make_float4(qv[0] * al[0], qv[1] * al[1], qv[2] * al[2], qv[3] * al[3]);
        f32x2 Q[4][2], A[4][2], e4[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            Q[0][p] = p ? pk2(qf.z, qf.w) : pk2(qf.x, qf.y);
            A[0][p] = p ? pk2(qaf.z, qaf.w) : pk2(qaf.x, qaf.y);
            e4[p] = t.e[3][p];
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
                k_tail_block<BITS>(grp, fc, st, t.bp, e4, Q, A, dst);
#pragma unroll
                for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
                k_tail_block<BITS>(grp, fc, st, t.bp, e4, Q, A, dst + 32);
            } else {
                slow_chunk(w, tok, 8);
            }
        };
        scan(
            [&](const uint4 *tile, int ntok) {
                if (ntok == kTileTok) walk_full_tile<BITS>(tile, chunk);
                else walk_tile<BITS>(tile, ntok, slow_chunk);
            },
            st.s, t.drift);
        float lo, hi;
        upk2(st.z, lo, hi);
        z_lane[0] = lo + hi;
    } else {
        f32x2 aE[4][2], qv2[G][2];
        scaled_alpha(t, aE);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float qv[4];
            load_half4(qv, q + size_t(g) * kD);
            qv2[g][0] = pk2(qv[0], qv[1]);
            qv2[g][1] = pk2(qv[2], qv[3]);
        }
        const auto dot = [&](int g, const f32x2 (&x)[2]) {
            float lo, hi;
            upk2(fma2(qv2[g][1], x[1], mul2(qv2[g][0], x[0])), lo, hi);
            return lo + hi;
        };
        const auto body = [&](const uint4 &w, int tok, int count) {
            uint32_t grp[4] = {w.x, w.y, w.z, w.w};
            const bool free8 = count >= 8 && tail_safe(t.safe, t.s);
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {     // one body, two trips: the code has to stay in the instruction cache
                float4 *dst = red4 + (((tok >> 2) + half) % kBlocks) * 32;
                const int n = count - 4 * half;
                if (free8 || (n >= 4 && tail_safe(t.safe4, t.s))) {
                    float v[G][4];
                    x_tail_block<BITS>(grp, fc, t.s, t.zp, t, aE, [&](auto kc, const f32x2 (&xh)[2]) {
#pragma unroll
                        for (int g = 0; g < G; ++g) v[g][decltype(kc)::value] = dot(g, xh);
                    });
#pragma unroll
                    for (int g = 0; g < G; ++g) dst[g * kBlocks * 32] = make_float4(v[g][0], v[g][1], v[g][2], v[g][3]);
                } else {
#pragma unroll 1
                    for (int j = 0; j < 4 && j < n; ++j) {
                        f32x2 xh[2];
                        x_tail_guarded<BITS>(grp, j, t.s, t.zp, t.alpha, slow, a.smin, a.smax, xh);
#pragma unroll
                        for (int g = 0; g < G; ++g) reinterpret_cast<float *>(dst + g * kBlocks * 32)[j] = dot(g, xh);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
            }
            // a pass is complete after kBlocks blocks, or with the last tokens of the tile
            if (((tok >> 2) + 2) % kBlocks == 0 || count <= 8) {
                const float v = reduce_units(red, lane);
                const int unit = lane >> 2;
                sink.put(unit / kBlocks, ((tok >> 2) / kBlocks * kBlocks + unit % kBlocks) * 4 + (lane & 3), v);
            }
        };
        scan([&](const uint4 *tile, int ntok) { walk_tile<BITS>(tile, ntok, body); }, t.s, t.drift);
#pragma unroll
        for (int g = 0; g < G; ++g) z_lane[g] = dot(g, t.zp);
    }
    if (!ok) {
        ring.drain(i);
        return;
    }
    if (!seg.append) {
        sink_end_shares(sink, z_lane, lane, 0);
        return;
    }
    // Append k_new as token T from the tail, then its own logit from the dequantised value.
    float xh[4];
    append_from_tail<BITS>(a.p, poff, a.tail + size_t(bh) * 2 * kD, a.tail_keep, a.x_new + size_t(bh) * kD + c0,
                           reinterpret_cast<uint4 *>(stream + size_t(a.T / C::TPW) * (kD * 4)) + lane, a.T, a.smin, a.smax,
                           seg.ckpt_out, c0, xh);
    if (!sink.begin_tile_short(ring.n_tiles)) return;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        float qv[4], s = 0.f;
        load_half4(qv, q + size_t(g) * kD);
#pragma unroll
        for (int c = 0; c < 4; ++c) s = fmaf(qv[c], xh[c], s);
        s = warp_sum(s);
        if (lane == 0) sink.put_self(g, s);
    }
    sink.finish(lane);
}

// ------------------------------------------------------------------------------------------ V side, one head

struct VTailState {
    f32x2 s[2];
    f32x2 acc[2], accp[2];     // sum w*q*s and sum P*q*s of the positions with power 0
};

// Up to eight tokens, one head (see k_tail_slow).  wts: (w, w, P, P) per token.
template <int BITS>
__device__ __noinline__ VTailState v_tail_slow(uint4 w, VTailState st, const float4 *slow, const float4 *wts, int count,
                                               SafeRange safe4, float smin, float smax)
{
    float be[4], tc[4];
    load_slow_consts(slow, be, tc);
    PairFields<BITS> fc;
    fc.init();
#pragma unroll 1
    for (int half = 0; half < 2; ++half, count -= 4, wts += 4) {
        const uint32_t grp[4] = {w.x, w.y, w.z, w.w};
        if (count >= 4 && tail_safe(safe4, st.s)) {
            static_for<4>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                const ulonglong2 wp = *reinterpret_cast<const ulonglong2 *>(wts + k);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const f32x2 q2 = fc.template code2<k>(grp[2 * p], grp[2 * p + 1]);
                    const f32x2 r = mul2(q2, st.s[p]);
                    st.acc[p] = fma2(wp.x, r, st.acc[p]);
                    st.accp[p] = fma2(wp.y, r, st.accp[p]);
                    st.s[p] = mul2(st.s[p], fma2(pk2(be[2 * p], be[2 * p + 1]), abs2(q2), pk2(tc[2 * p], tc[2 * p + 1])));
                }
            });
        } else {
            float s[4];
            upk2(st.s[0], s[0], s[1]);
            upk2(st.s[1], s[2], s[3]);
#pragma unroll 1
            for (int j = 0; j < 4 && j < count; ++j) {
                const ulonglong2 wp = *reinterpret_cast<const ulonglong2 *>(wts + j);
                float rh[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    rh[c] = guarded_scale_step(code_f_rt<BITS>(grp[c], j), s[c], be[c], tc[c], smin, smax);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const f32x2 r = pk2(rh[2 * p], rh[2 * p + 1]);
                    st.acc[p] = fma2(wp.x, r, st.acc[p]);
                    st.accp[p] = fma2(wp.y, r, st.accp[p]);
                }
            }
            st.s[0] = pk2(s[0], s[1]);
            st.s[1] = pk2(s[2], s[3]);
        }
        shift_words(w, 4 * BITS);
    }
    return st;
}

// Four tokens without guards, one head: one accumulator pair per position of the block.
template <int BITS>
__device__ __forceinline__ void v_tail_block(const uint32_t (&grp)[4], const PairFields<BITS> &fc, f32x2 (&s)[2],
                                             const f32x2 (&bp)[2], const f32x2 (&e4)[2], const float4 *wts,
                                             f32x2 (&acc)[4][2], f32x2 (&accp)[4][2])
{
    static_for<4>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        const ulonglong2 wp = *reinterpret_cast<const ulonglong2 *>(wts + k);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const f32x2 r = mul2(fc.template code2<k>(grp[2 * p], grp[2 * p + 1]), s[p]);
            acc[k][p] = fma2(wp.x, r, acc[k][p]);
            accp[k][p] = fma2(wp.y, r, accp[k][p]);
            s[p] = fma2(bp[p], abs2(r), s[p]);
        }
    });
#pragma unroll
    for (int p = 0; p < 2; ++p) s[p] = mul2(s[p], e4[p]);
}

// ------------------------------------------------------------------------------------------ softmax of a V warp

// Online softmax.  Weights of a tile: PREFIX (one head): (w, w, P, P) per token with the running sum P of the weights;
// otherwise [G][32] (w, w).
template <int G, bool PREFIX>
struct TailSoftmax {
    static constexpr int kFloat4 = PREFIX ? kTileTok : G * kTileTok / 2;
    FusedShared<G> *sh;
    float4 *wts;           // kFloat4 entries
    const float *mask;     // row of this batch or nullptr
    float scale2;          // scaling * log2(e)
    int t_begin;           // first token of this segment (mask index of local token 0)
    float m[G];            // running maximum (log2 units)
    float l[G];            // PREFIX: sum of the weights so far; otherwise this lane's share of it

    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int g = 0; g < G; ++g) { m[g] = -INFINITY; l[g] = 0.f; }
    }
    __device__ __forceinline__ static float redux_max(float v)
    {
        float r;
        asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
        return r;
    }
    // Fills the weights of tile i; corr[g] is what the accumulators of head g have to be scaled with (warp-uniform).
    __device__ __forceinline__ bool tile(int i, int ntok, int lane, float (&corr)[G])
    {
        const int slot = unsigned(i) % kLogitSlots;
        const float mk = (mask && lane < ntok) ? mask[t_begin + i * kTileTok + lane] * 1.4426950408889634f : 0.f;
        if (!mbar_wait_short(&sh->lfull[slot], (unsigned(i) / kLogitSlots) & 1, kStatLFullWait)) return false;
        float x[G];
#pragma unroll
        for (int g = 0; g < G; ++g) x[g] = sh->lring[slot][0][g][lane];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->lempty[slot]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float v = lane < ntok ? fmaf(x[g], scale2, mk) : -INFINITY;
            const float m_new = fmaxf(m[g], redux_max(v));
            const bool dead = m_new == -INFINITY;
            corr[g] = dead ? 1.f : exp2f(m[g] - m_new);
            const float w = dead ? 0.f : exp2f(v - m_new);
            m[g] = m_new;
            if constexpr (PREFIX) {
                float P = w;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float y = __shfl_up_sync(kFull, P, o);
                    if (lane >= o) P += y;
                }
                P = fmaf(l[0], corr[0], P);
                l[0] = __shfl_sync(kFull, P, 31);
                wts[lane] = make_float4(w, w, P, P);
            } else {
                l[g] = fmaf(l[g], corr[g], w);
                reinterpret_cast<float2 *>(wts)[g * kTileTok + lane] = make_float2(w, w);
            }
        }
        __syncwarp();
        return true;
    }
    // after the last tile: l = the sum of the weights, in every lane
    __device__ __forceinline__ void close()
    {
        if constexpr (!PREFIX) {
#pragma unroll
            for (int g = 0; g < G; ++g) l[g] = warp_sum(l[g]);
        }
    }
    // after close(): weight of the appended token, whose logit is the single entry of tile n_tiles
    __device__ __forceinline__ bool self(int n_tiles, int T, float (&out)[G][4], float (&w_self)[G])
    {
        const int slot = unsigned(n_tiles) % kLogitSlots;
        if (!mbar_wait_short(&sh->lfull[slot], (unsigned(n_tiles) / kLogitSlots) & 1, kStatLFullWait)) return false;
        const float mk = mask ? mask[T] * 1.4426950408889634f : 0.f;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float v = fmaf(sh->lring[slot][0][g][0], scale2, mk);
            const float m_new = fmaxf(m[g], v);
            const bool dead = m_new == -INFINITY;
            const float corr = dead ? 1.f : exp2f(m[g] - m_new);
            w_self[g] = dead ? 0.f : exp2f(v - m_new);
            l[g] = fmaf(l[g], corr, w_self[g]);
#pragma unroll
            for (int c = 0; c < 4; ++c) out[g][c] *= corr;
            m[g] = m_new;
        }
        return true;
    }
};

// ------------------------------------------------------------------------------------------ V warp

// store: store(m, l, sums, c0) with the un-normalised sums, give_up(c0) when a bounded wait ran out, and optionally
// end_zp(zero points, c0) for a scan without append (value form).  PREFIX needs one head and the zero points after the
// last token in seg.zp_end.
template <int BITS, int G, bool PREFIX, int STAGES, class Store>
__device__ __forceinline__ void v_tail_warp(const VArgs &a, const Seg &seg, int b, int h, int lane, uint8_t *ring_buf,
                                            uint64_t *ring_bar, float4 *slow, TailSoftmax<G, PREFIX> &src, Store &&store)
{
    using C = Codec<BITS>;
    static_assert(!PREFIX || G == 1, "running sums of the weights: one head");
    const int bh = b * a.Hkv + h, c0 = 4 * lane;
    const size_t poff = size_t(h) * kD + c0;
    uint8_t *stream = a.cache + size_t(bh) * a.n_super_cap * kD * 4;
    const int n_tok = seg.t_end - seg.t_begin;
    StreamRing<BITS, STAGES> ring{ring_buf, ring_bar, stream + size_t(seg.t_begin / C::TPW) * (kD * 4),
                                  (n_tok + kTileTok - 1) / kTileTok, n_tok, kStatVWait, kD * 4};
    ring.prologue(lane);
    PairFields<BITS> fc;
    fc.init();
    slow += lane;
    bool ok = true;
    int i = 0;
    const auto scan = [&](auto &&rescale, auto &&tile_body, f32x2 (&scale)[2], const uint32_t (&drift)[2]) {
        for (; i < ring.n_tiles; ++i) {
            const int ntok = min(kTileTok, n_tok - i * kTileTok);
            float corr[G];
            if (!(ok = src.tile(i, ntok, lane, corr))) break;
            rescale(corr);
            if (!(ok = ring.wait_short(i))) break;
            tile_body(ring.tile(i, lane), ntok);
            if ((i + 1) % kDriftTiles == 0) correct_drift(scale, drift);
            ring.release_and_refill(i, lane);   // also orders this tile's reads of wts before the next fill
        }
    };

    float out[G][4];
    TailChan t;
    load_tail_chan<BITS>(t, a.p, poff, seg.init, c0, a.smin, a.smax, slow);
    if constexpr (PREFIX) {
        f32x2 s[2] = {t.s[0], t.s[1]}, e4[2] = {t.e[3][0], t.e[3][1]}, acc[4][2], accp[4][2];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int p = 0; p < 2; ++p) acc[k][p] = accp[k][p] = 0ull;
        const auto slow_chunk = [&](const uint4 &w, int tok, int count) {
            VTailState st;
#pragma unroll
            for (int p = 0; p < 2; ++p) { st.s[p] = s[p]; st.acc[p] = acc[0][p]; st.accp[p] = accp[0][p]; }
            st = v_tail_slow<BITS>(w, st, slow, src.wts + tok, count, t.safe4, a.smin, a.smax);
#pragma unroll
            for (int p = 0; p < 2; ++p) { s[p] = st.s[p]; acc[0][p] = st.acc[p]; accp[0][p] = st.accp[p]; }
        };
        const auto chunk = [&](const uint4 &w, int tok) {
            if (tail_safe(t.safe, s)) {
                const float4 *wt = src.wts + tok;
                uint32_t grp[4] = {w.x, w.y, w.z, w.w};
                v_tail_block<BITS>(grp, fc, s, t.bp, e4, wt, acc, accp);
#pragma unroll
                for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
                v_tail_block<BITS>(grp, fc, s, t.bp, e4, wt + 4, acc, accp);
            } else {
                slow_chunk(w, tok, 8);
            }
        };
        scan(
            [&](const float (&corr)[G]) {
                if (corr[0] != 1.f) {       // warp-uniform; rare once the running maximum has settled
                    const f32x2 f = pk2(corr[0], corr[0]);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            acc[k][p] = mul2(acc[k][p], f);
                            accp[k][p] = mul2(accp[k][p], f);
                        }
                }
            },
            [&](const uint4 *tile, int ntok) {
                if (ntok == kTileTok) walk_full_tile<BITS>(tile, chunk);
                else walk_tile<BITS>(tile, ntok, slow_chunk);
            },
            s, t.drift);
        if (ok) {
            // sum_k tc^k * (acc_k - alpha * accp_k) + W * zp_end; the constants are loaded again rather than kept
            load_tail_chan<BITS>(t, a.p, poff, nullptr, c0, a.smin, a.smax, slow);
            const f32x2 minus = pk2(-1.f, -1.f);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const f32x2 nal = mul2(t.alpha[p], minus);
                f32x2 sum = fma2(nal, accp[0][p], acc[0][p]);
#pragma unroll
                for (int k = 1; k < 4; ++k) sum = fma2(t.e[k - 1][p], fma2(nal, accp[k][p], acc[k][p]), sum);
                upk2(sum, out[0][2 * p], out[0][2 * p + 1]);
            }
            if (n_tok > 0) {
                const float4 ze = *reinterpret_cast<const float4 *>(seg.zp_end + c0);
                out[0][0] = fmaf(src.l[0], ze.x, out[0][0]);
                out[0][1] = fmaf(src.l[0], ze.y, out[0][1]);
                out[0][2] = fmaf(src.l[0], ze.z, out[0][2]);
                out[0][3] = fmaf(src.l[0], ze.w, out[0][3]);
            }
        }
    } else {
        f32x2 aE[4][2], acc[G][2];
        scaled_alpha(t, aE);
#pragma unroll
        for (int g = 0; g < G; ++g) acc[g][0] = acc[g][1] = 0ull;
        const float2 *wts = reinterpret_cast<const float2 *>(src.wts);
        const auto body = [&](const uint4 &w, int tok, int count) {
            uint32_t grp[4] = {w.x, w.y, w.z, w.w};
            const bool free8 = count >= 8 && tail_safe(t.safe, t.s);
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                const float2 *wt = wts + tok + 4 * half;
                const int n = count - 4 * half;
                if (free8 || (n >= 4 && tail_safe(t.safe4, t.s))) {
                    f32x2 w4[G][4];
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(wt + g * kTileTok);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(wt + g * kTileTok + 2);
                        w4[g][0] = x.x; w4[g][1] = x.y; w4[g][2] = y.x; w4[g][3] = y.y;
                    }
                    x_tail_block<BITS>(grp, fc, t.s, t.zp, t, aE, [&](auto kc, const f32x2 (&xh)[2]) {
#pragma unroll
                        for (int g = 0; g < G; ++g)
#pragma unroll
                            for (int p = 0; p < 2; ++p) acc[g][p] = fma2(w4[g][decltype(kc)::value], xh[p], acc[g][p]);
                    });
                } else {
#pragma unroll 1
                    for (int j = 0; j < 4 && j < n; ++j) {
                        f32x2 xh[2];
                        x_tail_guarded<BITS>(grp, j, t.s, t.zp, t.alpha, slow, a.smin, a.smax, xh);
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const f32x2 w1 = *reinterpret_cast<const f32x2 *>(wt + g * kTileTok + j);
                            acc[g][0] = fma2(w1, xh[0], acc[g][0]);
                            acc[g][1] = fma2(w1, xh[1], acc[g][1]);
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) grp[c] >>= 4 * BITS;
            }
        };
        scan(
            [&](const float (&corr)[G]) {
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const f32x2 f = pk2(corr[g], corr[g]);
                    acc[g][0] = mul2(acc[g][0], f);
                    acc[g][1] = mul2(acc[g][1], f);
                }
            },
            [&](const uint4 *tile, int ntok) { walk_tile<BITS>(tile, ntok, body); }, t.s, t.drift);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            upk2(acc[g][0], out[g][0], out[g][1]);
            upk2(acc[g][1], out[g][2], out[g][3]);
        }
    }
    if (!ok) {
        ring.drain(i);
        store.give_up(c0);
        return;
    }
    src.close();
    if (seg.append) {
        float w_self[G], xh[4];
        if (!src.self(ring.n_tiles, a.T, out, w_self)) {
            store.give_up(c0);
            return;
        }
        append_from_tail<BITS>(a.p, poff, a.tail + size_t(bh) * 2 * kD, a.tail_keep, a.x_new + size_t(bh) * kD + c0,
                               reinterpret_cast<uint4 *>(stream + size_t(a.T / C::TPW) * (kD * 4)) + lane, a.T, a.smin,
                               a.smax, seg.ckpt_out, c0, xh);
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int c = 0; c < 4; ++c) out[g][c] = fmaf(w_self[g], xh[c], out[g][c]);
    } else {
        if constexpr (!PREFIX) store_end_zp(store, t.zp, c0, 0);
    }
    store.store(src.m, src.l, out, c0);
}

// Normalised fp16 result of a whole stream.
template <int G>
struct TailStore {
    __half *out;      // [G][kD] of this stream
    __device__ __forceinline__ void store(const float (&)[G], const float (&l)[G], const float (&acc)[G][4], int c0) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float inv = 1.0f / l[g];
            float o[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] = acc[g][c] * inv;
            store_half4(out + size_t(g) * kD + c0, o);
        }
    }
    __device__ __forceinline__ void give_up(int) const {}
};

}  // namespace adkv
