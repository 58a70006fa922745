// Pieces shared by the fused decode kernels: the logits ring between the K and V warp of a stream, the
// K-side sink that fills it and the V-side source that turns logits into online-softmax weights.
#pragma once
#include "adkv_decode.cuh"

namespace adkv {

// S = number of 128-channel slices of the head (head_dim / 128): each slice has its own K warp, which
// contributes a partial logit, and its own V warp, which sums the S partials.  The full barrier of a slot
// therefore collects S arrivals (one per K warp) and the empty barrier S arrivals (one per V warp).
template <int G, int S = 1, int TOK = kTileTok>
struct FusedShared {
    float lring[kLogitSlots][S][G][TOK];
    uint64_t lfull[kLogitSlots], lempty[kLogitSlots];
    __device__ __forceinline__ void init_barriers(int n_consumers)
    {
        for (int i = 0; i < kLogitSlots; ++i) {
            mbar_init(&lfull[i], S);
            mbar_init(&lempty[i], n_consumers);
        }
    }
};

template <int G, int S = 1, int TOK = kTileTok>
struct RingSink {
    FusedShared<G, S, TOK> *sh;
    int slot;
    int sl;      // this K warp's slice
    __device__ __forceinline__ bool begin_tile(int i)
    {
        slot = i % kLogitSlots;
        return mbar_wait_bounded(&sh->lempty[slot], ((i / kLogitSlots) & 1) ^ 1, kStatLEmptyWait);
    }
    template <int N>
    __device__ __forceinline__ void put(int, int g, int tok, float v, int lane)
    {
        if (lane < N) sh->lring[slot][sl][g][tok + lane] = v;
    }
    __device__ __forceinline__ void end_tile(int, int lane)
    {
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->lfull[slot]);
    }
    __device__ __forceinline__ void put_self(int g, float v) { sh->lring[slot][sl][g][0] = v; }
    __device__ __forceinline__ void finish(int lane) { end_tile(0, lane); }
};

// Weights of a tile for the V warp: [G][TOK] float2 (w, w), or with HALF_W [G][TOK] fp16 pairs (w, w) in the first
// half of the same array (the fp16-state kernels multiply in fp16x2).
template <bool HALF_W>
__device__ __forceinline__ void put_weight(float2 *wts, int idx, float w)
{
    if (HALF_W) {
        const __half2 h = __floats2half2_rn(w, w);
        reinterpret_cast<uint32_t *>(wts)[idx] = *reinterpret_cast<const uint32_t *>(&h);
    } else {
        wts[idx] = make_float2(w, w);
    }
}

template <int G, int S = 1, bool HALF_W = false, int TOK = kTileTok>
struct SoftmaxSrc {
    static constexpr int TPL = TOK / 32;   // tokens of a tile that a lane weighs: lane, lane + 32
    FusedShared<G, S, TOK> *sh;
    float2 *wts;           // [G][TOK], every weight stored twice (packed multiplier for a channel pair)
    const float *mask;     // row of this batch or nullptr
    float scale2;          // scaling * log2(e)
    int n_tiles;           // tiles of this segment
    int t_begin;           // first token of this segment (mask index of local token 0)
    float m[G], l[G];      // maximum (the same in all lanes) and this lane's share of the denominator (see denominator)

    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int g = 0; g < G; ++g) { m[g] = -INFINITY; l[g] = 0.f; }
    }
    // online-softmax update of head g with this lane's logits v (already in log2 units, -inf if invalid): v becomes the weights
    __device__ __forceinline__ void update(int g, float (&v)[TPL], float (&acc)[G][4])
    {
        float top = v[0];
#pragma unroll
        for (int k = 1; k < TPL; ++k) top = fmaxf(top, v[k]);
        const float m_new = fmaxf(m[g], warp_max(top));
        const bool dead = (m_new == -INFINITY);
        const float corr = dead ? 1.f : exp2f(m[g] - m_new);
        l[g] *= corr;
#pragma unroll
        for (int k = 0; k < TPL; ++k) {
            v[k] = dead ? 0.f : exp2f(v[k] - m_new);
            l[g] += v[k];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[g][c] *= corr;
        m[g] = m_new;
    }
    __device__ __forceinline__ bool tile_weights(int i, int ntok, int lane, float (&acc)[G][4])
    {
        const int slot = i % kLogitSlots;
        float mk[TPL];
#pragma unroll
        for (int k = 0; k < TPL; ++k)
            mk[k] = (mask && lane + 32 * k < ntok) ? mask[t_begin + i * TOK + lane + 32 * k] * 1.4426950408889634f : 0.f;
        if (!mbar_wait_bounded(&sh->lfull[slot], (i / kLogitSlots) & 1, kStatLFullWait)) return false;
        float x[G][TPL];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int k = 0; k < TPL; ++k) {
                x[g][k] = sh->lring[slot][0][g][lane + 32 * k];
#pragma unroll
                for (int j = 1; j < S; ++j) x[g][k] += sh->lring[slot][j][g][lane + 32 * k];
            }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->lempty[slot]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int k = 0; k < TPL; ++k) x[g][k] = lane + 32 * k < ntok ? fmaf(x[g][k], scale2, mk[k]) : -INFINITY;
            update(g, x[g], acc);
#pragma unroll
            for (int k = 0; k < TPL; ++k) put_weight<HALF_W>(wts, g * TOK + lane + 32 * k, x[g][k]);
        }
        __syncwarp();
        return true;
    }
    __device__ __forceinline__ bool self_weight(int lane, float (&acc)[G][4], float (&w_self)[G], int T)
    {
        const int slot = n_tiles % kLogitSlots;
        if (!mbar_wait_bounded(&sh->lfull[slot], (n_tiles / kLogitSlots) & 1, kStatLFullWait)) return false;
        const float mk = mask ? mask[T] * 1.4426950408889634f : 0.f;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float xs = sh->lring[slot][0][g][0];
#pragma unroll
            for (int k = 1; k < S; ++k) xs += sh->lring[slot][k][g][0];
            const float v = fmaf(xs, scale2, mk);
            // all lanes hold the same v: update() would count it 32 times, so do it by hand
            const float m_new = fmaxf(m[g], v);
            const bool dead = (m_new == -INFINITY);
            const float corr = dead ? 1.f : exp2f(m[g] - m_new);
            const float pw = dead ? 0.f : exp2f(v - m_new);
            l[g] = fmaf(l[g], corr, lane == 0 ? pw : 0.f);
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[g][c] *= corr;
            m[g] = m_new;
            w_self[g] = pw;
        }
        return true;
    }
    // Summed over the lanes once per stream: a sum per tile would put five shuffles in a row before its weights.
    __device__ __forceinline__ float denominator(int g) const { return warp_sum(l[g]); }
    __device__ __forceinline__ float norm(int g) const { return denominator(g); }
    __device__ __forceinline__ void store(const VArgs &a, int b, int h, int c0, const float (&acc)[G][4]) const
    {
        store_normalised<G>(*this, a, b, h, c0, acc);
    }
};

constexpr int kPartStride = 4 + kD;   // floats per (stream, segment, head): max (log2 units), denominator, 2 pad, kD sums

struct CkptArgs {
    float *k_ckpt, *v_ckpt;   // [B*Hkv][n_ckpt_cap][2][kD]; entry k = state before token (k+1)*interval
    int interval, n_ckpt_cap;
    bool mute_k;              // self-test (ADKV_FLAG_SELFTEST_MUTE_K): the K warps do nothing, so the waits behind them run out
};

// Device-side lengths: the sequence that comes r-th when they are ordered by length, longest first (equal ones by index).
// CTAs start in the order of their index, so the long streams start together and early and the short ones fill the gaps;
// in the order of the batch an SM may hold several long streams while its neighbours run dry.  Measured on a B200, lengths
// spread evenly between a twentieth of the longest and the longest, order of the batch -> longest first, 32 heads:
//    4-bit, 48 sequences x 3000 tokens 324 -> 252 us; 24 x 2000 154 -> 131 us; 2-bit, 8 KV heads, 96 x 3000 372 -> 304 us
// Every CTA ranks the lengths for itself, in shared memory: B * B / 64 comparisons a thread.  With many CTAs to an SM and no sequence
// of a few hundred tokens that is more than it gains, however large the cache: 128 sequences of 150 to 200 tokens in a cache for
// 4096, 4-bit, 32 heads, 101 us in the order of the batch, 112 us ranked; 2-bit, 8 KV heads, 48 sequences 30.3 us against 28.2 us
// ranked.  More than 128 sequences fill the chip several times over, so that its scheduler evens them out.
// A call, not inlined, and no early return: either would change the registers of the scans behind it (up to 5 % of a step).
constexpr int kRankMax = 128, kRankMinTokens = 512, kRankAlways = 8 * 148 /* SMs */;
template <int THREADS>
__device__ __noinline__ int longest_first(const int *__restrict__ seq_lens, int B, int r, int *key /* [kRankMax + 1] shared */)
{
    // length and index in one number, all different; lengths that no cache holds fall together at either end
    bool any_long = false;
    for (int i = threadIdx.x; i < kRankMax; i += THREADS) {
        const int len = i < B ? min(max(seq_lens[i], 0), 1 << 23) : 0;
        any_long |= len >= kRankMinTokens;
        key[i] = i < B ? len * kRankMax + (kRankMax - 1 - i) : -1;
    }
    if (threadIdx.x == 0) key[kRankMax] = r;
    const int n = __syncthreads_or(any_long || gridDim.x <= kRankAlways) ? B : 0;
    for (int b = threadIdx.x; b < n; b += THREADS) {
        const int mine = key[b];
        int before = 0;
        for (int i = 0; i < B; i += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(key + i);
            before += (v.x > mine) + (v.y > mine) + (v.z > mine) + (v.w > mine);
        }
        if (before == r) key[kRankMax] = b;
    }
    __syncthreads();
    return key[kRankMax];
}

}  // namespace adkv
