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

}  // namespace adkv
