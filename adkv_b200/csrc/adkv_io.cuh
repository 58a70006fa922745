// Sink and source of the unfused entry points: logits go to / weights come from fp16 rows in global memory
// (the reference's forward_qk / forward_ov contract, src/adkv/kernel/gemv.py:16-97).
#pragma once
#include "adkv_softmax.cuh"

namespace adkv {

constexpr int kStreamsPerCta = 2;   // unfused kernels: 2 streams per CTA, one warp each

template <int G, int TOK = kTileTok>
struct GlobalLogitSink {
    __half *row[G];   // logits row of each q head of this stream: [T+1]
    int T;
    __device__ __forceinline__ bool begin_tile(int) { return true; }
    template <int N>
    __device__ __forceinline__ void put(int i, int g, int tok, float v, int lane)
    {
        const int t = i * TOK + tok + lane;
        if (lane < N && t < T) row[g][t] = __float2half_rn(v);
    }
    __device__ __forceinline__ void end_tile(int, int) {}
    __device__ __forceinline__ void put_self(int g, float v) { row[g][T] = __float2half_rn(v); }
    __device__ __forceinline__ void finish(int) {}
};

// The weights of the next tile are fetched while the current one is replayed: with few streams a warp has its scheduler
// to itself, and a load that is waited for at every tile (about 700 cycles against 1500 of replay) would be paid in full.
template <int G, bool HALF_W = false, int TOK = kTileTok>
struct GlobalWeightSrc {
    static constexpr int TPL = TOK / 32;   // weights of a tile that a lane brings
    const __half *row[G];   // attention weights of each q head of this stream: [T+1]
    float2 *wts;            // every weight stored twice
    int T;
    __half next[G][TPL];
    __device__ __forceinline__ void fetch(int i, int lane)
    {
#pragma unroll
        for (int k = 0; k < TPL; ++k) {
            const int t = i * TOK + lane + 32 * k;
#pragma unroll
            for (int g = 0; g < G; ++g) next[g][k] = t < T ? row[g][t] : __half(0.f);
        }
    }
    __device__ __forceinline__ bool tile_weights(int i, int, int lane, float (&)[G][4])
    {
        if (i == 0) fetch(0, lane);
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int k = 0; k < TPL; ++k) put_weight<HALF_W>(wts, g * TOK + lane + 32 * k, __half2float(next[g][k]));
        fetch(i + 1, lane);
        __syncwarp();
        return true;
    }
    __device__ __forceinline__ bool self_weight(int, float (&)[G][4], float (&w_self)[G], int T)
    {
#pragma unroll
        for (int g = 0; g < G; ++g) w_self[g] = __half2float(row[g][T]);
        return true;
    }
    __device__ __forceinline__ float norm(int) const { return 1.f; }
    __device__ __forceinline__ void store(const VArgs &a, int b, int h, int c0, const float (&acc)[G][4]) const
    {
        store_normalised<G>(*this, a, b, h, c0, acc);
    }
};

}  // namespace adkv
