// Host-side helpers shared by the translation units of libadkv_b200.so.
#pragma once
#include "../../include/adkv_b200.h"
#include "adkv_device.cuh"

#define ADKV_HIDDEN __attribute__((visibility("hidden")))

namespace adkv {

constexpr int kSMs = 148, kSchedulers = 4 * kSMs;   // B200: what the choice of a kernel by number of streams counts in

// Whether a contracted step next to tail states takes the tensor-core kernel (adkv_tensor.cu), by the number of CTAs, one per stream
// or checkpoint segment, and the tokens of each (device_lengths: what the cache can hold of them).  Two CTAs share an SM, so up to
// 296 run at once, and up to 444 and 740 the last round is half full where the 64-thread CTAs of the other kernels pile up on
// some SMs.  A value costs this kernel about the same whatever the number of query heads, the others a multiply-add and an
// eighth of a sum over the lanes per head.  Device time on a B200, us, before -> this kernel (16 heads x 128 wide unless noted):
//   one head     4-bit 128 x 300 14.3 -> 11.2, 128 x 3000 71.7 -> 68.6, 256 x 3000 132 -> 110, 400 x 300 26.6 -> 24.3, 400 x 200
//                19.4 -> 19.8, 592 x 1500 102 -> 109; 2-bit 128 x 300 14.7 -> 12.3, 256 x 3000 139 -> 124, 440 x 1024 73 -> 70
//   two heads    4-bit 128 x 300 16.9 -> 11.4, 256 x 3000 158 -> 111, 740 x 256 37 -> 34, 740 x 1024 117 -> 98, 888 x 1024 118 -> 119
//   four heads   4-bit 128 x 300 19.1 -> 12.3, 256 x 3000 195 -> 118, 740 x 150 33 -> 30, 1184 x 256 59 -> 57, 1480 x 512 121 -> 112,
//                2368 x 512 182 -> 174, 2368 x 3000 973 -> 860; 2-bit 256 x 3000 209 -> 132, 2368 x 512 192 -> 185, x 3000 1033 -> 942.  The
//                kernel stays ahead beyond (4096 x 512 301 / 297, 2-bit 318 / 311), which the line does not use
//   segments     4-bit, one head, between checkpoints 512 tokens apart: 8 streams x 8000 30 -> 19; 2-bit, 4096 apart, 8 x 9000 199 -> 96
// Below 32 tokens set-up counts (148 x 16 tokens 5.0 -> 5.2, 296 x 32 tokens 6.7 -> 6.8).  Device-side lengths may be short whatever the cache
// holds: 384 sequences of four heads, 50 to 100 tokens 19 -> 18, 100 to 2000 tokens 146 -> 69; of one head, 768 x 600 61 -> 76.
// With one channel of every head at a bound 256 x 1000: one head 59 -> 51, four heads 76 -> 55; but where the line for one head ends, 444 x
// 1500 4-bit 110 -> 114, 2-bit 105 -> 113 (without 99 -> 86 and 98 -> 86), and for four, 4-bit 2368 x 512 208 -> 215.
static inline bool tensor_pays(int bits, int G, long long ctas, int tokens, bool device_lengths)
{
    if (device_lengths && (tokens < 128 || (G == 1 && ctas > kSMs))) return false;
    if (ctas <= kSMs) return tokens >= 32;
    if (ctas <= 2 * kSMs) return tokens >= 64;
    if (device_lengths) return tokens >= 512 && ctas <= (G == 2 ? 4 : 5) * kSMs;
    if (ctas <= 3 * kSMs) return tokens >= (G > 1 ? 100 : bits == 4 ? 256 : 128);
    if (ctas <= 5 * kSMs) return tokens >= (G == 4 ? 128 : 256) && G > 1;
    return G == 4 && (ctas <= 8 * kSMs ? tokens >= 256 : ctas <= 16 * kSMs && tokens >= 512);
}
// What that kernel can do: its values are pairs of fp16 numbers in units of 2^-11 of scale_max, which have 22 bits from a quarter of
// a unit on.  Bounds further apart than 2^13 (exp(-4) and exp(4) are 2^11.5) go to the kernels with fp32 values: between 1e-6 and 32768 a
// scale of 3e-4 would leave its values 11 bits.  Values never use a scale below the quantiser's eps.
static inline bool tensor_can(int G, float smin, float smax)
{
    return G <= 4 && smin == smin && smax >= kEps && smax <= 32768.f && smax <= 8192.f * fmaxf(smin, kEps);
}

static inline ParamPtrs to_ptrs(const adkv_params *p)
{
    return ParamPtrs{static_cast<const __half *>(p->zp_init), static_cast<const __half *>(p->scale_init),
                     static_cast<const __half *>(p->alpha), static_cast<const __half *>(p->beta),
                     static_cast<const __half *>(p->target)};
}

static inline bool params_ok(const adkv_params *p)
{
    return p && p->zp_init && p->scale_init && p->alpha && p->beta && p->target;
}

static inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
static inline bool aligned8(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; }

static inline bool params_aligned(const adkv_params *p)
{
    return aligned8(p->zp_init) && aligned8(p->scale_init) && aligned8(p->alpha) && aligned8(p->beta) &&
           aligned8(p->target);
}

static inline int launch_status()
{
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : int(e);
}

static inline int check_common(int B, int Hq, int Hkv, int T, int D, int n_super_cap, int bits, int n_written_end)
{
    if (D != 128 && D != 256 && D != 512) return ADKV_E_HEAD_DIM;
    if (bits != 2 && bits != 4) return ADKV_E_BITS;
    if (B < 0 || Hq <= 0 || Hkv <= 0 || T < 0 || n_super_cap < 0 || Hq % Hkv != 0) return ADKV_E_SHAPE;
    const int tpw = 32 / bits;
    if ((long long)(n_written_end + tpw - 1) / tpw > (long long)n_super_cap) return ADKV_E_CAPACITY;
    return 0;
}

// Tail states of the decode entry points: both or neither, 16-byte aligned, fp32 arithmetic only.
static inline int check_tails(const void *k_tail, const void *v_tail, unsigned flags)
{
    if (!k_tail && !v_tail) return 0;
    if (!k_tail || !v_tail || (flags & ADKV_FLAG_HALF_STATE)) return ADKV_E_FLAGS;
    if (!aligned16(k_tail) || !aligned16(v_tail)) return ADKV_E_ALIGN;
    return 0;
}

// Every translation unit that includes adkv_device.cuh has its own device status word; this defines the hidden
// function through which adkv_device_status reads and clears the one of the unit it is expanded in.
#define ADKV_DEFINE_TU_STATUS(fn_name)                                                \
    ADKV_HIDDEN int fn_name(int *out)                                                 \
    {                                                                                 \
        cudaError_t e = cudaMemcpyFromSymbol(out, adkv::g_status, sizeof(int));       \
        if (e != cudaSuccess) return int(e);                                          \
        const int zero = 0;                                                           \
        e = cudaMemcpyToSymbol(adkv::g_status, &zero, sizeof(int));                   \
        return e == cudaSuccess ? 0 : int(e);                                         \
    }

// Dispatch over (bits, group size, arithmetic).  CALL sees BITS, G, EXACT and ARITH (kArithCanon / kArithFma).
#define ADKV_DISPATCH_G(BITS_, EXACT_, G_, CALL) \
    switch (G_) {                                \
    case 1: { constexpr int BITS = BITS_; constexpr bool EXACT = EXACT_; constexpr int ARITH = EXACT_ ? 1 : 0; constexpr int G = 1; (void)EXACT; (void)ARITH; CALL; } break; \
    case 2: { constexpr int BITS = BITS_; constexpr bool EXACT = EXACT_; constexpr int ARITH = EXACT_ ? 1 : 0; constexpr int G = 2; (void)EXACT; (void)ARITH; CALL; } break; \
    case 4: { constexpr int BITS = BITS_; constexpr bool EXACT = EXACT_; constexpr int ARITH = EXACT_ ? 1 : 0; constexpr int G = 4; (void)EXACT; (void)ARITH; CALL; } break; \
    case 8: { constexpr int BITS = BITS_; constexpr bool EXACT = EXACT_; constexpr int ARITH = EXACT_ ? 1 : 0; constexpr int G = 8; (void)EXACT; (void)ARITH; CALL; } break; \
    default: return ADKV_E_SHAPE;                \
    }
#define ADKV_DISPATCH(bits_, exact_, G_, CALL)                            \
    if (bits_ == 4) {                                                     \
        if (exact_) { ADKV_DISPATCH_G(4, true, G_, CALL) } else { ADKV_DISPATCH_G(4, false, G_, CALL) } \
    } else {                                                              \
        if (exact_) { ADKV_DISPATCH_G(2, true, G_, CALL) } else { ADKV_DISPATCH_G(2, false, G_, CALL) } \
    }


// Dispatch over (bits, group size) for kernels without an EXACT parameter.
#define ADKV_DISPATCH_H(bits_, G_, CALL)                                              \
    switch ((bits_) * 16 + (G_)) {                                                    \
    case 4 * 16 + 1: { constexpr int BITS = 4; constexpr int G = 1; CALL; } break;    \
    case 4 * 16 + 2: { constexpr int BITS = 4; constexpr int G = 2; CALL; } break;    \
    case 4 * 16 + 4: { constexpr int BITS = 4; constexpr int G = 4; CALL; } break;    \
    case 4 * 16 + 8: { constexpr int BITS = 4; constexpr int G = 8; CALL; } break;    \
    case 2 * 16 + 1: { constexpr int BITS = 2; constexpr int G = 1; CALL; } break;    \
    case 2 * 16 + 2: { constexpr int BITS = 2; constexpr int G = 2; CALL; } break;    \
    case 2 * 16 + 4: { constexpr int BITS = 2; constexpr int G = 4; CALL; } break;    \
    case 2 * 16 + 8: { constexpr int BITS = 2; constexpr int G = 8; CALL; } break;    \
    default: return ADKV_E_SHAPE;                                                     \
    }

}  // namespace adkv
