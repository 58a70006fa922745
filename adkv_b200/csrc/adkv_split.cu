// Part of libadkv_b200.so (sm_100a).  See include/adkv_b200.h for the contract of every entry point.
//
// Decode over a checkpointed cache: with the recurrence state stored every `interval` tokens, the
// segments between checkpoints are independent, so every (stream, segment) gets its own K/V warp
// pair instead of one pair walking the whole sequence.  Segments leave un-normalised partial results
// (running maximum, denominator, weighted sums) in caller-provided scratch memory; a second small
// kernel merges them.  The idea of boundary state checkpoints is the reference paper's (appendix on
// long contexts); the reference code has no implementation of it.
#include "adkv_host.h"

#include <mutex>

#include "adkv_half.cuh"
#include "adkv_softmax.cuh"

namespace adkv {

// Tokens per tile (TOK), 64 in two stages or 32 in three, see kFusedStages (adkv_fused.cu).  The fp16-state kernel keeps 32 and with
// it more CTAs on an SM (see short_tiles_half), and so do 4-bit codes with eight query heads, where 64 take 38 KB of shared
// memory, up to intervals of 512.  Device time on a B200, 64 -> 32 tokens: intervals of 128, 512 streams x 2000 tokens 311 -> 275 us,
// 128 x 8000 305 -> 269 us; of 512, 512 x 2000 262 -> 248 us; of 1024, 8 x 2000 100 -> 103 us; 2-bit, of 128, 512 x 2000 317 -> 353 us.
template <int TOK>
constexpr int kSplitStages = TOK == 64 ? 2 : 3;

template <int G, bool HALF_W, int TOK>
struct PartialSrc : SoftmaxSrc<G, 1, HALF_W, TOK> {
    float *part;   // [G][kPartStride] of this (stream, segment)
    __device__ __forceinline__ void store(const VArgs &, int, int, int c0, const float (&acc)[G][4]) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float l = this->denominator(g);
            if (c0 == 0) {
                part[g * kPartStride] = this->m[g];
                part[g * kPartStride + 1] = l;
            }
            *reinterpret_cast<float4 *>(part + g * kPartStride + 4 + c0) =
                make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
        }
    }
    // The segment could not be finished (a bounded wait gave up; the status word says which): leave a partial
    // that turns the merged output of these heads into NaN, so that neither the scratch contents of an earlier
    // call nor an output that silently lacks a segment can pass for a result.
    __device__ __forceinline__ void give_up(int c0) const
    {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (c0 == 0) {
                part[g * kPartStride] = -INFINITY;
                part[g * kPartStride + 1] = __int_as_float(0x7fc00000);
            }
            *reinterpret_cast<float4 *>(part + g * kPartStride + 4 + c0) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
};

// Guarded chunk bodies as function calls (see k_chunk_guarded): measured 2-3 % faster for 4-bit codes with one query
// head per KV head at every batch and checkpoint interval tried; not measured for the other instantiations.
template <int BITS, int G>
constexpr bool kOutOfLineGuardedSegments = BITS == 4 && G == 1;

template <int BITS, int G, int MODE, int TOK>
__global__ void __launch_bounds__(64) decode_attn_split_kernel(KArgs ka, VArgs va, const float *__restrict__ mask,
                                                               long long mask_stride_b, float scaling, CkptArgs ck,
                                                               float *__restrict__ scratch)
{
    constexpr int ST = kSplitStages<TOK>;
    __shared__ alignas(128) uint8_t kbuf[ST * Tile<BITS, TOK>::BYTES];
    __shared__ alignas(128) uint8_t vbuf[ST * Tile<BITS, TOK>::BYTES];
    __shared__ alignas(16) float red[G * 8 * kRedRow];
    __shared__ alignas(16) float2 wts[G * TOK];
    __shared__ FusedShared<G, 1, TOK> fs;
    __shared__ uint64_t kbar[ST], vbar[ST];

    const int bh = blockIdx.x, b = bh / ka.Hkv, h = bh % ka.Hkv;
    const int j = blockIdx.y, n_seg = gridDim.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; ++i) { mbar_init(&kbar[i], 1); mbar_init(&vbar[i], 1); }
        fs.init_barriers(1);
        mbar_init_fence();
    }
    __syncthreads();

    const int T = ka.T;
    Seg seg;
    seg.t_begin = j * ck.interval;
    seg.t_end = min(T, (j + 1) * ck.interval);
    seg.append = (j == n_seg - 1);
    seg.slice = 0;
    const size_t stream_ckpt = size_t(bh) * ck.n_ckpt_cap;
    const bool write_ckpt = seg.append && (T + 1) % ck.interval == 0;
    const size_t out_idx = write_ckpt ? stream_ckpt + (T + 1) / ck.interval - 1 : 0;
    if (warp == 0) {
        if (ck.mute_k) return;
        seg.init = j ? ck.k_ckpt + (stream_ckpt + j - 1) * 2 * kD : nullptr;
        seg.ckpt_out = write_ckpt ? ck.k_ckpt + out_idx * 2 * kD : nullptr;
        RingSink<G, 1, TOK> sink{&fs, 0, 0};
        k_scan<BITS, G, MODE, RingSink<G, 1, TOK>, ST, false, kOutOfLineGuardedSegments<BITS, G>, TOK>(ka, seg, b, h, lane, kbuf, kbar,
                                                                                                       red, sink);
    } else {
        seg.init = j ? ck.v_ckpt + (stream_ckpt + j - 1) * 2 * kD : nullptr;
        seg.ckpt_out = write_ckpt ? ck.v_ckpt + out_idx * 2 * kD : nullptr;
        using Src = PartialSrc<G, MODE == kModeHalf, TOK>;
        Src src;
        src.sh = &fs;
        src.wts = wts;
        src.mask = mask ? mask + size_t(b) * mask_stride_b : nullptr;
        src.scale2 = scaling * 1.4426950408889634f;
        src.n_tiles = (seg.t_end - seg.t_begin + TOK - 1) / TOK;
        src.t_begin = seg.t_begin;
        src.part = scratch + (size_t(bh) * n_seg + j) * G * kPartStride;
        src.init();
        v_scan<BITS, G, MODE, Src, ST, false, kOutOfLineGuardedSegments<BITS, G>, TOK>(va, seg, b, h, lane, vbuf, vbar, wts, src);
    }
}

// out[b, hq, c] = sum_j acc_j[c] * 2^(m_j - M) / sum_j l_j * 2^(m_j - M),  M = max_j m_j.
// Bound by the latency of its loads, a few hundred nanoseconds each: the maxima and denominators of all segments are read side
// by side, a segment per thread, and the sums eight segments at a time.  One after the other, the merge was up to a sixth of the
// step (one B200, whole step): 128 heads x 32 segments 112.8 -> 109.3 us, 32 x 63 49.9 -> 42.5 us, 64 x 39 56.8 -> 51.9 us.
__global__ void __launch_bounds__(kD) merge_partials_kernel(const float *__restrict__ scratch, __half *__restrict__ out,
                                                            int Hq, int Hkv, int n_seg)
{
    __shared__ float w[kD], part_max[kD / 32], part_sum[kD / 32];
    const int bhq = blockIdx.x, b = bhq / Hq, hq = bhq % Hq, G = Hq / Hkv, h = hq / G, g = hq % G;
    const int c = threadIdx.x;
    // Launched as a programmatic dependent of the segment kernel (its launch latency is paid while that kernel
    // still runs): wait here until the segment kernel has completed and its partials are visible.  Without
    // that launch attribute the instruction does nothing.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float *base = scratch + (size_t(b * Hkv + h) * n_seg * G + g) * kPartStride;
    const size_t seg_stride = size_t(G) * kPartStride;
    float M = -INFINITY;
    for (int j = c; j < n_seg; j += kD) M = fmaxf(M, base[j * seg_stride]);
    M = warp_max(M);
    if (c % 32 == 0) part_max[c / 32] = M;
    __syncthreads();
    M = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3]));
    float L = 0.f, A = 0.f;
    for (int j0 = 0; j0 < n_seg; j0 += kD) {
        const int n = min(kD, n_seg - j0);
        if (c < n) {
            const float2 ml = *reinterpret_cast<const float2 *>(base + (j0 + c) * seg_stride);
            w[c] = ml.x == -INFINITY ? 0.f : exp2f(ml.x - M);
            L = fmaf(ml.y, w[c], L);
        }
        __syncthreads();
        const float *acc = base + j0 * seg_stride + 4 + c;
#pragma unroll 8
        for (int j = 0; j < n; ++j) A = fmaf(acc[j * seg_stride], w[j], A);
        __syncthreads();
    }
    L = warp_sum(L);
    if (c % 32 == 0) part_sum[c / 32] = L;
    __syncthreads();
    L = (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
    out[size_t(bhq) * kD + c] = __float2half_rn(A / L);
}

// The same for a handful of segments: every thread reads them all at once, which takes one round trip and no barrier.  Whole
// step, fp16 state, device time on a B200, merge_partials_kernel -> this: 32 heads x 5 segments 9.8 -> 8.2 us, 8 x 4 25.6 -> 24.6 us,
// 512 x 4 83.5 -> 81.9 us.
constexpr int kMergeFew = 6;
__global__ void __launch_bounds__(kD) merge_few_kernel(const float *__restrict__ scratch, __half *__restrict__ out, int Hq, int Hkv,
                                                       int n_seg)
{
    const int bhq = blockIdx.x, b = bhq / Hq, hq = bhq % Hq, G = Hq / Hkv, h = hq / G, g = hq % G;
    const int c = threadIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // as in merge_partials_kernel
    const float *base = scratch + (size_t(b * Hkv + h) * n_seg * G + g) * kPartStride;
    const size_t seg_stride = size_t(G) * kPartStride;
    float m[kMergeFew], l[kMergeFew], acc[kMergeFew], M = -INFINITY, L = 0.f, A = 0.f;
#pragma unroll
    for (int j = 0; j < kMergeFew; ++j) {
        const bool there = j < n_seg;
        m[j] = there ? base[j * seg_stride] : -INFINITY;
        l[j] = there ? base[j * seg_stride + 1] : 0.f;
        acc[j] = there ? base[j * seg_stride + 4 + c] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kMergeFew; ++j) M = fmaxf(M, m[j]);
#pragma unroll
    for (int j = 0; j < kMergeFew; ++j) {
        const float w = m[j] == -INFINITY ? 0.f : exp2f(m[j] - M);
        L = fmaf(l[j], w, L);
        A = fmaf(acc[j], w, A);
    }
    out[size_t(bhq) * kD + c] = __float2half_rn(A / L);
}

}  // namespace adkv

using namespace adkv;

ADKV_HIDDEN int adkv_tensor_decode_attn(const KArgs &ka, const VArgs &va, const float *mask, long long mask_stride_b, float scaling,
                                        int B, int bits, const int *seq_lens, int n_rank, const CkptArgs &ck, int n_seg,
                                        float *scratch, cudaStream_t s);

ADKV_DEFINE_TU_STATUS(adkv_tu_status_split)

// The merge follows the segment kernel on the same stream as its programmatic dependent: set up early, started
// when the segment kernel is done (griddepcontrol.wait in the kernel orders the memory).
static int launch_merge(const float *scratch, __half *out, int B, int Hq, int Hkv, int n_seg, cudaStream_t s)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(B * Hq);
    cfg.blockDim = dim3(kD);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const auto kernel = n_seg <= kMergeFew ? merge_few_kernel : merge_partials_kernel;
    if (cudaLaunchKernelEx(&cfg, kernel, scratch, out, Hq, Hkv, n_seg) != cudaSuccess) {
        // the step has appended its token by now: where the merge may not wait beside it, it follows as an ordinary launch
        cudaGetLastError();
        kernel<<<cfg.gridDim, cfg.blockDim, 0, s>>>(scratch, out, Hq, Hkv, n_seg);
    }
    return launch_status();
}

extern "C" {

long long adkv_decode_attn_ckpt_scratch_bytes(int B, int Hq, int Hkv, int T, int interval)
{
    if (B < 0 || Hq <= 0 || Hkv <= 0 || T < 0 || interval <= 0 || Hq % Hkv != 0) return ADKV_E_SHAPE;
    return (long long)B * Hq * (T / interval + 1) * kPartStride * (long long)sizeof(float);
}

int adkv_decode_attn_ckpt(const void *q, void *k_cache, void *v_cache, const void *k_new, const void *v_new,
                          const adkv_params *kp, const adkv_params *vp, void *k_tail, void *v_tail, void *k_ckpt,
                          void *v_ckpt, int interval, int n_ckpt_cap, const void *mask, long long mask_stride_b, void *out, void *scratch,
                          long long scratch_bytes, int B, int Hq, int Hkv, int T, int D, int n_super_cap, int bits,
                          float scaling, float scale_min, float scale_max, unsigned flags, void *stream)
{
    if (!q || !k_cache || !v_cache || !k_new || !v_new || !out || !params_ok(kp) || !params_ok(vp) || !scratch ||
        !k_ckpt || !v_ckpt)
        return ADKV_E_NULL;
    if (D != kD) return ADKV_E_HEAD_DIM;   // checkpointed decode: 128-wide heads only
    if (int rc = check_common(B, Hq, Hkv, T, D, n_super_cap, bits, T + 1)) return rc;
    if (int rc = check_tails(k_tail, v_tail, flags)) return rc;
    if (interval <= 0 || interval % kTileTok != 0 || n_ckpt_cap < 0) return ADKV_E_SHAPE;
    if ((T + 1) / interval > n_ckpt_cap) return ADKV_E_CAPACITY;
    if (!aligned16(k_cache) || !aligned16(v_cache) || !aligned8(q) || !aligned8(out) || !aligned8(k_new) ||
        !aligned8(v_new) || !params_aligned(kp) || !params_aligned(vp) || !aligned16(k_ckpt) || !aligned16(v_ckpt) ||
        !aligned16(scratch))
        return ADKV_E_ALIGN;
    if (scratch_bytes < adkv_decode_attn_ckpt_scratch_bytes(B, Hq, Hkv, T, interval)) return ADKV_E_SCRATCH;
    if (B == 0) return 0;
    const bool keep = flags & ADKV_FLAG_TAIL_KEEP;
    const KArgs ka{static_cast<const __half *>(q), static_cast<uint8_t *>(k_cache),
                   static_cast<const __half *>(k_new), to_ptrs(kp), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D,
                   static_cast<float *>(k_tail), keep};
    const VArgs va{static_cast<uint8_t *>(v_cache), static_cast<const __half *>(v_new), static_cast<__half *>(out),
                   to_ptrs(vp), Hq, Hkv, T, n_super_cap, scale_min, scale_max, D, static_cast<float *>(v_tail), keep};
    const CkptArgs ck{static_cast<float *>(k_ckpt), static_cast<float *>(v_ckpt), interval, n_ckpt_cap,
                      (flags & ADKV_FLAG_SELFTEST_MUTE_K) != 0};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool exact = !(flags & ADKV_FLAG_FAST_REPLAY);
    const int n_seg = T / interval + 1;
    if (n_seg > 65535) return ADKV_E_SHAPE;
    const dim3 grid(B * Hkv, n_seg);
    if (ka.tail && !exact && tensor_can(Hq / Hkv, scale_min, scale_max) &&
        tensor_pays(bits, Hq / Hkv, (long long)B * Hkv * n_seg, min(T, interval), false)) {
        if (int rc = adkv_tensor_decode_attn(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, B, bits, nullptr, 0, ck, n_seg,
                                             static_cast<float *>(scratch), s))
            return rc;
    } else if (flags & ADKV_FLAG_HALF_STATE) {
        ADKV_DISPATCH_H(bits, Hq / Hkv,
                        (decode_attn_split_kernel<BITS, G, kModeHalf, 32><<<grid, 64, 0, s>>>(
                          ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, ck,
                          static_cast<float *>(scratch))))
    } else if (bits == 4 && Hq / Hkv == 8 && interval <= 512) {
        const auto kernel = exact ? decode_attn_split_kernel<4, 8, kArithCanon, 32> : decode_attn_split_kernel<4, 8, kArithFma, 32>;
        kernel<<<grid, 64, 0, s>>>(ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, ck, static_cast<float *>(scratch));
    } else {
        ADKV_DISPATCH(bits, exact, Hq / Hkv,
                      (decode_attn_split_kernel<BITS, G, ARITH, 64><<<grid, 64, 0, s>>>(
                          ka, va, static_cast<const float *>(mask), mask_stride_b, scaling, ck,
                          static_cast<float *>(scratch))))
    }
    if (int rc = launch_status()) return rc;
    return launch_merge(static_cast<const float *>(scratch), static_cast<__half *>(out), B, Hq, Hkv, n_seg, s);
}

}  // extern "C"

// =========================================================================================
// The same decode step for callers that are not in a position to provide scratch memory.
//
// Some hosts of this library cannot allocate: an inference server that has handed every byte of HBM
// to its own block pool at start-up has nothing left for cudaMalloc to give (and would not want the
// fragmentation), and a plugin that is only ever passed device pointers by its host runtime has no
// allocator to ask.  For them the partial results live in the fixed array below instead of a
// caller-owned buffer.  Every process that loads the library pays for the array on every GPU it
// touches until it exits, which is why it is kept to ADKV_STATIC_SCRATCH_BYTES.
namespace adkv {

static __device__ __align__(256) float g_static_scratch[ADKV_STATIC_SCRATCH_BYTES / sizeof(float)];

// In host code `g_static_scratch` is only a handle for the runtime, not a device address: handing it
// to a kernel would fault or, where the GPU can reach host memory, quietly use the wrong memory.
// The device address is asked for once per device, with that device current, and remembered.
constexpr int kMaxDevices = 64;
static float *g_static_scratch_addr[kMaxDevices];
static bool g_static_scratch_known[kMaxDevices];
static std::mutex g_static_scratch_lock;

static int static_scratch_of_current_device(float **addr)
{
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return launch_status();
    if (dev < 0 || dev >= kMaxDevices) return ADKV_E_SHAPE;
    std::lock_guard<std::mutex> guard(g_static_scratch_lock);
    if (!g_static_scratch_known[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess) return launch_status();
        g_static_scratch_addr[dev] = static_cast<float *>(p);
        g_static_scratch_known[dev] = true;
    }
    *addr = g_static_scratch_addr[dev];
    return 0;
}

}  // namespace adkv

extern "C" {

int adkv_decode_attn_ckpt_static(const void *q, void *k_cache, void *v_cache, const void *k_new, const void *v_new,
                                 const adkv_params *kp, const adkv_params *vp, void *k_tail, void *v_tail,
                                 void *k_ckpt, void *v_ckpt, int interval, int n_ckpt_cap, const void *mask, long long mask_stride_b, void *out,
                                 int B, int Hq, int Hkv, int T, int D, int n_super_cap, int bits, float scaling,
                                 float scale_min, float scale_max, unsigned flags, void *stream)
{
    const long long need = adkv_decode_attn_ckpt_scratch_bytes(B, Hq, Hkv, T, interval);
    if (need < 0) return int(need);
    if (need > (long long)ADKV_STATIC_SCRATCH_BYTES) return ADKV_E_STATIC_MAX;
    float *scratch = nullptr;
    if (int rc = static_scratch_of_current_device(&scratch)) return rc;
    // Nothing in the array has to start at zero: the segment kernel writes every slot the merge kernel
    // reads -- its result, or a NaN marker where a bounded wait gave up -- so what an earlier call left
    // behind is always overwritten.
    return adkv_decode_attn_ckpt(q, k_cache, v_cache, k_new, v_new, kp, vp, k_tail, v_tail, k_ckpt, v_ckpt, interval,
                                 n_ckpt_cap, mask, mask_stride_b, out, scratch, (long long)ADKV_STATIC_SCRATCH_BYTES, B, Hq, Hkv,
                                 T, D, n_super_cap, bits, scaling, scale_min, scale_max, flags, stream);
}

}  // extern "C"
