// Tensor memory and tcgen05 wrappers (one CTA, kind::f16 with fp32 accumulators) of the decode kernel in adkv_tensor.cu.
#pragma once
#include "adkv_device.cuh"

namespace adkv {

__device__ __forceinline__ void tmem_alloc(uint32_t *at, uint32_t columns)   // one whole warp; blocks, without a limit of its own, until another kernel on the SM has given its columns back
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(at)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t columns)   // the warp that allocated
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory matrix whose M (or N) index runs along 16-byte rows of eight halves, without swizzle: element (m, k) lies at
// (m / 8) * mn_stride + (k / 8) * k_stride + (k % 8) * 16 + (m % 8) * 2.
__device__ __forceinline__ uint64_t mn_major_desc(const void *p, uint32_t k_stride, uint32_t mn_stride)
{
    return uint64_t((smem_u32(p) >> 4) & 0x3fffu) | uint64_t(k_stride >> 4) << 16 | uint64_t(mn_stride >> 4) << 32 | uint64_t(1) << 46;
}
// fp16 x fp16 -> fp32; a_mn: A is M-major in shared memory (else K-major, in tensor memory); B is N-major; neg_a: minus A
__host__ __device__ constexpr uint32_t mma_desc(int M, int N, bool a_mn, bool neg_a)
{
    return 1u << 4 | uint32_t(neg_a) << 13 | uint32_t(a_mn) << 15 | 1u << 16 | uint32_t(N >> 3) << 17 | uint32_t(M >> 4) << 24;
}
// one lane of a converged warp, known to the compiler as one: products issued under `if (lane == 0)` take four times as long to issue
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void mma_smem(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc),
                 "r"(uint32_t(accumulate)) : "memory");
}
__device__ __forceinline__ void mma_tmem(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc),
                 "r"(uint32_t(accumulate)) : "memory");
}
// the barrier gets one arrival when the matrix products issued so far by this thread are done
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// a warp's 32 lanes x N columns; finished at tmem_wait_ld / tmem_wait_st
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[N], uint32_t at)
{
    static_assert(N == 1 || N == 4 || N == 8 || N == 16, "");
    if constexpr (N == 1)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(at));
    else if constexpr (N == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
    else if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                       "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(at));
}
// the registers become valid: they are passed through so that no use of them moves before the wait
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[N])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ void tmem_st4(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// mbar_wait_bounded with the SM's cycle counter for a clock, which makes less code at every wait: one that reads the timer, inline or
// called, costs a step 1 to 4 %.  A poll waits by itself, up to 3.9 us here, so a warp that waits takes few issue slots.
constexpr uint32_t kWaitCycles = 2000000000u;   // a second at 1.965 GHz; the counter starts again after 2.2 times that
__device__ __forceinline__ uint32_t cycles()
{
    uint32_t t;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
    return t;
}
template <class Done>
__device__ __forceinline__ bool wait_polled(const Done &done, int code)
{
    bool ok = done();
    if (!ok) {
        uint32_t spent = 0, last = cycles();   // from one round to the next: two readings within a round may be moved together
        do {
            const uint32_t now = cycles();
            __nanosleep(64);
            ok = done();
            spent += now - last;
            last = now;
        } while (!ok && spent < kWaitCycles);
    }
    ok = __all_sync(kFull, ok);
    if (!ok && (threadIdx.x & 31) == 0) atomicExch(&g_status, code);
    return ok;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int code)
{
    return wait_polled([&] { return mbar_try_wait(bar, parity); }, code);
}
// two barriers (the second may be absent) with one vote
__device__ __forceinline__ bool mbar_wait_both(uint64_t *a, uint32_t parity_a, uint64_t *b, uint32_t parity_b, int code)
{
    return wait_polled([&] {
        const bool first = mbar_try_wait(a, parity_a), second = !b || mbar_try_wait(b, parity_b);
        return first && second;
    }, code);
}

}  // namespace adkv
