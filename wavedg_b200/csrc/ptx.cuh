// Device helpers over PTX: mbarriers with bounded waits, bulk (TMA) and per-thread asynchronous
// copies between global and shared memory.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "launch.hpp"

namespace wdg
{
    // --------------------------------------------------------- PTX helpers
    __device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

    __device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
    {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    }
    __device__ __forceinline__ void fence_mbar_init()
    {
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
    {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                     : "memory");
    }
    // 1-D bulk copy global -> shared through the TMA unit; dst, src and bytes
    // are multiples of 16 (checked by the host before use_tma is set)
    __device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
    {
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(dst)),
            "l"(src), "r"(bytes), "r"(smem_u32(bar))
            : "memory");
    }
    // the same piece of global memory into L2 only
    __device__ __forceinline__ void bulk_prefetch(const void *src, uint32_t bytes)
    {
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
    }
    __device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
    {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        return ok != 0;
    }
    // try_wait with a suspend-time hint: the thread sleeps until the phase
    // completes or the hint (ns) runs out, instead of spinning on the issue port
    __device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t *bar, uint32_t parity)
    {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity), "r"(100000u)
            : "memory");
        return ok != 0;
    }
    __device__ __forceinline__ uint64_t globaltimer_ns()
    {
        uint64_t t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        return t;
    }
    // bounded wait: gives up after limit_ns of wall time (the copies it waits for take
    // microseconds; the limit only guards against a lost completion).  Stage launches pass the
    // handle's limit (StageArgs::wait_ns, 2 s unless set); other kernels use the default.
    __device__ __forceinline__ uint64_t wait_limit(unsigned long long ns) { return ns ? ns : kWaitLimitNs; }
    __device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint64_t limit_ns = kWaitLimitNs)
    {
        if (mbar_try_wait(bar, parity))
            return true;
        const uint64_t t0 = globaltimer_ns();
        for (;;)
        {
            if (mbar_try_wait_sleep(bar, parity))
                return true;
            if (globaltimer_ns() - t0 > limit_ns)
                return false;
        }
    }

    // per-thread asynchronous global -> shared copies (LDGSTS); used for the
    // neighbour traces, which are scattered 8-byte pieces unsuited to TMA
    template <int BYTES>
    __device__ __forceinline__ void cp_async(void *dst, const void *src)
    {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES)
                     : "memory");
    }
    __device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    template <int PENDING>
    __device__ __forceinline__ void cp_async_wait()
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
    }

    // every cp.async of this thread, committed to a group or not
    __device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

    __device__ __forceinline__ void bulk_s2g(void *dst, const void *src, uint32_t bytes)
    {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
                     "r"(bytes)
                     : "memory");
    }
    __device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
    __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
    __device__ __forceinline__ void bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
    __device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
    __device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
} // namespace wdg
