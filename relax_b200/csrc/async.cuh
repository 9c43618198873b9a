// async.cuh -- mbarriers and bulk asynchronous copies.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace relax {
namespace {
namespace async {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the phase `parity` of an mbarrier to complete
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (int it = 0; it < (1 << 22); it++)
        if (mbar_try(bar, parity)) return true;
    return false;
}

// the phase also waits for `bytes` of bulk copies (this thread arrives)
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// this thread's accesses to shared memory so far before later asynchronous
// copies into it (with a barrier between this fence and the copy)
__device__ __forceinline__ void fence_reads() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// bytes (a multiple of 16) from src to dst (both on 16 bytes), completing on bar
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

}  // namespace async
}  // namespace
}  // namespace relax
