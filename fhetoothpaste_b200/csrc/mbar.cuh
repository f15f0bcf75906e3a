// Shared-memory barriers with transaction counts, and bulk copies that complete on them.
#pragma once

#include <stdint.h>

namespace tp {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
// After mbar_init, before a barrier that lets other threads, blocks or copies use it.
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// Waits for the phase of parity `ph`; gives up (false) after a few seconds.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t ph, uint32_t tries = 1u << 22) {
    for (uint32_t i = 0; i < tries; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(b)), "r"(ph)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Orders this thread's shared-memory writes before bulk copies that read them.
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// `bytes` (a multiple of 16) of this block's shared memory to block `rank` of the cluster, at the
// place where `dst` lies in this block; counted on that block's barrier at the place of `bar`.
__device__ __forceinline__ void bulk_to_block(const void* dst, const void* src, uint32_t bytes, const uint64_t* bar,
                                              uint32_t rank) {
    asm volatile(
        "{\n\t.reg .u32 d, b;\n\t"
        "mapa.shared::cluster.u32 d, %0, %4;\n\t"
        "mapa.shared::cluster.u32 b, %3, %4;\n\t"
        "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [d], [%1], %2, [b];\n\t}" ::"r"(
            smem_u32(dst)),
        "r"(smem_u32(src)), "r"(bytes), "r"(smem_u32(bar)), "r"(rank)
        : "memory");
}

}  // namespace tp
