// Tensor-core plumbing shared by the tcgen05 kernels: mbarriers with bounded
// waits, bulk copies into shared memory, ordering fences.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace pgpu {

constexpr int PGPU_STATUS_TIMEOUT = 3;  // device status word: a bounded wait gave up
constexpr int TC_SPIN = 1 << 20;        // try_wait rounds before giving up

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
// Bounded wait for the completion of the phase of `bar` with parity `parity`.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    const uint32_t a = smem_u32(bar);
    for (int it = 0; it < TC_SPIN; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bulk copy global -> shared (this GPU's memory, no multicast), completion on `bar`.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Ahead of a CTA's early end, once a wait has given up: the bulk copies that the
// calling thread has issued into a ring of `stages` buffers (`issued` loads so far,
// each completing a phase of its stage's full[]) are waited for, bounded too, and
// so are the MMAs that it has issued (through `bar`, not used before).
__device__ __forceinline__ bool drain_loads(uint64_t *full, uint32_t stages, uint32_t issued) {
    bool ok = true;
    for (uint32_t i = issued > stages ? issued - stages : 0; i < issued; i++)
        ok &= mbar_wait(&full[i % stages], (i / stages) & 1);
    return ok;
}
__device__ __forceinline__ bool drain_mmas(uint64_t *bar) {
    tc_commit(bar);
    return mbar_wait(bar, 0);
}

}  // namespace pgpu
