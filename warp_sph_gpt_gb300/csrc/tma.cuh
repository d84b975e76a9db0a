// tma.cuh -- Blackwell bulk-copy (TMA, non-tensor) and mbarrier primitives in
// inline PTX, for staging contiguous particle ranges in shared memory.
//
// A 1D bulk copy moves `bytes` (a multiple of 16) from a 16-byte aligned
// global address into shared memory and signals completion on an mbarrier as
// transaction bytes.  Waits are bounded: callers poll a fixed number of times
// and report a timeout instead of spinning forever.
#pragma once

#include <stdint.h>

namespace sd {

constexpr uint32_t kPollNs = 2000;  // suspend-time hint of one poll

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Make barrier initialisation visible to the asynchronous (TMA) proxy.
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Order this thread's earlier generic-proxy shared-memory accesses before
// later asynchronous-proxy writes (buffer reuse).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Arrive once and add `bytes` to the expected transaction count of the phase.
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Plain arrival (count 1) on the barrier's current phase.
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 1D bulk copy global -> shared, completing `bytes` transactions on bar.
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// One poll.  With a suspend-time hint of 2 us warps that wait beside working ones
// take fewer issue slots: steps of 100k particles with spheres in the water 1,147
// -> 1,109 us, above it 1,214 -> 1,185, of 792k 3,557 -> 3,465 (the porosity pass;
// the surrogate's kernels are as fast without).  How long a wait lasts that nothing
// ends does not depend on it: such a poll returns after 3.8 us with the hint and
// without, so the limit of 2^20 polls that the kernels pass is 4 s.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kPollNs)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase with the given parity to complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit) {
    for (int i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

}  // namespace sd
