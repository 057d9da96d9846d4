// Thin wrappers over the sm_90+/sm_100a asynchronous-copy PTX used by the tile kernels:
// one-dimensional bulk copies from global to shared memory (the TMA engine's untiled form,
// cp.async.bulk), the shared-memory mbarrier they complete on, and prefetches into L2. No
// multicast form is used anywhere: every copy has exactly one destination CTA, the one that
// issued it.
//
// Both addresses of a bulk copy must be 16-byte aligned and the size a multiple of 16 bytes.
#pragma once

#include <stdint.h>

namespace nb200 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, int arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(arrivals) : "memory");
}

// Makes a freshly initialised mbarrier visible to the asynchronous proxy (the copy engine).
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Orders the shared-memory accesses of this thread, and of those it has met at a barrier, before copies that it starts from here on.
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// One arrival that also announces `bytes` of copy traffic the barrier must see before the
// current phase completes.
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// Waits for phase `parity` of `bar`, giving up after `limit` polls. Returns false on give-up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int limit) {
    for (int i = 0; i < limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
    }
    return false;
}

// global -> shared, completion counted in bytes on `bar`.
__device__ __forceinline__ void bulk_load(void *smem_dst, const void *gmem_src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// One 4-byte word global -> shared, on its own: where no bulk copy can bring an array because its 16-byte boundaries lie elsewhere. The words
// that a thread has started have landed for it, and behind a barrier for the others, once it has called copies_landed.
__device__ __forceinline__ void copy_word(void *smem_dst, const void *gmem_src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Asks for the L2 lines of `count` 4-byte elements at `p` (the 16-byte-aligned part of the range), 64 MB at most: what lies
// further on would be gone from L2 again before anything reads it.
__device__ __forceinline__ void prefetch_l2(const void *p, int count) {
    const uintptr_t from = (reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15);
    const uintptr_t to = (reinterpret_cast<uintptr_t>(p) + 4 * (uintptr_t)(count < 1 << 24 ? count : 1 << 24)) & ~uintptr_t(15);
    if (to > from)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"((uint32_t)(to - from)) : "memory");
}

}  // namespace nb200
