// TMA bulk copies between global and shared memory, completed on an mbarrier
// whose wait is bounded in time; shared by the kernels that hold worlds in
// shared memory.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fs3d {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the mbarrier phase for at most limit_ns nanoseconds of the global
// timer (try_wait itself may suspend for a while, so the bound is on time, not
// on tries); false if it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, uint64_t limit_ns) {
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0;; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(phase)
            : "memory");
        if (done) return true;
        if (it > 64) __nanosleep(64);
        if ((it & 63u) == 63u && global_ns() - t0 > limit_ns) return false;
    }
}

// The bulk-copy wait's limit: two seconds, far beyond any copy's time (one
// slab of at most a few hundred KB); 20 ms under the copy-stall test hook, so
// a test that makes every wait run out stays short.
constexpr uint64_t kCopyWaitNs = 2000000000ull, kCopyWaitInjectedNs = 20000000ull;

// tells the mbarrier's current phase how many bytes to expect
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// one bulk copy whose bytes the mbarrier has been told to expect
__device__ __forceinline__ void bulk_copy_in(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// TMA bulk copy global -> shared, completion counted in bytes on `bar`
// (`expect` = bytes, or more under the test hook above)
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint32_t expect,
                                          uint64_t* bar) {
    mbar_expect(bar, expect);
    bulk_copy_in(smem_dst, gsrc, bytes, bar);
}

// TMA bulk copy shared -> global, waited for before the buffer is reused
__device__ __forceinline__ void bulk_store_wait(void* gdst, const void* smem_src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(smem_src)),
                 "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace fs3d
