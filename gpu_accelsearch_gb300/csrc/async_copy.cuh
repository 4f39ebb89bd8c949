// async_copy.cuh -- mbarriers with bounded waits and bulk asynchronous copies
// (TMA) into and out of shared memory.
#pragma once

#include <cuda.h>

#include "accel_common.cuh"

namespace accel {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// Wait for the barrier's phase with the thread suspended (no polling
// instructions), at most about 1 us per try; false after 2^15 tries (tens
// of milliseconds), far beyond any copy of a tile.
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity), "r"(1000u)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity) {
#pragma unroll 1
    for (int it = 0; it < (1 << 15); it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// One box of a 3-D tensor map (coordinates x = column, y = row, z =
// segment) into shared memory (128-byte aligned); elements past the
// tensor's edges arrive as zeros and count toward the transaction bytes.
__device__ __forceinline__ void tensor_copy_g2s(void* sdst, const CUtensorMap* map, int x, int y, int z,
                                                unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(smem_addr(sdst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// bytes (a multiple of 16) from global to shared, both 16-byte aligned
__device__ __forceinline__ void bulk_copy_g2s(void* sdst, const void* gsrc, unsigned bytes,
                                              unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(sdst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// bytes (a multiple of 16) from shared to global, both 16-byte aligned; the
// writers of the shared bytes have fenced (fence_async_proxy) and met at a
// barrier.  bulk_s2g_wait_read: the issuing thread's copies have read their
// shared memory (the stores themselves are complete when the kernel is).
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_copy_s2g(void* gdst, const void* ssrc, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gdst), "r"(smem_addr(ssrc)),
                 "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_s2g_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
}

}  // namespace accel
