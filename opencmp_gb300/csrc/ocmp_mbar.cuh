// Shared-memory barriers (mbarrier) and bulk copies of the kernels that stage their operands
// asynchronously. Every wait is bounded.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ocmp {

constexpr long long kWaitCycles = 2000000000LL;     // about one second at the boost clock

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait; false when it gave up or another role already did (*abort)
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, volatile int* abort) {
    const long long t0 = clock64();
    while (!mbar_try(a, parity)) {
        if (*abort) return false;
        if (clock64() - t0 > kWaitCycles) return false;
    }
    return true;
}
// bytes (a multiple of 16) from 16-byte-aligned global to 16-byte-aligned shared memory; completes on mbar
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(mbar)
                 : "memory");
}

}  // namespace ocmp
