// lsm_bulk_copy.cuh - bulk copies (TMA) into shared memory, completed on an mbarrier, and the bounded wait for
// one.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "lsm_sync.cuh"

namespace fo {

__device__ __forceinline__ uint32_t shared_address(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbarrier_init(uint64_t* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(bar)), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Source, destination and size are multiples of 16 bytes (the caller rounds).
__device__ __forceinline__ void bulk_load(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes)
                 : "memory");
    if (bytes > 0)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                shared_address(smem)),
            "l"(gmem), "r"(bytes), "r"(shared_address(bar))
            : "memory");
}
__device__ __forceinline__ bool mbarrier_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(shared_address(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// One thread's wait for the copies expected on `bar`. It gives up by the clock alone, after limit_ns, and then
// raises status->barrier_timeout: a timeout raised elsewhere is no reason to leave, because a copy in
// flight still writes this CTA's shared memory. One that has not ended by then is left behind.
__device__ __forceinline__ bool wait_bulk(uint64_t* bar, uint32_t parity, DeviceStatus* status,
                                          unsigned long long limit_ns = kBarrierTimeoutNs) {
    if (mbarrier_try_wait(bar, parity)) return true;
    const unsigned long long start = global_timer_ns();
    while (!mbarrier_try_wait(bar, parity)) {
        if (global_timer_ns() - start <= limit_ns) continue;
        atomicExch(&status->barrier_timeout, 1u);
        return false;
    }
    return true;
}

}  // namespace fo
