// lsm_sync.cuh - bounded waits between CTAs that run at the same time. Every wait gives up after a time
// limit and raises status->barrier_timeout, so a CTA that never arrives ends the kernel with an
// error the host reports, not a hang.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "lsm_device.cuh"

namespace fo {

__device__ __forceinline__ unsigned ld_volatile_u32(const unsigned* p) {
    return *(const volatile unsigned*)p;
}

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ld_relaxed_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// A warp's patience in a polling loop (all CTAs co-resident: cooperative launch). Every lane calls
// again() after each unsuccessful poll, however the lanes entered the loop; lane 0 looks at the
// clock every 256 polls and its decision is broadcast. False once `limit_ns` has passed, which
// raises status->barrier_timeout, or another waiter has raised it: the warp gives up, and every CTA
// leaves at its next wait.
constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;
struct BoundedWait {
    DeviceStatus* st;
    unsigned long long limit_ns;
    unsigned spins;
    unsigned long long start;

    __device__ __forceinline__ explicit BoundedWait(DeviceStatus* status, unsigned long long limit = kBarrierTimeoutNs)
        : st(status), limit_ns(limit), spins(0), start(0) {}
    __device__ __forceinline__ bool again() {
        if ((++spins & 255u) != 0) return true;
        int give_up = 0;
        if ((threadIdx.x & 31) == 0) {
            give_up = ld_volatile_u32(&st->barrier_timeout) != 0;
            const unsigned long long now = global_timer_ns();
            if (start == 0) {
                start = now;
            } else if (now - start > limit_ns) {
                atomicExch(&st->barrier_timeout, 1u);
                give_up = 1;
            }
        }
        return __shfl_sync(0xffffffffu, give_up, 0) == 0;
    }
};

// Warp-wide wait until status->arrivals reaches `target`: lane 0 reads it and every decision is taken on its
// broadcast value. False (in every lane) when the wait gave up. No kernel of the engine counts arrivals
// between CTAs any more (lsm_exchange.cuh polls the values themselves); the bounded-wait test runs it.
__device__ inline bool wait_arrivals(DeviceStatus* st, unsigned target,
                                     unsigned long long limit_ns = kBarrierTimeoutNs) {
    BoundedWait wait(st, limit_ns);
    __syncwarp();
    for (;;) {
        unsigned seen = 0;
        if ((threadIdx.x & 31) == 0) seen = ld_relaxed_gpu(&st->arrivals);
        if (__shfl_sync(0xffffffffu, seen, 0) >= target) break;
        if (!wait.again()) return false;
    }
    __threadfence();
    return true;
}

}  // namespace fo
