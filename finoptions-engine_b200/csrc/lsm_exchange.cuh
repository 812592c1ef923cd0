// lsm_exchange.cuh - grid-wide sums between the co-resident CTAs of the backward pass.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fo_core.cuh"
#include "lsm_common.cuh"
#include "lsm_sync.cuh"

namespace fo {

constexpr int kExchangeSlots = 8;               // sums a CTA sends: six in use, two spare
constexpr int kUsedSlots = 6;
constexpr int kExchangeWarps = 8;
constexpr int kExchangeLoads = 5;                // CTA lines a lane reads together (148 CTAs: one round)

// Grid-wide sums. A CTA's totals travel as one line of eight 16-byte double-doubles whose lowest bits are
// the exchange's phase (moving hi's lowest bit into lo costs nothing, lo loses 2^-105 of the sum), so
// a reader that sees the phase in both halves has the value: no counter is written, fenced and
// waited for first. Two buffers alternate and a buffer's phase flips each time it is reused; a CTA
// writes exchange s + 2 only after reading s + 1 from every CTA, which each wrote only after it
// had read s.
// The totals keep some hundred bits of the binary64 numbers they sum and round to the number nearest to
// the exact sum, as those of dd_add do; with dd_add throughout, and the displaced bits sent beside, a row
// took 1.1 us longer (2^20 paths: 357 us a pass against 302).
__device__ __forceinline__ double2 with_phase(dd v, uint64_t phase) {
    const double hi = bits_to_double((double_to_bits(v.hi) & ~1ull) | phase);
    const double lo = v.lo + (v.hi - hi);
    return make_double2(hi, bits_to_double((double_to_bits(lo) & ~1ull) | phase));
}
__device__ __forceinline__ void store_relaxed(double2* p, double2 v) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ double2 load_relaxed(const double2* p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool has_phase(double2 v, uint64_t phase) {
    return (double_to_bits(v.x) & 1ull) == phase && (double_to_bits(v.y) & 1ull) == phase;
}
// Adds a double-double to a running sum whose parts are renormalised once at the end: the chain of
// high parts is one addition a step.
__device__ __forceinline__ void add_to(dd& sum, dd v) {
    const dd s = two_sum(sum.hi, v.hi);
    sum.hi = s.hi;
    sum.lo = (sum.lo + v.lo) + s.lo;
}
__device__ __forceinline__ dd shfl_dd_xor(dd v, int mask) {
    return dd{__shfl_xor_sync(0xffffffffu, v.hi, mask), __shfl_xor_sync(0xffffffffu, v.lo, mask)};
}
// Sums over the four lanes that hold the same slot (lane & 7); every lane ends with its slot's sum.
__device__ __forceinline__ dd slot_sum(dd v) {
    // The lower lane's value first on both sides, so that both form the same sum.
#pragma unroll
    for (int mask = kExchangeSlots; mask < 32; mask <<= 1) {
        const dd o = shfl_dd_xor(v, mask);
        const bool upper = (threadIdx.x & mask) != 0;
        dd first = upper ? o : v;
        add_to(first, upper ? v : o);
        v = first;
    }
    return fast_two_sum(v.hi, v.lo);
}

// Shared memory of a CTA of kWarps warps.
template <int kWarps>
struct ExchangeSmem {
    double red[kWarps][kExchangeSlots];        // per warp and slot
    dd share[kExchangeWarps][kExchangeSlots];  // the exchange warps' shares of the grid's totals
    int failed;                                // a wait gave up (the caller clears it)
};

// The grid's totals from the CTAs' per-warp sums (sm.red), by the first kExchangeWarps warps of each, which meet
// at named barrier 1: warp 0 sends this CTA's totals (CTA `block` of `blocks`), all read the others',
// and warp 0 adds the warps' shares. `partials` holds exchange_words(blocks) words, zero before exchange 0.
// Returns slot (lane & 7) in every lane of warp 0. sm.failed is set when a wait gave up.
template <int kWarps>
__device__ __forceinline__ dd exchange_totals(ExchangeSmem<kWarps>& sm, double2* partials, int block, int blocks,
                                              unsigned seq, DeviceStatus* status,
                                              unsigned long long limit_ns = kBarrierTimeoutNs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = lane & (kExchangeSlots - 1);
    double2* buffer = partials + size_t(seq & 1u) * kExchangeSlots * blocks;
    const uint64_t phase = ((seq >> 1) & 1u) ^ 1u;  // the buffers start at phase 0
    dd total = dd_make(0.0);
    if (warp == 0) {
        constexpr int kShare = kWarps * kExchangeSlots / 32;  // warp sums a lane adds
        double mine[kShare];
#pragma unroll
        for (int i = 0; i < kShare; ++i) mine[i] = sm.red[lane / kExchangeSlots + i * (32 / kExchangeSlots)][slot];
#pragma unroll
        for (int i = 0; i < kShare; ++i) add_to(total, dd_make(mine[i]));
        total = slot_sum(total);
        if (blocks > 1 && lane < kUsedSlots)
            store_relaxed(&buffer[size_t(block) * kExchangeSlots + slot], with_phase(total, phase));
    }
    if (blocks == 1) return total;
    dd sum = dd_make(0.0);
    constexpr int kCtasPerWarp = 32 / kExchangeSlots, kRound = kExchangeWarps * kCtasPerWarp;
    for (int first = 0; first < blocks; first += kRound * kExchangeLoads) {
        double2 v[kExchangeLoads];
        unsigned missing = 0;  // loads of this lane without their value yet
#pragma unroll
        for (int i = 0; i < kExchangeLoads; ++i) {
            const int b = first + i * kRound + warp * kCtasPerWarp + lane / kExchangeSlots;
            v[i] = make_double2(0.0, 0.0);
            if (b < blocks && slot < kUsedSlots) missing |= 1u << i;
        }
        BoundedWait wait(status, limit_ns);
        for (;;) {
#pragma unroll
            for (int i = 0; i < kExchangeLoads; ++i) {
                const int b = first + i * kRound + warp * kCtasPerWarp + lane / kExchangeSlots;
                if ((missing >> i) & 1u) v[i] = load_relaxed(&buffer[size_t(b) * kExchangeSlots + slot]);
            }
#pragma unroll
            for (int i = 0; i < kExchangeLoads; ++i)
                if (has_phase(v[i], phase)) missing &= ~(1u << i);
            if (__all_sync(0xffffffffu, missing == 0)) break;
            if (!wait.again()) {
                if (lane == 0) sm.failed = 1;
                break;
            }
        }
#pragma unroll
        for (int i = 0; i < kExchangeLoads; ++i) add_to(sum, dd{v[i].x, v[i].y});
    }
    sum = slot_sum(sum);
    if (lane < kExchangeSlots) sm.share[warp][slot] = sum;
    named_barrier_sync(1, kExchangeWarps * 32);
    if (warp != 0) return sum;
    dd grid = sm.share[lane / kExchangeSlots][slot];
    add_to(grid, sm.share[lane / kExchangeSlots + 4][slot]);
    static_assert(kExchangeWarps == 8 && kExchangeSlots == 8, "two shares a lane");
    return slot_sum(grid);
}

}  // namespace fo
