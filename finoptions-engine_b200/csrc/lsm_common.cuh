// lsm_common.cuh - device building blocks shared by the single-contract and batch LSM kernels:
// the seeded path simulation with event phases, deterministic
// warp / CTA / grid reductions, the exercise rule and the in-the-money power-sum accumulator.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "lsm_device.cuh"
#include "lsm_normals.cuh"

namespace fo {

constexpr unsigned long long kNone = ~0ull;

// A kernel launched by launch_early (lsm_kernels.h) may start before the one ahead of it in the stream has
// ended: it touches nothing of its, nor of any earlier one's, before await_prior_grid. let_next_grid_start
// lets it start as soon as every CTA of this one has; without it, when they leave. Kernels that fill SMs
// unevenly do not call it: the next one's CTAs would crowd onto the free SMs (65,536 paths of 52 weeks: 273 us
// for a contract's kernels with it in the backward pass, 248 without, 256 one kernel after the other).
__device__ __forceinline__ void await_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_grid_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// Seeded path simulation
// ---------------------------------------------------------------------------------------------

struct SimResult {
    int code;  // 0 ok, kNormalRejection, 3 non-finite transition
    int interval;
    double spot;
    double normal;
};

// One GBM step by a growth factor: the state after it, or false for a non-finite transition. A finite
// product of non-negative factors has a high word below the exponent's, so one integer comparison
// passes it; the absorbed state (0 times an overflowed factor) and the failures take the branch.
__device__ __forceinline__ bool gbm_step(double spot, double growth, double* next) {
    *next = spot * growth;
    if (uint32_t(__double2hiint(*next)) < 0x7ff00000u) return true;
    if (spot == 0.0) *next = 0.0;
    return fo_isfinite(*next);
}

// Simulates one path; calls store(row, value) at every observation, step(i, coefficients, normal,
// growth) after every interval and cash(node, state before, amount) after every cash dividend.
// Mirrors simulate_one_seeded (seeded.rs:399-459) including the terminal-dividend phase order.
// kInline: a chunk's four steps are unrolled; otherwise (an observer of hundreds of instructions) they
// loop, with the growth factors parked in shared memory. C: steps a chunk, 2 for paths of at most two
// intervals (half the normals and exponentials of a chunk of four would be thrown away). A chunk's normals and growth
// factors are formed side by side (they do not depend on the state): the four exponentials share
// the polynomial's constants, which a kernel of this register budget otherwise sets up again for
// each of them (25 of a step's 62 instructions measured).
struct IgnoreStep {
    __device__ __forceinline__ void operator()(uint32_t, const StepCoef&, double, double) const {}
};
struct IgnoreCash {
    __device__ __forceinline__ void operator()(uint32_t, double, double) const {}
};

template <bool kInline = true, int C = kChunkNormals, int T, typename Store, typename Step = IgnoreStep,
          typename Cash = IgnoreCash>
__device__ __forceinline__ SimResult simulate_path(const DevicePlan& plan, NormalSmem<T>& normals,
                                                   const PhiloxKeys& keys, uint32_t domain, uint32_t path,
                                                   Store&& store, Step&& step = Step{}, Cash&& cash = Cash{}) {
    const uint32_t intervals = plan.intervals;
    NormalStream<T> s;
    s.init(normals, domain, path);
    double spot = plan.sim_start;
    SimResult r{0, 0, 0.0, 0.0};
    if (plan.row_node[0] == 0) store(0, spot);
    for (uint32_t i = 0; i < intervals; i += C) {
        double z[C], growth[C];
        if (!s.template next<C>(keys, i, intervals, z)) {
            r.code = kNormalRejection;
            r.interval = int(i);
            return r;
        }
#pragma unroll
        for (uint32_t j = 0; j < C; ++j) {
            const StepCoef c = plan.steps[i + j];  // padded to whole chunks
            growth[j] = fo_exp(fo_fma(c.diffusion, z[j], c.log_drift));
        }
        if constexpr (!kInline) {
#pragma unroll
            for (uint32_t j = 0; j < C; ++j) normals.parked[j][threadIdx.x] = growth[j];
        }
        const auto advance = [&](uint32_t j, double factor, double normal) -> bool {
            double next;
            if (!gbm_step(spot, factor, &next)) {
                r.code = 3;
                r.interval = int(i + j);
                r.spot = spot;
                r.normal = normal;
                return false;
            }
            step(i + j, plan.steps[i + j], normal, factor);
            spot = next;
            const NodeEvent ev = plan.events[i + j + 1];
            const auto pay = [&] {
                const double before = spot;
                spot = apply_cash_dividend(plan.policy, ev.dividend_amount, before);
                cash(i + j + 1, before, ev.dividend_amount);
            };
            const int32_t phase = ev.flags & (kEventDividend | kEventTerminal);
            if (phase == (kEventDividend | kEventTerminal)) pay();
            if (ev.row >= 0) store(ev.row, spot);
            if (phase == kEventDividend) pay();
            return true;
        };
        if constexpr (kInline) {
#pragma unroll
            for (uint32_t j = 0; j < C; ++j) {
                if (j > 0 && i + j >= intervals) return r;
                if (!advance(j, growth[j], z[j])) return r;
            }
        } else {
            const uint32_t steps = min(uint32_t(C), intervals - i);
#pragma unroll 1
            for (uint32_t j = 0; j < steps; ++j)
                if (!advance(j, normals.parked[j][threadIdx.x], s.normal(i + j))) return r;
        }
    }
    return r;
}

// simulate_path for caller-supplied standard normals: normals[i * paths + path] drives interval i
// (GbmPathPlan::simulate with an external shock matrix, path.rs:139-175). The buffer was checked for
// non-finite values before the launch; only a non-finite transition fails here.
template <typename Store>
__device__ __forceinline__ SimResult simulate_path_external(const DevicePlan& plan, const double* normals,
                                                            uint64_t paths, uint64_t path, Store&& store) {
    double spot = plan.sim_start;
    SimResult r{0, 0, 0.0, 0.0};
    if (plan.row_node[0] == 0) store(0, spot);
    for (uint32_t i = 0; i < plan.intervals; ++i) {
        const double z = normals[uint64_t(i) * paths + path];
        const StepCoef c = plan.steps[i];
        const double next = gbm_advance(spot, c.diffusion, c.log_drift, z);
        if (!fo_isfinite(next)) {
            r.code = 3;
            r.interval = int(i);
            r.spot = spot;
            r.normal = z;
            return r;
        }
        spot = next;
        const NodeEvent ev = plan.events[i + 1];
        const bool dividend = (ev.flags & kEventDividend) != 0;
        const bool terminal = (ev.flags & kEventTerminal) != 0;
        if (dividend && terminal) spot = apply_cash_dividend(plan.policy, ev.dividend_amount, spot);
        if (ev.row >= 0) store(ev.row, spot);
        if (dividend && !terminal) spot = apply_cash_dividend(plan.policy, ev.dividend_amount, spot);
    }
    return r;
}

// ---------------------------------------------------------------------------------------------
// Reductions
// ---------------------------------------------------------------------------------------------

constexpr int kSlots = 16;  // T_0..T_8, U_0..U_4, non-finite count, spare
constexpr int kBadSlot = kMomentSlots;  // in-the-money paths with a non-finite predictor or response


// Butterfly "transpose" reduction of S values across a warp: at each stage a lane keeps half of
// its remaining values and adds its partner's copy of that half, so S values need S - 1 + log2
// shuffles instead of 5 S. Lane l ends holding the warp total of value (l % S) (S a power of two
// no larger than 32).
template <int S>
__device__ __forceinline__ double warp_transpose_reduce(double (&v)[S]) {
    const int lane = threadIdx.x & 31;
    double buf[S];
#pragma unroll
    for (int k = 0; k < S; ++k) buf[k] = v[k];
#pragma unroll
    for (int half = S / 2; half >= 1; half >>= 1) {
        // partner offset = half; lanes with (lane & half) keep the upper half.
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const double send = upper ? buf[k] : buf[k + half];
            const double keep = upper ? buf[k + half] : buf[k];
            buf[k] = keep + __shfl_xor_sync(0xffffffffu, send, half);
        }
    }
    double total = buf[0];
#pragma unroll
    for (int off = S; off < 32; off <<= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
    return total;
}


__device__ __forceinline__ dd shfl_dd_down(dd v, int off) {
    dd o;
    o.hi = __shfl_down_sync(0xffffffffu, v.hi, off);
    o.lo = __shfl_down_sync(0xffffffffu, v.lo, off);
    return o;
}

// The sum of red[w * S + slot] over the CTA's warps w, in double-double by the same tree for every slot:
// emit(slot, sum) by one lane each. A slot takes as many lanes as there are warps, so a warp of a CTA of
// eight combines four slots at once in three additions, where 16 slots took it two trees of five
// (the upper levels of a 32-lane tree only add zeros): fits of 4,096 states x 8 strikes 166.9 -> 164.4 ms,
// the moments of 4,096 paths 18.2 -> 16.7 us.
template <int S, typename Emit>
__device__ __forceinline__ void combine_warps(const double* red, Emit&& emit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int width = warps <= 8 ? 8 : warps <= 16 ? 16 : 32, slots = 32 / width;
    for (int first = warp * slots; first < S; first += warps * slots) {
        const int slot = first + lane / width, from = lane % width;
        dd v = dd_make(slot < S && from < warps ? red[from * S + slot] : 0.0);
        for (int off = width / 2; off > 0; off >>= 1) v = dd_add(v, shfl_dd_down(v, off));
        if (from == 0 && slot < S) emit(slot, v);
    }
}

// Warp sums in double, combined across the CTA's warps in double-double into the CTA partial.
template <int S>
__device__ __forceinline__ void cta_reduce_to(double (&acc)[S], double* smem /* [32 * S] */, double2* dst,
                                              size_t slot_stride = 1) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double total = warp_transpose_reduce<S>(acc);
    // lane l holds value l % S: lanes 0..S-1 publish
    if (lane < S) smem[warp * S + lane] = total;
    __syncthreads();
    combine_warps<S>(smem, [&](int slot, dd v) { dst[size_t(slot) * slot_stride] = make_double2(v.hi, v.lo); });
    __syncthreads();
}

// Slot `slot` of partials[b * S + slot] summed over b in a fixed order, by one warp; lane 0 has the sum.
template <int S>
__device__ __forceinline__ dd sum_slot(const double2* partials, int blocks, int slot) {
    const int lane = threadIdx.x & 31;
    // Issue the first eight partials of this lane before adding any, so their L2 latencies overlap; the
    // additions keep the fixed block order.
    constexpr int kBatch = 8;
    double2 v[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
        const int b = lane + 32 * i;
        v[i] = b < blocks ? __ldcg(&partials[b * S + slot]) : make_double2(0.0, 0.0);
    }
    dd acc = dd_make(0.0);
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
        if (lane + 32 * i < blocks) acc = dd_add(acc, dd{v[i].x, v[i].y});
    for (int b = lane + 32 * kBatch; b < blocks; b += 32) {
        const double2 w = __ldcg(&partials[b * S + slot]);
        acc = dd_add(acc, dd{w.x, w.y});
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc = dd_add(acc, shfl_dd_down(acc, off));
    return acc;
}

// The first S slots by as many warps of a CTA.
template <int S>
__device__ __forceinline__ void grid_combine(const double2* partials, int blocks, dd* out /* smem [S] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < S) {
        const dd acc = sum_slot<S>(partials, blocks, warp);
        if (lane == 0) out[warp] = acc;
    }
    __syncthreads();
}

// CTA reduction of S per-thread doubles to double-double totals in shared memory. Warp sums are
// formed in double by the transpose reduction, then combined over the CTA's warps in double-double in a
// fixed order, so the totals do not depend on timing.
template <int S>
__device__ __forceinline__ void cta_reduce_dd(double (&acc)[S], double* red /* [32 * S] */, dd* out /* [S] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double total = warp_transpose_reduce<S>(acc);
    if (lane < S) red[warp * S + lane] = total;
    __syncthreads();
    combine_warps<S>(red, [&](int slot, dd v) { out[slot] = v; });
    __syncthreads();
}

__device__ __forceinline__ bool exercise_rule(int tie_rule, double intrinsic, double continuation) {
    return tie_rule == 0 ? intrinsic > continuation : intrinsic >= continuation;
}

// Whether a spot is below kRuleSpotLimit, by its high word (spots are not negative).
constexpr uint32_t kRuleLimitHigh = 0x4c700000u;
static_assert(kRuleSpotLimit == 0x1p200, "high word 0x4c700000");
__device__ __forceinline__ bool within_rule(double spot) { return uint32_t(__double2hiint(spot)) < kRuleLimitHigh; }

// The decision of an in-the-money spot that the row's ExerciseRule does not cover. No ordinary market
// gets here, but it stays in line: a call in a path loop costs the loop's registers.
enum Decision : int { kDecideContinue = 0, kDecideExercise = 1, kDecideNonFinite = 2 };

template <int D>
__device__ __forceinline__ int decide_general(const FitModel* model, double spot, double strike, int tie_rule) {
    double continuation;
    if (!predict_continuation_d<D>(*model, divide(spot, make_divisor(strike)), &continuation)) return kDecideNonFinite;
    return exercise_rule(tie_rule, spot - strike, continuation) ? kDecideExercise : kDecideContinue;
}

struct RowSums {
    double acc[kSlots];
};

// A non-negative number's finiteness by its high word (a NaN or an infinity has it at the exponent's
// maximum or, with the sign set, above).
__device__ __forceinline__ bool finite_nonnegative(double v) { return uint32_t(__double2hiint(v)) < 0x7ff00000u; }

// The sums of one in-the-money path but for its count (acc[0]).
__device__ __forceinline__ void accumulate_centred(RowSums& r, double t, double y) {
    double pw = t;
    r.acc[kPowerSums] += y;
#pragma unroll
    for (int k = 1; k < kPowerSums; ++k) {
        r.acc[k] += pw;
        if (k < kResponseSums) r.acc[kPowerSums + k] = fo_fma(y, pw, r.acc[kPowerSums + k]);
        pw *= t;
    }
}

__device__ __forceinline__ void accumulate_moments(RowSums& r, double x, double y, double pivot) {
    accumulate_centred(r, x - pivot, y);
}

}  // namespace fo
