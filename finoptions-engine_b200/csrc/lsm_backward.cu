// lsm_backward.cu - the backward induction of one contract (policy.rs:215-296, 471-601).
//
//   moments_kernel    every fitted row's regression but for its responses: in-the-money count, mean,
//                     scale, recurrence and norms depend on the simulated states alone, so all rows
//                     are reduced and solved side by side.
//   backward_kernel   the serial part, a persistent cooperative kernel: per row one grid-wide exchange of
//                     the response sums R_k = sum y z^k (k <= degree), a small matrix product for the
//                     coefficients, and the exercise rule applied to every path.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "lsm_bulk_copy.cuh"
#include "lsm_common.cuh"
#include "lsm_device.cuh"
#include "lsm_exchange.cuh"
#include "lsm_fit_warp.cuh"
#include "lsm_kernels.h"
#include "lsm_row_solve.cuh"
#include "lsm_sync.cuh"

namespace fo {

// Double-double sum over a warp in a fixed order, in lane 0. The low parts are summed beside the
// high ones and folded in once, so a level costs a shuffle and one dependent addition.
__device__ __forceinline__ dd warp_sum_dd(dd v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const dd o = shfl_dd_down(v, off);
        const dd s = two_sum(v.hi, o.hi);
        v.hi = s.hi;
        v.lo = (v.lo + o.lo) + s.lo;
    }
    return fast_two_sum(v.hi, v.lo);
}

// In-the-money moneyness: the correctly rounded quotient by the strike.
__device__ __forceinline__ double moneyness(double spot, const Divisor& strike) {
    const double x = strike.inv != 0.0 ? divide_above(spot, strike) : spot / strike.b;
    return finite_nonnegative(x) ? x : spot / strike.b;
}

// ---------------------------------------------------------------------------------------------
// Moments of every fitted row.
// ---------------------------------------------------------------------------------------------

// A grid of a.blocks CTAs per row, each over a contiguous range of paths; a row's last CTA adds the
// CTA totals in order, solves the row (lsm_fit_warp.cuh with zero responses) and writes its record.
// The power sums are taken about the in-the-money mean of the row's first thousand paths, which
// lies within a fraction of a standard deviation of the row's. Where it does not (a few in-the-money
// paths), the row's sums are taken again about its own mean: by the last CTA alone, or by a second
// launch (kAgain) where the caller announced one, whose CTAs leave at once for every other row. 52 weeks, 2^20
// paths, strike at 1.6 times the spot: 1,906 us a call by the last CTA, 1,308 so.
// It reads the stored rows once, at about half the FP64 rate and half of HBM's: 2^20 paths x 51 rows take
// 143 us, 200 us with every power added by itself.
constexpr int kMomentThreads = 256;
constexpr int kMomentCtasPerSm = 4;
constexpr int kPivotLoads = 4;  // the pivot's sample: the row's first kPivotLoads * kMomentThreads paths
constexpr int kHugeSlot = kBadSlot + 1;  // in-the-money paths beyond kRuleSpotLimit

// A path's t is its correctly rounded quotient by the strike less the pivot. (One fma with the strike's
// reciprocal takes 10 us less at 2^20 paths x 51 rows, but shifts every path, and so the recorded mean,
// by the reciprocal's rounding.)
template <int D>
__device__ __forceinline__ void add_row_moments(RowSums& s, uint32_t& itm, const double* spots, uint64_t lo, uint64_t hi,
                                                const Divisor& Kd, double pivot, uint32_t order,
                                                unsigned long long* nonfinite) {
    constexpr int kLoads = 4;
    const bool divides = !(Kd.b > 0x1p-800);  // a quotient could overflow, or there is no reciprocal
    for (uint64_t base = lo + threadIdx.x; base < hi; base += kLoads * kMomentThreads) {
        double sp[kLoads];
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const uint64_t p = base + uint64_t(u) * kMomentThreads;
            sp[u] = p < hi ? __ldg(&spots[p]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            if (!(sp[u] > Kd.b)) continue;
            double x = divide_above(sp[u], Kd);
            if (divides || !within_rule(sp[u])) {
                x = sp[u] / Kd.b;
                if (!finite_nonnegative(x)) {
                    s.acc[kBadSlot] += 1.0;
                    if (nonfinite)
                        atomicMin(nonfinite, ((unsigned long long)order << 32) | (base + uint64_t(u) * kMomentThreads));
                    continue;
                }
                if (!within_rule(sp[u])) s.acc[kHugeSlot] += 1.0;
            }
            const double t = x - pivot;
            itm += 1;
            // T_1 .. T_2D: the powers up to t^D are formed, the higher ones are products of two of them
            // added in one fma.
            double power[D + 1];
            power[0] = 1.0;
#pragma unroll
            for (int k = 1; k <= D; ++k) {
                power[k] = k == 1 ? t : power[k / 2] * power[k - k / 2];
                s.acc[k] += power[k];
            }
#pragma unroll
            for (int k = 1; k <= D; ++k) s.acc[D + k] = fo_fma(power[D], power[k], s.acc[D + k]);
        }
    }
}

template <int D, bool kAgain>
__global__ void __launch_bounds__(kMomentThreads, kMomentCtasPerSm) moments_kernel(MomentArgs a) {
    __shared__ double red[32 * kSlots];
    __shared__ dd total[kSlots];
    __shared__ FitModel model;
    __shared__ int last;
    const DevicePlan& plan = a.plan;
    if (!kAgain && blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < a.exchange_words; i += blockDim.x) a.exchange[i] = make_double2(0.0, 0.0);
    if (*(const volatile unsigned long long*)&a.status->train_sim_fail != kNone) return;
    const uint32_t E = plan.rows - 1;
    const uint32_t row = (plan.origin_row ? 1u : 0u) + blockIdx.y;
    const uint32_t order = E - 1 - row;
    const uint64_t P = plan.train_paths;
    const double* spots = a.slab + uint64_t(row - plan.first_stored_row) * P;
    const Divisor Kd = make_divisor(plan.strike);
    FitRecord& rec = a.records[row];
    double pivot = 1.0;
    if constexpr (kAgain) {
        if (rec.again == 0) return;
        pivot = rec.pivot;
    } else if constexpr (D > 0) {
        double loc[2] = {0.0, 0.0}, sample[kPivotLoads];
#pragma unroll
        for (int u = 0; u < kPivotLoads; ++u) {
            const uint64_t p = threadIdx.x + u * kMomentThreads;
            sample[u] = p < P ? __ldg(&spots[p]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kPivotLoads; ++u) {
            if (!(sample[u] > Kd.b)) continue;
            const double x = moneyness(sample[u], Kd);
            if (!finite_nonnegative(x)) continue;
            loc[0] += 1.0;
            loc[1] += x;
        }
        cta_reduce_dd<2>(loc, red, total);
        if (total[0].hi > 0.0) pivot = dd_round(dd_div(total[1], total[0]));
        __syncthreads();
    }
    RowSums s;
#pragma unroll
    for (int k = 0; k < kSlots; ++k) s.acc[k] = 0.0;
    uint32_t itm_paths = 0;
    const uint64_t span = (P + gridDim.x - 1) / gridDim.x;
    const uint64_t lo = min(P, span * blockIdx.x), hi = min(P, lo + span);
    add_row_moments<D>(s, itm_paths, spots, lo, hi, Kd, pivot, order, kAgain ? nullptr : &a.status->fit_nonfinite);
    s.acc[0] = double(itm_paths);
    cta_reduce_dd<kSlots>(s.acc, red, total);
    if (gridDim.x > 1) {
        double2* mine = a.partials + (size_t(blockIdx.y) * gridDim.x) * kSlots;
        if (threadIdx.x < kSlots)
            mine[size_t(blockIdx.x) * kSlots + threadIdx.x] = make_double2(total[threadIdx.x].hi, total[threadIdx.x].lo);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(&rec.arrived, 1u) + 1u == gridDim.x;
        __syncthreads();
        if (!last) return;
        __threadfence();
        const int lane = threadIdx.x & 31;
        for (int slot = threadIdx.x >> 5; slot < kSlots; slot += kMomentThreads / 32) {
            dd v = dd_make(0.0);
            for (unsigned b = lane; b < gridDim.x; b += 32) {
                const double2 w = __ldcg(&mine[size_t(b) * kSlots + slot]);
                v = dd_add(v, dd{w.x, w.y});
            }
            v = warp_sum_dd(v);
            if (lane == 0) total[slot] = v;
        }
        __syncthreads();
    }
    const uint64_t itm = uint64_t(total[0].hi), bad = uint64_t(total[kBadSlot].hi), population = itm + bad;
    const bool huge = total[kHugeSlot].hi > 0.0;
    const uint32_t required = uint32_t(D + 1);
    double mean = pivot;
    if (!kAgain && D > 0 && population >= required && bad == 0 && pivot_too_far(total, pivot, itm, &mean)) {
        pivot = mean;
        if (a.relaunch) {
            if (threadIdx.x == 0) {
                rec.pivot = pivot;
                rec.arrived = 0;
                rec.again = 1;
            }
            return;
        }
#pragma unroll
        for (int k = 0; k < kSlots; ++k) s.acc[k] = 0.0;
        itm_paths = 0;
        add_row_moments<D>(s, itm_paths, spots, 0, P, Kd, pivot, order, nullptr);
        s.acc[0] = double(itm_paths);
        __syncthreads();  // the totals were read above
        cta_reduce_dd<kSlots>(s.acc, red, total);
    }
    if (threadIdx.x >= 32) return;
    int kind;
    if (population == 0) {
        kind = plan.support == 1 ? kRuleContinue : kRuleNoSupport;
    } else if (population < required && plan.support == 1) {
        kind = kRuleContinue;
    } else if (population < required || bad > 0) {
        kind = kRuleFitFailed;  // InsufficientObservations / non-finite population
    } else {
        fit_continuation_warp(total, pivot, itm, D, plan.rank_tolerance, plan.rank_limit, &model);
        kind = model.status == kFitOk ? kRuleRegression : kRuleFitFailed;
        constexpr int kModelWords = int(sizeof(FitModel) / sizeof(double2));
        static_assert(sizeof(FitModel) % sizeof(double2) == 0, "FitModel is 16-byte aligned");
        if (threadIdx.x < kModelWords)
            reinterpret_cast<double2*>(&rec.model)[threadIdx.x] = reinterpret_cast<const double2*>(&model)[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        rec.kind = kind;
        rec.itm = population;
        rec.pivot = pivot;
        rec.beyond_rule = huge ? 1 : 0;
        rec.origin_continuation = 0.0;
        rec.diag_status = -1;
    }
}

// ---------------------------------------------------------------------------------------------
// The serial pass.
// ---------------------------------------------------------------------------------------------

constexpr int kFetchThread = (kExchangeWarps + 1) * 32;
static_assert(kUsedSlots == kMaxColumns + 1, "R_0..R_4 and the non-finite responses");
constexpr int kBadResponses = kMaxColumns;

struct BackwardSmem {
    ExchangeSmem<kBackwardThreads / 32> exchange;
    RowBasis basis[2];  // of the row being decided and of the row being staged, by row parity
    RowSolution row;    // of the row being decided
    int failed;         // the wait for a copy timed out
    uint64_t loaded;  // mbarrier of the staged row's spots
};

// The row's coefficients into its record, by one warp of CTA 0; and the failure of a row whose response sums
// leave no finite coefficient.
template <int D>
__device__ __forceinline__ void write_coefficients(const RowSolution& row, FitRecord& rec) {
    const int lane = threadIdx.x & 31;
    if (lane <= D) rec.model.coef[lane] = row.coef[lane];
    if (lane != 0 || row.kind == kRuleRegression) return;
    rec.kind = kRuleFitFailed;
    if (row.bad_responses) return;
    rec.model.status = kFitNonFinite;
    rec.model.aux = row.broken;
}

// A CTA owns ppt * blockDim consecutive paths, a thread every blockDim-th of them. When the population
// fits on chip (kHbm false), their discounted values, the current row's spots and the staged row's
// spots live in this CTA's shared memory for the whole backward pass, so the only HBM traffic is
// one read of each stored row, one bulk copy per CTA (8-byte asynchronous copies by every thread
// kept the load / store unit busy for 2,600 cycles a row, ahead of the exchange). Larger populations (kHbm true) keep each path's value in
// HBM at a.values[p] and read the spots straight from the stored rows; the arithmetic and its order
// are the same, so a path's decisions do not depend on where its value lives.
//
// A pass applies row k's rule to the thread's paths, discounts them to row k - 1
// (policy.rs:1049-1063) and adds row k - 1's response sums. Between passes the first eight
// warps exchange the sums, the ninth prepares the row after and a thread of the tenth fetches its spots.
// Bound by the latency of the row exchanges: a row takes 2.2 us at 4,096 paths (poll 0.4), 2.7 us at 65,536
// (0.8) and 5.8 us at 2^20 (1.8, the pass 2.1), against 9.5, 9.6 and 17.4 us when a row's moments were solved
// inside it, arrivals were counted and the totals read by slot. 512 threads instead of 1,024 halve the per-warp reduction and keep the rule
// and the sums in registers (2^20 paths: 0.29 ms against 0.36).
template <int D, bool kHbm>  // D == plan.degree (launch_backward dispatches on it)
__global__ void __launch_bounds__(kBackwardThreads, 1) backward_kernel(BackwardArgs a) {
    __shared__ BackwardSmem sm;
    extern __shared__ __align__(16) double backward_dyn[];
    const DevicePlan& plan = a.plan;
    if (*(const volatile unsigned long long*)&a.status->train_sim_fail != kNone)
        return;  // training simulation failed: every CTA reads the same word and leaves
    constexpr int T = kBackwardThreads;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t P = plan.train_paths;
    const uint64_t chunk = uint64_t(a.ppt) * T, first = blockIdx.x * chunk;
    const uint32_t paths = uint32_t(first < P ? min(chunk, P - first) : 0);  // this CTA's
    const int owned = int((paths + T - 1 - threadIdx.x) / T);               // this thread's
    // Two spot buffers alternate; each has room for the element that aligns a row's copy.
    double* values = backward_dyn;
    double* spots = backward_dyn + chunk;
    double* spots_next = spots + chunk + 2;
    const double K = plan.strike;
    const Divisor Kd = make_divisor(K);
    const uint32_t E = plan.rows - 1;
    const int lowest = plan.origin_row ? 1 : 0;
    auto row_ptr = [&](int row) { return a.slab + uint64_t(uint32_t(row) - plan.first_stored_row) * P + first; };
    // A row's copy starts at the 16-byte boundary at or below the CTA's first path.
    auto alignment = [&](const double* p) { return int((reinterpret_cast<uintptr_t>(p) >> 3) & 1u); };
    auto value = [&](int j) -> double& {
        if constexpr (kHbm) return a.values[first + uint64_t(j) * T + threadIdx.x];
        else return values[j * T + threadIdx.x];
    };
    {
        const double* terminal = row_ptr(int(E));
#pragma unroll 4
        for (int j = 0; j < owned; ++j) {
            const double d = __ldcs(&terminal[j * T + threadIdx.x]) - K;
            value(j) = d > 0.0 ? d : 0.0;
        }
    }
    if (threadIdx.x == 0) {
        sm.failed = 0;
        sm.exchange.failed = 0;
        sm.row.rule = never_exercise();
        mbarrier_init(&sm.loaded, 1);
    }
    double sums[kExchangeSlots];
    auto clear_sums = [&] {
#pragma unroll
        for (int k = 0; k < kExchangeSlots; ++k) sums[k] = 0.0;
    };
    // One thread starts a row's copy; its last element, when the copy's size is odd, travels by itself
    // and is published by the CTA barrier that follows.
    auto fetch = [&](int row) {
        if constexpr (!kHbm) {
            const double* src = row_ptr(row);
            const int shift = alignment(src);
            const uint32_t count = paths + shift;
            bulk_load(spots_next, src - shift, (count & ~1u) * uint32_t(sizeof(double)), &sm.loaded);
            if (count & 1u) spots_next[count - 1] = __ldcs(src - shift + count - 1);
        }
    };
    // The same thread waits for it, ahead of that barrier (every thread polling the mbarrier takes 600
    // cycles).
    uint32_t copies = 0;  // completed copies
    auto wait_copy = [&] {
        if constexpr (!kHbm) {
            if (!wait_bulk(&sm.loaded, copies & 1u, a.status)) sm.failed = 1;
            copies += 1;
        }
    };
    // Decides `row` (none when negative) and stages `next` (none when below the lowest fitted row),
    // whose order is `order`.
    auto pass = [&](int row, int next, uint32_t order) {
        const bool decide = row >= 0, stage = next >= lowest;
        const RowBasis& basis = sm.basis[next & 1];
        const ExerciseRule& rule = sm.row.rule;
        const double disc = stage ? basis.discount : 1.0;
        const double* cur_row = decide ? row_ptr(row) : nullptr;
        const double* next_row = stage ? row_ptr(next) : nullptr;
        const double* cur_spots = spots + (decide ? alignment(cur_row) : 0);
        const double* next_spots = spots_next + (stage ? alignment(next_row) : 0);
        const bool strict = plan.tie_rule == 0;
        if ((!decide || rule.general == 0) && (!stage || basis.general == 0)) {
            const double slope = basis.slope, shift = basis.shift;
            const auto loop = [&](auto decides, auto stages, auto strict_rule) {
                const ExerciseRule r = rule;  // held in registers across the pass
#pragma unroll 4
                for (int j = 0; j < owned; ++j) {
                    const int at = j * T + threadIdx.x;
                    double v = value(j);
                    if constexpr (decltype(decides)::value) {
                        const double d = (kHbm ? __ldcg(&cur_row[at]) : cur_spots[at]) - K;
                        const double c = rule_continuation<D>(r, d);
                        v = d > 0.0 && (decltype(strict_rule)::value ? d > c : d >= c) ? d : v;
                    }
                    if constexpr (decltype(stages)::value) {
                        const double d = (kHbm ? __ldcg(&next_row[at]) : next_spots[at]) - K;
                        v *= disc;
                        const double z = fo_fma(d, slope, shift);
                        const double y = d > 0.0 ? v : 0.0;
                        double pw = z;
                        sums[0] += y;
#pragma unroll
                        for (int k = 1; k <= D; ++k) {
                            sums[k] = fo_fma(y, pw, sums[k]);
                            if (k < D) pw *= z;
                        }
                        if (!finite_nonnegative(v)) {
                            const unsigned long long key = ((unsigned long long)order << 32) | (first + uint64_t(at));
                            atomicMin(&a.status->fit_payoff_fail, key);
                            if (d > 0.0) {
                                sums[kBadResponses] += 1.0;
                                atomicMin(&a.status->fit_nonfinite, key);
                            }
                        }
                    }
                    value(j) = v;
                }
            };
            using Yes = std::true_type;
            using No = std::false_type;
            if (decide && stage) {
                if (strict) loop(Yes{}, Yes{}, Yes{});
                else loop(Yes{}, Yes{}, No{});
            } else if (decide) {
                if (strict) loop(Yes{}, No{}, Yes{});
                else loop(Yes{}, No{}, No{});
            } else {
                loop(No{}, Yes{}, Yes{});
            }
            return;
        }
        // A row outside the rules' range: the same pass through the model itself.
        struct {
            double mean, scale, inv_scale, alpha[kMaxDegree], beta[kMaxDegree], coef[kMaxColumns];
        } model{};
        if (decide) {
            const RowBasis& b = sm.basis[row & 1];
            model.mean = b.mean;
            model.scale = b.scale;
            model.inv_scale = b.inv_scale;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                model.alpha[j] = b.alpha[j];
                model.beta[j] = b.beta[j];
            }
#pragma unroll
            for (int j = 0; j <= D; ++j) model.coef[j] = sm.row.coef[j];
        }
#pragma unroll 1
        for (int j = 0; j < owned; ++j) {
            const int at = j * T + threadIdx.x;
            const uint64_t p = first + uint64_t(at);
            double v = value(j);
            if (decide && sm.row.kind == kRuleRegression) {
                const double sp = kHbm ? __ldcg(&cur_row[at]) : cur_spots[at];
                if (sp > K) {
                    double continuation;
                    if (!predict_continuation_d<D>(model, divide(sp, Kd), &continuation))
                        atomicMin(&a.status->fit_predict_fail, ((unsigned long long)(order - 1) << 32) | p);
                    else if (exercise_rule(plan.tie_rule, sp - K, continuation))
                        v = sp - K;
                }
            }
            if (stage) {
                const double sp = kHbm ? __ldcg(&next_row[at]) : next_spots[at];
                v *= disc;
                const unsigned long long key = ((unsigned long long)order << 32) | p;
                if (!fo_isfinite(v)) atomicMin(&a.status->fit_payoff_fail, key);
                if (sp > K) {
                    if (!fo_isfinite(v)) {
                        sums[kBadResponses] += 1.0;
                        atomicMin(&a.status->fit_nonfinite, key);
                    } else {
                        const double z =
                            D == 0 ? 0.0 : divide(divide(sp, Kd) - basis.mean, Divisor{basis.scale, basis.inv_scale});
                        double pw = z;
                        sums[0] += v;
#pragma unroll
                        for (int k = 1; k <= D; ++k) {
                            sums[k] = fo_fma(v, pw, sums[k]);
                            if (k < D) pw *= z;
                        }
                    }
                }
            }
            value(j) = v;
        }
    };
    // The thread's sums to sm.exchange.red, slot by slot.
    auto reduce_warps = [&] {
        const double total = warp_transpose_reduce<kExchangeSlots>(sums);
        if (lane < kExchangeSlots) sm.exchange.red[warp][lane] = total;
        clear_sums();
    };
    const auto prepare = [&](int at) {
        prepare_basis<D>(a.records[at], K, plan.disc_from_later[at], &sm.basis[at & 1]);
    };
    clear_sums();
    unsigned seq = 0;
    uint32_t order = 0;
    int row = int(E) - 1;
    __syncthreads();  // the mbarrier is ready
    if (row >= lowest) {
        if (warp == kExchangeWarps) prepare(row);
        if (threadIdx.x == kFetchThread) {
            fetch(row);
            wait_copy();
        }
        __syncthreads();
        pass(-1, row, order);
    }
    for (; row >= lowest; --row, ++order) {
        const RowBasis& basis = sm.basis[row & 1];
        const int kind = basis.kind;
        if (kind == kRuleFitFailed) {  // identical in every CTA
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicMin(&a.status->fit_failed_order, order);
            return;
        }
        double* swap = spots;
        spots = spots_next;
        spots_next = swap;
        const bool fits = kind == kRuleRegression;
        if (fits) reduce_warps();
        else clear_sums();
        __syncthreads();
        if (warp < kExchangeWarps) {
            if (fits) {
                const double total = dd_round(exchange_totals(sm.exchange, a.partials, int(blockIdx.x), int(gridDim.x), seq, a.status));
                if (warp == 0)
                    solve_row<D>(basis, total, __shfl_sync(0xffffffffu, total, kBadResponses) > 0.5, &sm.row);
            } else if (threadIdx.x == 0) {
                sm.row.rule = never_exercise();
                sm.row.kind = kind;
            }
        } else if (row - 1 >= lowest) {
            if (warp == kExchangeWarps) prepare(row - 1);
            if (threadIdx.x == kFetchThread) {
                fetch(row - 1);
                wait_copy();
            }
        }
        __syncthreads();
        if (sm.failed != 0 || sm.exchange.failed != 0) return;
        if (fits && blockIdx.x == 0 && warp == kExchangeWarps) write_coefficients<D>(sm.row, a.records[row]);
        if (sm.row.kind == kRuleFitFailed) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicMin(&a.status->fit_failed_order, order);
            return;
        }
        if (fits) ++seq;
        pass(row, row - 1, order + 1);
    }
    // Common origin decision (policy.rs:265-281): mean of values discounted to the origin.
    if (plan.origin_row) {
        for (int j = 0; j < owned; ++j) {
            const double w = value(j) * plan.origin_discount;
            if (!fo_isfinite(w))
                atomicMin(&a.status->fit_payoff_fail,
                          ((unsigned long long)order << 32) | (first + uint64_t(j) * T + threadIdx.x));
            sums[0] += w;
        }
        reduce_warps();
        __syncthreads();
        dd total = dd_make(0.0);
        if (warp < kExchangeWarps) total = exchange_totals(sm.exchange, a.partials, int(blockIdx.x), int(gridDim.x), seq, a.status);
        if (blockIdx.x == 0 && threadIdx.x == 0 && sm.exchange.failed == 0) {
            const double mean = dd_round(dd_div(total, dd_make(double(P))));
            const double intrinsic = plan.initial_spot - K > 0.0 ? plan.initial_spot - K : 0.0;
            FitRecord& rec = a.records[0];
            rec.kind = kRuleOrigin;
            rec.origin_exercise = exercise_rule(plan.tie_rule, intrinsic, mean) ? 1 : 0;
            rec.origin_continuation = mean;
            rec.itm = 0;
            rec.diag_status = -1;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------------

// CTAs per row of the moments launch: one wave of the device over all rows (a CTA's pivot and reduction
// cost as much as some 4,000 of its paths), no more than keeps 2,048 paths each, and no more than
// the workspace holds totals for (one CTA a row needs none).
int moment_blocks(uint64_t paths, uint32_t rows, int sms, size_t workspace_bytes) {
    const uint64_t by_work = (paths + 2047) / 2048;
    const uint64_t by_device = uint64_t(sms) * kMomentCtasPerSm / rows;
    const uint64_t by_space = workspace_bytes / moment_workspace_bytes(rows, 1);
    return int(std::max<uint64_t>(1, std::min(std::min(by_work, by_device), by_space)));
}

size_t moment_workspace_bytes(uint32_t rows, int blocks) { return sizeof(double2) * kSlots * rows * size_t(blocks); }

template <int D>
static cudaError_t launch_moments_d(const MomentArgs& args, int rows, int blocks, cudaStream_t stream) {
    // Not by launch_early: with an event recorded behind it for another stream, a call took 25 us more (52 weeks,
    // 2^20 paths: 1,250 us against 1,218).
    const dim3 grid{unsigned(blocks), unsigned(rows)};
    moments_kernel<D, false><<<grid, kMomentThreads, 0, stream>>>(args);
    if constexpr (D > 0)
        if (args.relaunch) moments_kernel<D, true><<<grid, kMomentThreads, 0, stream>>>(args);
    return cudaGetLastError();
}

cudaError_t launch_moments(const MomentArgs& args, int blocks, cudaStream_t stream) {
    const uint32_t lowest = args.plan.origin_row ? 1u : 0u, E = args.plan.rows - 1;
    if (E <= lowest) return cudaSuccess;
    const int rows = int(E - lowest);
    switch (args.plan.degree) {  // validated to 0..4 on the host
        case 0: return launch_moments_d<0>(args, rows, blocks, stream);
        case 1: return launch_moments_d<1>(args, rows, blocks, stream);
        case 2: return launch_moments_d<2>(args, rows, blocks, stream);
        case 3: return launch_moments_d<3>(args, rows, blocks, stream);
        default: return launch_moments_d<4>(args, rows, blocks, stream);
    }
}

size_t backward_smem_bytes(int ppt) { return sizeof(double) * (3 * size_t(ppt) * kBackwardThreads + 4); }

int backward_max_ppt() {
    // Dynamic shared memory available next to the kernel's static shared memory.
    cudaFuncAttributes attr{};
    cudaFuncGetAttributes(&attr, backward_kernel<kMaxDegree, false>);  // every degree has the same static shared memory
    int optin = 0, device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    const size_t fixed = attr.sharedSizeBytes + backward_smem_bytes(0);
    const size_t avail = size_t(optin) > fixed ? size_t(optin) - fixed : 0;
    return int(avail / (sizeof(double) * 3 * kBackwardThreads));
}

int backward_max_blocks(int device) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;  // one CTA per SM
}

template <int D, bool kHbm>
static cudaError_t launch_backward_d(const BackwardArgs& args, int blocks, int ppt, cudaStream_t stream) {
    const size_t smem = kHbm ? 0 : backward_smem_bytes(ppt);
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(backward_kernel<D, kHbm>), smem,
                                             sizeof(BackwardSmem) + 256);
    if (e != cudaSuccess) return e;
    // The launch itself refuses a grid that cannot be resident (cudaErrorCooperativeLaunchTooLarge).
    void* params[] = {const_cast<BackwardArgs*>(&args)};
    return cudaLaunchCooperativeKernel((const void*)backward_kernel<D, kHbm>, dim3(blocks), dim3(kBackwardThreads),
                                       params, smem, stream);
}

template <bool kHbm>
static cudaError_t launch_backward_storage(const BackwardArgs& args, int blocks, int ppt, cudaStream_t stream) {
    switch (args.plan.degree) {  // validated to 0..4 on the host
        case 0: return launch_backward_d<0, kHbm>(args, blocks, ppt, stream);
        case 1: return launch_backward_d<1, kHbm>(args, blocks, ppt, stream);
        case 2: return launch_backward_d<2, kHbm>(args, blocks, ppt, stream);
        case 3: return launch_backward_d<3, kHbm>(args, blocks, ppt, stream);
        default: return launch_backward_d<4, kHbm>(args, blocks, ppt, stream);
    }
}

cudaError_t launch_backward(const BackwardArgs& args, int blocks, int ppt, cudaStream_t stream) {
    return args.values ? launch_backward_storage<true>(args, blocks, ppt, stream)
                       : launch_backward_storage<false>(args, blocks, ppt, stream);
}

}  // namespace fo
