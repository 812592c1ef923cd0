// lsm_evaluate.cuh - the fixed policy of a single contract as its evaluation kernels apply it
// (evaluate_kernel, evaluate_greeks_kernel): one staged row per observation and the decision at it.
#pragma once

#include <stdint.h>

#include "lsm_common.cuh"
#include "lsm_kernels.h"

namespace fo {

struct EvalRow {
    ExerciseRule rule;
    double discount;
    double pad;
};

__device__ __forceinline__ EvalRow make_eval_row(const DevicePlan& plan, const FitRecord* records, uint32_t row) {
    EvalRow er{never_exercise(), plan.disc_to_origin[row], 0.0};
    if (row + 1 < plan.rows) {
        const int32_t kind = records[row].kind;
        if (kind == kRuleRegression) er.rule = make_exercise_rule(records[row].model, plan.degree, plan.strike);
        else if (kind == kRuleNoSupport) er.rule.general = 1;
    }
    return er;
}

// Whether path p, in the money by `excess` at `row`, exercises there. Rows without training support
// count it; a continuation that is not finite fails the evaluation.
template <int D>
__device__ __forceinline__ bool decide_row(const DevicePlan& plan, const FitRecord* records, DeviceStatus* status,
                                           const ExerciseRule& rule, uint32_t row, uint64_t p, double spot,
                                           double excess, unsigned* itm_counts) {
    if (rule.general == 0 && within_rule(spot))
        return exercise_rule(plan.tie_rule, excess, rule_continuation<D>(rule, excess));
    const int32_t kind = records[row].kind;
    if (kind == kRuleNoSupport) atomicAdd(&itm_counts[row], 1u);
    if (kind != kRuleRegression) return false;
    const int decision = decide_general<D>(&records[row].model, spot, plan.strike, plan.tie_rule);
    if (decision == kDecideNonFinite) atomicMin(&status->eval_fail, ((unsigned long long)row << 33) | (p << 1));
    return decision == kDecideExercise;
}

// Whether the calling CTA is the last of its launch to get here, its writes and all others' visible. The
// counter (status->arrivals) is left at zero for the next launch.
__device__ __forceinline__ bool last_cta(DeviceStatus* status) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(&status->arrivals, 1u) + 1u == gridDim.x;
        if (last) status->arrivals = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// Price, second moment, standard deviation and standard error from the CTA partials, by one CTA.
__device__ __forceinline__ void finalize_price(const double2* partials, int blocks, uint64_t paths, double* out) {
    __shared__ dd total[2];
    grid_combine<2>(partials, blocks, total);
    if (threadIdx.x != 0) return;
    const dd n = dd_make(double(paths));
    const dd mean = dd_div(total[0], n);
    // M2 = sum x^2 - (sum x)^2 / n
    dd m2 = dd_sub(total[1], dd_mul(total[0], mean));
    if (m2.hi < 0.0) m2 = dd_make(0.0);
    out[0] = dd_round(mean);
    out[1] = dd_round(m2);
    if (paths > 1) {
        const dd var = dd_div(m2, dd_make(double(paths - 1)));
        const double sd = dd_round(dd_sqrt(var));
        out[2] = sd;
        out[3] = sd / sqrt(double(paths));
    } else {
        out[2] = 0.0;
        out[3] = 0.0;
    }
}

}  // namespace fo
