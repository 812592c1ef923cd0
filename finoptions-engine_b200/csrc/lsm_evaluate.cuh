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

}  // namespace fo
