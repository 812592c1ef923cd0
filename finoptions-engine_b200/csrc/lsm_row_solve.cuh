// lsm_row_solve.cuh - a fitted row's regression once its response sums are known. The moments kernel has
// solved everything that does not depend on the responses (mean, scale, recurrence, norms); what is
// left is the projections on the basis, the coefficients and the exercise rule, by one warp.
//
// The responses are summed against powers of z, R_k = sum y z^k, and projected on the basis first: the
// coefficients of a nearly dependent design keep the accuracy that the orthogonal basis gives them.
// (A matrix from the R_k straight to the powers' coefficients is the inverse of their Gram matrix: rows of
// five to twelve paths lose twice as much, and decide paths differently near a condition of 1e7.) The
// rule is formed from the coefficients by make_exercise_rule's operations in its order, so the pass over
// the paths decides by the very rule that the evaluation forms from the record.
#pragma once

#include <stdint.h>

#include "fo_core.cuh"
#include "lsm_device.cuh"

namespace fo {

#ifdef __CUDACC__

// What a row's pass needs of its moments: z = excess * slope + shift, the basis in powers of z and its
// norms.
struct RowBasis {
    double slope, shift;
    double discount;                         // into this row from the one after it
    double power[kMaxColumns][kMaxColumns];  // p_j = sum_i power[j][i] z^i
    double norm[kMaxColumns], inv_norm[kMaxColumns];
    double reach[kMaxColumns];               // |z|^i at kRuleSpotLimit
    double mean, scale, inv_scale;           // rows outside the rule's range go through the model
    double alpha[kMaxDegree], beta[kMaxDegree];
    int kind;
    int general;
};

struct RowSolution {
    ExerciseRule rule;
    double coef[kMaxColumns];  // in the orthogonal basis
    int kind;
    int bad_responses;         // a response was not finite
    int broken;                // the first basis function without a finite coefficient, or 0
};

// One warp prepares a row's basis from its record, lane i the coefficient of z^i.
template <int D>
__device__ __forceinline__ void prepare_basis(const FitRecord& rec, double strike, double discount, RowBasis* out) {
    const int lane = threadIdx.x & 31;
    const FitModel& m = rec.model;
    const int kind = rec.kind;
    const double mean = m.mean, scale = m.scale;
    const bool fitted = kind == kRuleRegression;
    const double norm = lane < kMaxColumns ? m.norm[lane] : 0.0;
    const double inv_norm = make_divisor(norm).inv;
    double current = lane == 0 ? 1.0 : 0.0, previous = 0.0;
#pragma unroll
    for (int j = 0; j <= D; ++j) {
        if (lane < kMaxColumns) out->power[j][lane] = current;
        if (j < D) {
            const double below = __shfl_up_sync(0xffffffffu, current, 1);
            const double next =
                fo_fma(-m.beta[j], previous, fo_fma(-m.alpha[j], current, lane > 0 ? below : 0.0));
            previous = current;
            current = next;
        }
    }
    const double slope = D > 0 && fitted ? 1.0 / (strike * scale) : 0.0;
    const double shift = D > 0 && fitted ? (1.0 - mean) / scale : 0.0;
    const double z = fo_fma(kRuleSpotLimit, slope, fo_fabs(shift));
    double reach = 1.0;
#pragma unroll
    for (int i = 1; i < kMaxColumns; ++i) reach = i <= lane ? reach * z : reach;
    if (lane < kMaxColumns) {
        out->norm[lane] = norm;
        out->inv_norm[lane] = inv_norm;
        out->reach[lane] = reach;
    }
    if (lane < kMaxDegree) {
        out->alpha[lane] = m.alpha[lane];
        out->beta[lane] = m.beta[lane];
    }
    if (lane == 0) {
        out->slope = slope;
        out->shift = shift;
        out->discount = discount;
        out->mean = mean;
        out->scale = scale;
        out->inv_scale = m.inv_scale;
        out->kind = kind;
        out->general = fitted && (rec.beyond_rule != 0 || !(strike > 0x1p-100 && strike < 0x1p100) ||
                                  !(scale > 0x1p-100 && scale < 0x1p100));
    }
}

// A row's coefficients and rule from its response sums (lane k's `response` is R_k), by one warp: lane j the
// j-th projection and coefficient, then lane i the coefficient of z^i.
template <int D>
__device__ __forceinline__ void solve_row(const RowBasis& basis, double response, bool bad_responses, RowSolution* out) {
    const int lane = threadIdx.x & 31;
    const int j = lane <= D ? lane : 0;
    double projection = 0.0;
#pragma unroll
    for (int i = 0; i <= D; ++i) {
        const double r = __shfl_sync(0xffffffffu, response, i);
        projection = i <= j ? fo_fma(basis.power[j][i], r, projection) : projection;
    }
    const double coef = divide(projection, Divisor{basis.norm[j], basis.inv_norm[j]});
    const unsigned broken = __ballot_sync(0xffffffffu, !(fo_isfinite(projection) && fo_isfinite(coef)));
    double c = lane == 0 ? coef : 0.0;
#pragma unroll
    for (int k = 1; k <= D; ++k) c = fo_fma(__shfl_sync(0xffffffffu, coef, k), basis.power[k][j], c);
    const bool covered = __all_sync(0xffffffffu, lane > D || fo_fabs(c) * basis.reach[j] < 0x1p1000);
    if (lane < kMaxColumns) {
        out->rule.c[lane] = lane <= D ? c : 0.0;
        out->coef[lane] = coef;
    }
    if (lane == 0) {
        out->rule.slope = basis.slope;
        out->rule.shift = basis.shift;
        out->rule.general = basis.general != 0 || !covered;
        out->kind = bad_responses || broken != 0 ? kRuleFitFailed : kRuleRegression;
        out->bad_responses = bad_responses ? 1 : 0;
        out->broken = broken != 0 ? __ffs(int(broken)) - 1 : 0;
    }
}

#endif  // __CUDACC__

}  // namespace fo
