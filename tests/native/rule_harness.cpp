// Host build of the exercise rule (finoptions-engine_b200/csrc/fo_core.cuh) for the CPU test suite:
// the rule of a fitted row and the reference predictor, on the same spots.
#include <cstdint>

#include "../../finoptions-engine_b200/csrc/fo_core.cuh"

using namespace fo;

// model: mean, scale, alpha[4], beta[4], coef[5]. Writes per spot the rule's continuation and the
// predictor's (and whether it is finite); returns the rule's `general` flag.
extern "C" int harness_rule(const double* model, int degree, double strike, const double* spots, uint64_t n,
                            double* by_rule, double* by_predictor, int32_t* finite) {
    FitModel m{};
    m.mean = model[0];
    m.scale = model[1];
    m.inv_scale = make_divisor(m.scale).inv;
    for (int j = 0; j < kMaxDegree; ++j) {
        m.alpha[j] = model[2 + j];
        m.beta[j] = model[6 + j];
    }
    for (int j = 0; j < kMaxColumns; ++j) m.coef[j] = model[10 + j];
    const ExerciseRule rule = make_exercise_rule(m, degree, strike);
    for (uint64_t i = 0; i < n; ++i) {
        const double d = spots[i] - strike;
        switch (degree) {
            case 0: by_rule[i] = rule_continuation<0>(rule, d); break;
            case 1: by_rule[i] = rule_continuation<1>(rule, d); break;
            case 2: by_rule[i] = rule_continuation<2>(rule, d); break;
            case 3: by_rule[i] = rule_continuation<3>(rule, d); break;
            default: by_rule[i] = rule_continuation<4>(rule, d); break;
        }
        by_predictor[i] = 0.0;
        finite[i] = predict_continuation(m, degree, divide(spots[i], make_divisor(strike)), &by_predictor[i]) ? 1 : 0;
    }
    return rule.general;
}

extern "C" double harness_never(double spot, double strike) {
    return rule_continuation<4>(never_exercise(), spot - strike);
}

// The in-the-money quotient without range checks against IEEE division: mismatches among n spots.
extern "C" uint64_t harness_divide_above(const double* spots, uint64_t n, double strike) {
    const Divisor d = make_divisor(strike);
    uint64_t wrong = 0;
    for (uint64_t i = 0; i < n; ++i) {
        const double q = divide_above(spots[i], d), want = spots[i] / strike;
        wrong += fo_isfinite(q) && double_to_bits(q) != double_to_bits(want);
    }
    return wrong;
}
