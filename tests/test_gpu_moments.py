"""The moments of a contract's rows where their launch turns: a training population much larger than the
evaluation's, whose partials the workspace is shared with. Against the oracle, with the parity bars of the
engine's contract; and the recorded means against extended precision."""

from __future__ import annotations

import ctypes

import finoptions as fo
import numpy as np
import pytest
from finoptions import _abi
from finoptions._requests import lsm_call_request
from test_gpu_backward_shapes import check, contract

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths, evaluation_paths", [(300001, 64), (300001, 1), (40000, 300001), (2049, 1)])
def test_populations_of_different_sizes_match_the_oracle(native_executor, paths, evaluation_paths) -> None:
    check(native_executor, contract(paths, evaluation_paths=evaluation_paths))


@pytest.mark.parametrize("strike", [130.0, 160.0, 190.0])
def test_rows_taken_again_on_the_whole_grid_match_the_oracle(native_executor, strike) -> None:
    # A handful of in-the-money paths in most rows, few or none in the sample that sets the pivot, on both sides
    # of the population that one CTA sums again by itself. A degree-2 design of a few paths is
    # near-singular, and its condition carries that rounding.
    for paths in (131072, 131073, 400003):
        check(native_executor, contract(paths, strike=strike, degree=2), condition_rtol=1e-6)


@pytest.mark.parametrize("strike", [97.0, 101.7, 104.3, 113.9])
def test_recorded_means_are_the_rounded_means_of_the_quotients(executor, strike) -> None:
    # A quotient's rounding averages out over the paths; what is left is the rounding of the mean itself, half a
    # unit in the last place, and a little for the 2,000 and more paths' average.
    times = tuple(i / 12 for i in range(13))
    stream = fo.RandomStream(seed=3, domain=7)
    market = {
        "initial_spot": 100.0,
        "schedule": fo.EventSchedule(times=times, dividends=(), exercise_nodes=tuple(range(1, 12)), expiry_node=12),
        "curve": fo.LogDiscountCurve(times=times, log_discounts=(0.0, *(-0.03 * t for t in times[1:]))),
        "dividend_yield_curve": fo.CumulativeDividendYieldCurve(
            times=times, cumulative_yields=(0.0, *(0.02 * t for t in times[1:]))),
        "volatility": fo.ConstantVolatility(0.3), "dividend_policy": fo.DividendPolicy.LIQUIDATOR, "executor": executor}
    paths = 40001
    states = fo.simulate_gbm_on_device(**market, paths=paths, random_stream=stream).states.cpu().numpy()
    result = fo.price_lsm_call(**market, strike=strike, method=fo.Lsm(
        training_paths=paths, evaluation_paths=64, training_stream=stream,
        evaluation_stream=fo.RandomStream(seed=3, domain=8), polynomial_degree=3,
        insufficient_exercise_support=fo.InsufficientExerciseSupportPolicy.CONTINUE))
    fits = [d for d in result.fit_diagnostics if type(d) is fo.RegressionFitDiagnostics]
    assert len(fits) == 11
    for fit, spots in zip(fits, states[:11], strict=True):
        x = spots[spots > strike].astype(np.longdouble) / np.longdouble(strike)
        assert fit.in_the_money_paths == x.size
        assert abs(fit.predictor_mean - x.mean()) <= 0.55 * np.spacing(fit.predictor_mean), fit.node


@pytest.mark.parametrize("paths, strike, degree, exercise, kernels", [
    (4096, 100.0, 4, 6, 6), (131072, 160.0, 1, 6, 6), (131073, 160.0, 1, 6, 7), (131073, 100.0, 1, 6, 6),
    (131073, 160.0, 0, 6, 6), (131073, 160.0, 4, 1, 5)])
def test_the_kernel_count_is_what_a_launch_enqueues(native_executor, paths, strike, degree, exercise, kernels) -> None:
    # Reset, simulation, moments (again for far strikes above 2^17 paths, where there is a pivot), backward,
    # diagnostic, evaluation.
    request = lsm_call_request(**{**contract(paths, strike=strike, degree=degree),
                                  "exercise_nodes": list(range(exercise))})
    plan, err, count = ctypes.c_void_p(), _abi.FoError(), ctypes.c_uint64()
    lib = _abi.load()
    assert lib.fo_lsm_call_plan_create(native_executor.raw, ctypes.byref(request.struct), ctypes.byref(plan),
                                       ctypes.byref(err)) == 0, err.message
    try:
        assert lib.fo_lsm_call_plan_kernel_count(plan, ctypes.byref(count)) == 0
        assert count.value == kernels
    finally:
        lib.fo_lsm_call_plan_destroy(plan)
