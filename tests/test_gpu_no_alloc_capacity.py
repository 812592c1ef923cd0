"""The allocation-free entry's capacity: what its scratch held when the backward pass ran 1,024 threads a CTA
(half as many CTAs for a population of one path a thread) it still holds."""

from __future__ import annotations

import ctypes

import pytest
from finoptions import _abi
from finoptions._requests import lsm_call_request, lsm_call_result

import _oracle

pytestmark = pytest.mark.gpu


# The largest populations accepted beside these date counts: 63 CTAs of 1,024 threads, 41 of them.
@pytest.mark.parametrize("dates, evaluation_paths, paths", [(130, 256, 64450), (130, 300000, 63837), (200, 1000, 41884)])
def test_the_largest_population_still_fits(dates, evaluation_paths, paths) -> None:
    t = [i / dates for i in range(dates + 1)]
    request = lsm_call_request(
        initial_spot=100.0, strike=100.0, schedule_times=t, curve_times=t,
        log_discounts=[0.0] + [-0.04 * v for v in t[1:]], dividend_yield_times=t,
        cumulative_dividend_yields=[0.0] + [0.02 * v for v in t[1:]], dividend_nodes=[], dividend_amounts=[],
        exercise_nodes=list(range(1, dates)), expiry_node=dates, annualized_volatility=0.25, dividend_policy=0,
        training_paths=paths, evaluation_paths=evaluation_paths, training_seed=11, training_domain=1,
        evaluation_seed=11, evaluation_domain=2, polynomial_degree=2, rank_tolerance=1e-12, condition_limit=1e8,
        tie_rule=0, insufficient_exercise_support=1)
    result, err = lsm_call_result(request.exercise_rows), _abi.FoError()
    assert _abi.load().fo_price_lsm_call_f64_noalloc(ctypes.byref(request.struct), None, ctypes.byref(result.struct),
                                                     ctypes.byref(err)) == 0, err.message
    got, want = result.as_tuple(), _oracle.price_lsm_call(request)
    assert got[0] == pytest.approx(want[0], rel=1e-9)
    assert got[2] == pytest.approx(want[2], rel=1e-9)
