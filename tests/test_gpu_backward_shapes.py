"""The backward pass at the population sizes where its split turns: one CTA and the exchange between
several, a full and a partial last CTA, odd populations (whose rows start between two 16-byte
boundaries), one and several moment CTAs a row, and rows whose in-the-money paths lie far from the
sample that sets their pivot. Against the oracle, with the parity bars of the engine's contract."""

from __future__ import annotations

import ctypes

import pytest
from finoptions import _abi
from finoptions._requests import lsm_call_request, lsm_call_result

import _oracle

pytestmark = pytest.mark.gpu


def contract(paths: int, *, dates: int = 6, degree: int = 4, strike: float = 100.0, origin: bool = True, tie: int = 0,
             evaluation_paths: int = 4099, volatility: float = 0.3) -> dict:
    t = [i / dates for i in range(dates + 1)]
    return dict(
        initial_spot=100.0, strike=strike, schedule_times=t, curve_times=t,
        log_discounts=[0.0 if i == 0 else -0.03 * v for i, v in enumerate(t)], dividend_yield_times=t,
        cumulative_dividend_yields=[0.0 if i == 0 else 0.02 * v for i, v in enumerate(t)], dividend_nodes=[2],
        dividend_amounts=[1.5], exercise_nodes=list(range(0 if origin else 1, dates)), expiry_node=dates,
        annualized_volatility=volatility, dividend_policy=0, training_paths=paths, evaluation_paths=evaluation_paths,
        training_seed=19, training_domain=1, evaluation_seed=19, evaluation_domain=2, polynomial_degree=degree,
        rank_tolerance=1e-12, condition_limit=1e12, tie_rule=tie, insufficient_exercise_support=1)


def check(native_executor, kwargs: dict, condition_rtol: float = 1e-8) -> None:
    req = lsm_call_request(**kwargs)
    res, err = lsm_call_result(req.exercise_rows), _abi.FoError()
    assert _abi.load().fo_price_lsm_call_f64(native_executor.raw, ctypes.byref(req.struct), ctypes.byref(res.struct),
                                             ctypes.byref(err)) == 0, err.message
    got, want = res.as_tuple(), _oracle.price_lsm_call(req)
    assert got[0] == pytest.approx(want[0], rel=1e-9)
    assert got[2] == pytest.approx(want[2], rel=1e-9)
    assert got[3] == pytest.approx(want[3], rel=1e-9)
    assert got[4:6] == want[4:6]
    for g, w in zip(got[6], want[6], strict=True):
        assert g[:8] == (w[:2] + (w[2], pytest.approx(w[3], rel=1e-9) if w[3] is not None else None) + w[4:8])
        if g[8] is not None:
            assert g[8] == pytest.approx(w[8], rel=condition_rtol)
            assert g[9] == pytest.approx(w[9], rel=1e-12)
            assert g[10] == pytest.approx(w[10], rel=1e-12)


@pytest.mark.parametrize("paths", [7, 511, 512, 513, 1023, 4097, 75776, 75777, 131071, 151553, 600001])
def test_population_sizes_match_the_oracle(native_executor, paths) -> None:
    check(native_executor, contract(paths))


@pytest.mark.parametrize("degree", [0, 1, 2, 3])
def test_degrees_and_tie_rules_match_the_oracle(native_executor, degree) -> None:
    check(native_executor, contract(20011, degree=degree, tie=degree % 2, origin=degree != 2))


@pytest.mark.parametrize("strike", [130.0, 160.0, 190.0])
def test_rows_with_few_paths_in_the_money_match_the_oracle(native_executor, strike) -> None:
    # Down to a handful of in-the-money paths, none of them in the pivot's sample: the moments are taken
    # again about the row's own mean. Their conditions carry the rounding of a near-singular design.
    check(native_executor, contract(150001, strike=strike, degree=2), condition_rtol=1e-6)


def test_no_fitted_row_prices_the_origin_decision_alone(native_executor) -> None:
    for paths in (400, 100003):
        kwargs = {**contract(paths), "exercise_nodes": [0]}
        check(native_executor, kwargs)
        check(native_executor, kwargs)  # the exchange buffer starts over
