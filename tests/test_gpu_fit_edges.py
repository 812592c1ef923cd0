"""Batch fits at the populations where their split turns - a round of 256 paths, groups of four rounds,
the rounds whose values stay on chip (near 13,824 paths), a team of CTAs (above 32,768) - and beyond the
spots the exercise rule covers; and contracts of one to three intervals. Against the oracle and the
single-contract Greeks, with the parity bars of the engine's contract."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
from _workloads import grouped_columns, grouped_request, ragged_columns, ragged_request, ragged_row_as_call
from finoptions import _abi
from finoptions._requests import lsm_call_greeks, lsm_call_request, lsm_call_result
from test_gpu_batch import check_against_oracle
from test_gpu_batch_tuning import autotune, set_shape
from test_gpu_ragged import gpu_ragged_greeks

import _oracle

pytestmark = pytest.mark.gpu


@pytest.fixture
def check_executors(native_executor):
    """Prices a grouped request through the persistent launch and the phase kernels: both within the
    oracle's bars and equal to each other in every bit."""

    def check(req) -> None:
        out = []
        for phases in (0, 1):
            set_shape(native_executor, (2, 1, 8, 0, phases))
            out.append(check_against_oracle(native_executor, req))
        for a, b in zip(*out, strict=True):
            np.testing.assert_array_equal(a, b)

    yield check
    autotune(native_executor)


@pytest.mark.parametrize("paths", [255, 257, 1279, 2048, 13823, 13825, 16641, 32768, 32769])
def test_fit_populations_match_the_oracle(check_executors, paths) -> None:
    c = grouped_columns(2, 3, seed=paths, min_exercise=3, max_exercise=7)
    check_executors(grouped_request(c, paths))


@pytest.mark.parametrize("degree, spot, strike, volatility", [(1, 1.6e60, 1e30, 0.02), (4, 1.5e60, 1.5e60, 0.3)])
def test_fits_beyond_the_rules_range_match_the_oracle(check_executors, degree, spot, strike, volatility) -> None:
    c = grouped_columns(2, 3, seed=5, min_exercise=4, max_exercise=6)
    c.initial_spots[:] = spot
    c.strikes[:] = np.tile(strike * np.array([0.9, 1.0, 1.1]), 2)
    c.volatilities[:] = volatility
    check_executors(grouped_request(c, 1500, degree=degree))


@pytest.mark.parametrize("degree", [0, 4])
def test_contracts_of_one_to_three_intervals(native_executor, degree) -> None:
    c = ragged_columns(9, seed=59, min_paths=200, max_paths=70000, min_exercise=1, max_exercise=3)
    out, delta, vega, d_l, offsets, _ = gpu_ragged_greeks(native_executor, ragged_request(c, degree=degree), c)
    for r in range(c.rows):
        kw = ragged_row_as_call(c, r, degree=degree)
        req = lsm_call_request(**kw)
        res, err = lsm_call_result(req.exercise_rows), _abi.FoError()
        g, g_l, _d = lsm_call_greeks(len(kw["schedule_times"]), len(kw["dividend_nodes"]))
        assert _abi.load().fo_price_lsm_call_greeks_f64(native_executor.raw, ctypes.byref(req.struct),
                                                        ctypes.byref(res.struct), ctypes.byref(g),
                                                        ctypes.byref(err)) == 0, err.message
        got, want = res.as_tuple(), _oracle.price_lsm_call(req)
        assert got[0] == pytest.approx(want[0], rel=1e-9), r
        assert got[2] == pytest.approx(want[2], rel=1e-9), r
        assert got[4:6] == want[4:6], r
        assert out[0][r] == pytest.approx(got[0], rel=1e-12, abs=1e-13), r
        assert delta[r] == pytest.approx(g.delta, rel=1e-10, abs=1e-12), r
        assert vega[r] == pytest.approx(g.vega, rel=1e-10, abs=1e-10), r
        np.testing.assert_allclose(d_l[offsets[r]:offsets[r + 1]], g_l, rtol=1e-9, atol=1e-10, err_msg=str(r))
