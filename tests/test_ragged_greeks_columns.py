"""The node capacity that a ragged Greeks call asks for: enough for every row's mesh, and columns too short
for their rows still raise before the engine reads them."""

from __future__ import annotations

import dataclasses

import finoptions as fo
import pytest
from _workloads import ragged_columns
from finoptions.batch_lsm import _mesh_nodes_bound


def contracts(cash: bool):
    c = ragged_columns(7, seed=3, min_paths=2, max_paths=9, min_exercise=1, max_exercise=5)
    return fo.LsmRaggedContracts(
        initial_spots=c.initial_spots, strikes=c.strikes, maturities=c.maturities, rates=c.rates,
        volatilities=c.volatilities, exercise=fo.RaggedExerciseTimes(offsets=c.exercise_offsets, times=c.exercise_times),
        training_paths=c.paths, evaluation_paths=c.paths,
        cash_dividends=fo.RaggedCashDividends(offsets=c.dividend_offsets, times=c.dividend_times,
                                              amounts=c.dividend_amounts) if cash else None)


@pytest.mark.parametrize("cash", [False, True])
def test_the_bound_covers_every_mesh(cash) -> None:
    assert _mesh_nodes_bound(contracts(cash)) >= contracts(cash).mesh_nodes()


def test_short_columns_raise() -> None:
    whole = contracts(True)
    short_times = fo.RaggedExerciseTimes(offsets=whole.exercise.offsets[:3], times=whole.exercise.times[:int(whole.exercise.offsets[2])])
    for change in ({"maturities": whole.maturities[:3]}, {"exercise": short_times}):
        with pytest.raises(IndexError):
            _mesh_nodes_bound(dataclasses.replace(whole, **change))
