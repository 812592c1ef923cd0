"""The moments of a contract's rows where their launch turns: a training population much larger than the
evaluation's, whose partials the workspace is shared with. Against the oracle, with the parity bars of the
engine's contract."""

from __future__ import annotations

import pytest
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
