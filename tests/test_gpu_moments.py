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
