"""The chunked path stream and the decisions it feeds, at the sizes where they turn: normals per path
around the chunk of four and the reserve's threshold, path counts around a block, and markets so
large or small that rows are decided by their records instead of by their rules."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
from finoptions import _abi
from finoptions._requests import lsm_call_request, lsm_call_result

import _oracle
from _workloads import weekly_call_kwargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 103])
def test_normals_of_every_chunk_shape_match_the_oracle(native_executor, count) -> None:
    """Bit for bit up to the tail at r; a tail normal r - log(u) / r follows the last bit of the
    platform's log (half an ulp of x < r each side, and its division), so within 4 u."""
    for paths in (1, 255, 257, 40000):
        out = np.empty(paths * count)
        err = _abi.FoError()
        assert _abi.load().fo_sample_standard_normals_f64(
            native_executor.raw, 0xFEDCBA9876543, 5, 17, paths, count,
            out.ctypes.data_as(_abi.c_double_p), out.size, ctypes.byref(err)) == 0, err.message
        want = _oracle.normals(0xFEDCBA9876543, 5, 17, paths, count).ravel()
        inner = np.abs(want) <= 3.6541528853610088
        assert (out.view(np.uint64) == want.view(np.uint64))[inner].all()
        assert (np.abs(out - want) <= 4 * 2.0**-53 * np.abs(want)).all()


@pytest.mark.parametrize("scale", [2.0**-140, 2.0**140, 1.0])
@pytest.mark.parametrize("degree", [1, 4])
def test_markets_beyond_the_rules_range_price_like_the_oracle(native_executor, scale, degree) -> None:
    kwargs = {**weekly_call_kwargs(4099), "initial_spot": 100.0 * scale, "strike": 98.0 * scale,
              "polynomial_degree": degree}
    req = lsm_call_request(**kwargs)
    got, err = lsm_call_result(req.exercise_rows), _abi.FoError()
    assert _abi.load().fo_price_lsm_call_f64(native_executor.raw, ctypes.byref(req.struct), ctypes.byref(got.struct),
                                             ctypes.byref(err)) == 0, err.message
    result, want = got.as_tuple(), _oracle.price_lsm_call(req)
    assert result[0] == pytest.approx(want[0], rel=1e-9)
    assert result[4:6] == want[4:6]
