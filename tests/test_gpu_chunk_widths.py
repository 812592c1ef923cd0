"""A strike's result does not depend on which strikes an evaluation item prices beside it: strips with
strikes that their rule does not decide (beyond its range, or without training support) and meshes of more
rows than shared memory holds rules for, at every width, through both executors, in every bit.

Driftless states of a volatility of 1e-12: a continuation differs from the exercise value by the states'
spread alone, which is a few thousand roundings of the state, so that two ways to round one continuation
would decide some path differently.
"""

from __future__ import annotations

import finoptions as fo
import numpy as np
import pytest
from test_gpu_batch_tuning import autotune, set_shape

pytestmark = pytest.mark.gpu

COLUMNS = ("prices", "sample_standard_deviations", "standard_errors", "early_exercise_paths", "expiry_paths",
           "regression_nodes", "no_training_support_nodes", "insufficient_exercise_support_nodes")
CONTINUE, FAIL = fo.InsufficientExerciseSupportPolicy.CONTINUE, fo.InsufficientExerciseSupportPolicy.FAIL


def strip(executor, *, groups: int, unit: float, times: np.ndarray, paths: int, support) -> dict:
    """States near `unit` with eight strikes each around their spot, exercised at `times` (of maturity 1)."""
    rng = np.random.default_rng(groups)
    spots = unit * rng.uniform(0.95, 1.05, groups)
    return {
        "groups": fo.LsmStrikeGroups(
            group_offsets=(np.arange(groups + 1) * 8).astype(np.uint32), initial_spots=spots,
            strikes=(spots[:, None] * np.linspace(0.8, 1.2, 8)).reshape(-1), maturities=np.ones(groups),
            rates=np.zeros(groups), volatilities=np.full(groups, 1e-12),
            dividends=fo.ContinuousDividendYieldBatch(np.zeros(groups))),
        "mesh": fo.ExplicitExerciseMesh(
            schedules=fo.RaggedExerciseTimes((np.arange(groups + 1) * times.size).astype(np.int64),
                                             np.tile(times, groups)),
            origin_exercise=fo.OriginExercise.EXCLUDED),
        "executor": executor,
        "method": fo.Lsm(training_paths=paths, evaluation_paths=paths,
                         training_stream=fo.RandomStream(seed=5, domain=0),
                         evaluation_stream=fo.RandomStream(seed=5, domain=1 << 20),
                         insufficient_exercise_support=support, polynomial_degree=4, rank_tolerance=1e-15,
                         condition_limit=9e14)}


CASES = {
    # Strikes on both sides of 2^100, beyond which a rule's powers are not trusted.
    "beyond the range": dict(groups=16, unit=2.0**100, times=np.arange(1, 24) / 24, paths=16384, support=CONTINUE),
    # More rows than eight strikes' rules fit beside the sampler's tables.
    "many rows": dict(groups=4, unit=100.0, times=np.arange(1, 400) / 400, paths=4096, support=CONTINUE),
    # The upper strikes have no in-the-money path, under the failing policy.
    "unsupported": dict(groups=16, unit=100.0, times=np.arange(1, 24) / 24, paths=16384, support=FAIL),
}


@pytest.mark.parametrize("name", CASES)
def test_results_do_not_depend_on_the_strikes_priced_together(executor, native_executor, name) -> None:
    request = strip(executor, **CASES[name])
    results = {}
    try:
        for phases in (0, 1):
            for width in (1, 2, 8):
                set_shape(native_executor, (2, 1, width, 0, phases))
                batch = fo.price_lsm_call_grouped_batch(**request)
                results[phases, width] = {c: np.array(getattr(batch, c)) for c in COLUMNS}
    finally:
        autotune(native_executor)
    first = results[0, 1]
    assert first["regression_nodes"].sum() > 0
    assert (first["no_training_support_nodes"].sum() > 0) == (name == "unsupported")
    for key, result in results.items():
        for column in COLUMNS:
            np.testing.assert_array_equal(result[column], first[column], err_msg=f"{key} {column}")
