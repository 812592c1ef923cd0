"""The exercise rule (one fma to standardise, the continuation in powers of z), compiled for the host,
against the fitted polynomial in extended precision and against the reference predictor.

The bound counts roundings. A coefficient of a power comes from at most four basis steps of two fused
operations and a sum, so with A_k the coefficients of the same recurrence in absolute values it is
within 16 u A_k; Horner adds 8 u, and z is within 4 u (|z| + |shift|) of its value, worth at most its
derivative. u = 2^-53.
"""

from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import _oracle

HERE = Path(__file__).resolve().parent
BUILD = HERE / "native" / "_build"
U = 2.0**-53


@pytest.fixture(scope="module")
def harness() -> ctypes.CDLL:
    BUILD.mkdir(parents=True, exist_ok=True)
    lib = BUILD / "librule_harness.so"
    src = HERE / "native" / "rule_harness.cpp"
    core = HERE.parent / "finoptions-engine_b200" / "csrc" / "fo_core.cuh"
    if not lib.is_file() or lib.stat().st_mtime < max(src.stat().st_mtime, core.stat().st_mtime):
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", str(src), "-o", str(lib)],
                       check=True)
    h = ctypes.CDLL(str(lib))
    h.harness_rule.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_void_p, ctypes.c_uint64,
                               ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    h.harness_never.argtypes = [ctypes.c_double, ctypes.c_double]
    h.harness_never.restype = ctypes.c_double
    h.harness_divide_above.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_double]
    h.harness_divide_above.restype = ctypes.c_uint64
    return h


def fitted(rng: np.random.Generator, degree: int, n: int, strike: float, sigma: float, moneyness: float):
    """A fitted model in the order mean, scale, alpha, beta, coef, and its in-the-money spots."""
    spots = strike / moneyness * np.exp(sigma * rng.standard_normal(16 * n + 400))
    spots = spots[spots > strike][:n]
    y = np.maximum(spots * np.exp(0.3 * sigma * rng.standard_normal(spots.size)) - strike, 0.0) * 0.99
    code, model, _ = _oracle.fit_regression(spots / strike, y, degree)
    return code, model, spots


def evaluate(h, model: np.ndarray, degree: int, strike: float, spots: np.ndarray):
    by_rule, by_predictor = np.empty(spots.size), np.empty(spots.size)
    finite = np.empty(spots.size, dtype=np.int32)
    general = h.harness_rule(model.ctypes.data, degree, strike, spots.ctypes.data, spots.size, by_rule.ctypes.data,
                             by_predictor.ctypes.data, finite.ctypes.data)
    return general, by_rule, by_predictor, finite


def bound_and_value(model: np.ndarray, degree: int, strike: float, spots: np.ndarray):
    """The rounding bound above and the continuation in extended precision."""
    wide = np.longdouble
    mean, scale = wide(model[0]), wide(model[1])
    alpha, beta, coef = model[2:6].astype(wide), model[6:10].astype(wide), model[10:15].astype(wide)
    z = (spots.astype(wide) / wide(strike) - mean) / scale if degree else np.zeros(spots.size, dtype=wide)
    previous, current = np.zeros_like(z), np.ones_like(z)
    value = coef[0] * current
    a_previous, a_current, a_total = np.zeros(6, dtype=wide), np.zeros(6, dtype=wide), np.zeros(6, dtype=wide)
    a_current[0] = 1
    a_total[0] = abs(coef[0])
    for j in range(degree):
        previous, current = current, (z - alpha[j]) * current - beta[j] * previous
        value = value + coef[j + 1] * current
        up = np.roll(a_current, 1)
        up[0] = 0
        a_previous, a_current = a_current, up + abs(alpha[j]) * a_current + abs(beta[j]) * a_previous
        a_total = a_total + abs(coef[j + 1]) * a_current
    power = np.abs(z)[:, None] ** np.arange(6)
    shift = abs((1 - mean) / scale) if degree else wide(0)
    slack = power @ a_total * 24 * U
    if degree:
        slack = slack + (power[:, :5] * (np.arange(1, 6) * a_total[1:])).sum(axis=1) * 4 * U * (np.abs(z) + shift)
    return slack, value


@pytest.mark.parametrize("degree", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("strike", [100.0, 0.37, 2.0**-99, 2.0**99])
def test_rule_is_the_fitted_polynomial(harness, degree, strike) -> None:
    rng = np.random.default_rng(5 + degree)
    for trial in range(12):
        n = 6 + 9 * trial if trial % 3 == 0 else 4000
        code, model, spots = fitted(rng, degree, n, strike, 0.03 + 0.06 * (trial % 6), (0.8, 1.0, 1.2)[trial % 3])
        if code != 0:
            continue
        general, by_rule, by_predictor, finite = evaluate(harness, model, degree, strike, spots)
        # Covered unless a power of z could overflow below the spot limit 2^200 (degree 4 at 2^-99).
        assert general == int(degree * (200 - np.log2(strike * model[1])) >= 1000)
        assert finite.all()
        slack, value = bound_and_value(model, degree, strike, spots)
        assert (np.abs(by_rule - value) <= slack).all()
        # The same decisions as the predictor's wherever the two sides differ by more than both roundings.
        clear = np.abs((spots - strike) - value) > 4 * slack + 64 * U * np.abs(value)
        assert ((spots - strike > by_rule) == (spots - strike > by_predictor))[clear].all()


@pytest.mark.parametrize("change", ["tiny_strike", "huge_strike", "tiny_scale", "huge_scale", "infinite_coefficient",
                                    "nan_coefficient", "overflowing_powers"])
def test_rows_whose_arithmetic_could_overflow_are_general(harness, change) -> None:
    model = np.array([1.1, 0.2, 0.3, 0.2, 0.1, 0.1, 0.0, 1.0, 1.5, 2.0, 8.0, 4.0, 0.5, 0.1, 0.02])
    strike = {"tiny_strike": 2.0**-101, "huge_strike": 2.0**101}.get(change, 100.0)
    if change.endswith("scale"):
        model[1] = 2.0**-101 if change == "tiny_scale" else 2.0**101
    if change == "infinite_coefficient":
        model[12] = np.inf
    if change == "nan_coefficient":
        model[14] = np.nan
    if change == "overflowing_powers":
        model[1] = 2.0**-80  # (2^200 / (100 scale))^4 is past 2^1024
    assert evaluate(harness, model, 4, strike, np.array([strike * 1.5]))[0] == 1


def test_rows_that_never_exercise_continue_at_every_covered_spot(harness) -> None:
    for spot in (101.0, 1e10, 2.0**200):
        assert harness.harness_never(spot, 100.0) == np.inf


@pytest.mark.parametrize("strike", [100.0, 0.37, 1.0, 3.0**-40, 2.0**-900, 2.0**900])
def test_in_the_money_quotient_is_correctly_rounded(harness, strike) -> None:
    rng = np.random.default_rng(3)
    spots = strike * np.concatenate([1.0 + rng.random(200000), np.exp(30.0 * rng.random(50000)),
                                     1.0 + U * 2 * np.arange(1, 200)])
    spots = spots[(spots > strike) & np.isfinite(spots)]
    assert harness.harness_divide_above(spots.ctypes.data, spots.size, strike) == 0
