"""A fitted row's coefficients and rule as the backward pass forms them from its response sums: the rule
is, in every bit, the one that the evaluation forms from the recorded coefficients, and the coefficients
are the projections on the orthogonal basis.

The bound counts roundings, u = 2^-53: a power's coefficient is within 16 u of the same recurrence in
absolute values, a projection adds five fused operations, the division and the rounding of the sums one
each; 32 u of sum_i A_ji |R_i| / norm_j covers them.
"""

from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import _oracle

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
BUILD = HERE / "native" / "_build"
CSRC = HERE.parent / "finoptions-engine_b200" / "csrc"
U = 2.0**-53
CASE = np.dtype([("mean", "f8"), ("scale", "f8"), ("alpha", "f8", 4), ("beta", "f8", 4), ("norm", "f8", 5),
                 ("strike", "f8"), ("response", "f8", 5)])
RULE = np.dtype([("slope", "f8"), ("shift", "f8"), ("c", "f8", 5), ("general", "i4"), ("pad", "i4")])
RESULT = np.dtype([("rule", RULE), ("recorded", RULE), ("coef", "f8", 5), ("kind", "i4"), ("broken", "i4"),
                   ("bad_responses", "i4"), ("pad", "i4"), ("tail", "f8")])


@pytest.fixture(scope="module")
def harness() -> ctypes.CDLL:
    lib = BUILD / "librow_harness.so"
    src = HERE / "native" / "row_harness.cu"
    deps = [src, CSRC / "lsm_row_solve.cuh", CSRC / "lsm_device.cuh", CSRC / "fo_core.cuh"]
    if not lib.is_file() or lib.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        BUILD.mkdir(parents=True, exist_ok=True)
        subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17",
                        "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(lib)], check=True)
    dll = ctypes.CDLL(str(lib))
    dll.row_solve.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    assert (dll.row_bytes(0), dll.row_bytes(1)) == (CASE.itemsize, RESULT.itemsize)
    return dll


def solve(h: ctypes.CDLL, cases: np.ndarray, degree: int) -> np.ndarray:
    out = np.zeros(cases.size, dtype=RESULT)
    assert h.row_solve(cases.ctypes.data, cases.size, degree, out.ctypes.data) == 0
    return out


def rows(degree: int):
    """Fitted rows, near-singular designs of a few paths among them: cases, the projections in extended
    precision and the bound on them."""
    rng = np.random.default_rng(31 + degree)
    wide = np.longdouble
    cases, exact, bound = [], [], []
    for trial in range(600):
        n = int(rng.integers(degree + 2, 13)) if trial % 3 else int(rng.integers(100, 5000))
        strike = float(rng.uniform(20.0, 500.0))
        spots = strike * (1.0 + np.abs(rng.standard_normal(n)) * rng.choice((0.01, 0.2, 0.6)))
        x, y = spots / strike, np.maximum(spots - strike, 0.0) * rng.uniform(0.2, 1.4, n)
        code, model, _ = _oracle.fit_regression(x, y, degree, rank_tolerance=1e-12, condition_limit=1e14)
        if code != 0:
            continue
        z = (x - model[0]) / model[1] if degree else np.zeros(n)
        zw, yw = z.astype(wide), y.astype(wide)
        p_prev, p, a_prev, a = np.zeros(n, wide), np.ones(n, wide), np.zeros(6, wide), np.eye(6, dtype=wide)[0]
        case = np.zeros((), dtype=CASE)
        case["mean"], case["scale"], case["strike"] = model[0], model[1], strike
        case["alpha"], case["beta"] = model[2:6], model[6:10]
        case["response"] = [float((yw * zw**k).sum()) for k in range(5)]
        want, slack = np.zeros(5), np.zeros(5)
        for j in range(degree + 1):
            norm = float((p * p).sum())
            case["norm"][j] = norm
            want[j] = float((yw * p).sum() / wide(norm))
            slack[j] = float(32 * U * (a[:5] * np.abs(case["response"])).sum() / norm)
            if j < degree:
                alpha, beta = wide(model[2 + j]), wide(model[6 + j])
                p_prev, p = p, (zw - alpha) * p - beta * p_prev
                up = np.roll(a, 1)
                up[0] = 0
                a_prev, a = a, up + abs(alpha) * a + abs(beta) * a_prev
        cases.append(case)
        exact.append(want)
        bound.append(slack)
    return np.array(cases, dtype=CASE), np.array(exact), np.array(bound)


@pytest.mark.parametrize("degree", [0, 1, 2, 3, 4])
def test_the_pass_decides_by_the_recorded_rule(harness, degree) -> None:
    cases, exact, bound = rows(degree)
    assert cases.size > 400
    got = solve(harness, cases, degree)
    assert (got["kind"] == 4).all() and (got["bad_responses"] == 0).all()
    for field in ("slope", "shift", "c", "general"):
        assert got["rule"][field].tobytes() == got["recorded"][field].tobytes(), field
    assert (np.abs(got["coef"] - exact) <= bound).all()


def test_a_row_without_finite_coefficients_fails_at_the_first_of_them(harness) -> None:
    cases, _, _ = rows(4)
    cases = cases[:5].copy()
    for j in range(5):
        cases["response"][j] = 0.0
        cases["response"][j][j] = np.inf
    got = solve(harness, cases, 4)
    assert (got["kind"] == 5).all() and got["broken"].tolist() == [0, 1, 2, 3, 4]
