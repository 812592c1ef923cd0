"""Threads, each with an executor of its own, price contracts whose kernels need different amounts of shared
memory at the same time: what one launch needs does not depend on the other's."""

from __future__ import annotations

import ctypes
import subprocess
import threading
from pathlib import Path

import finoptions as fo
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
BUILD = HERE / "native" / "_build"
CSRC = HERE.parent / "finoptions-engine_b200" / "csrc"


def market(dates: int, executor: fo.CudaExecutor) -> dict:
    times = tuple(i / dates for i in range(dates + 1))
    return {
        "initial_spot": 100.0, "strike": 100.0,
        "schedule": fo.EventSchedule(times=times, dividends=(), exercise_nodes=tuple(range(1, dates)),
                                     expiry_node=dates),
        "curve": fo.LogDiscountCurve(times=times, log_discounts=(0.0, *(-0.03 * t for t in times[1:]))),
        "dividend_yield_curve": fo.CumulativeDividendYieldCurve(
            times=times, cumulative_yields=(0.0, *(0.02 * t for t in times[1:]))),
        "volatility": fo.ConstantVolatility(0.3), "dividend_policy": fo.DividendPolicy.LIQUIDATOR,
        "executor": executor,
        "method": fo.Lsm(training_paths=256, evaluation_paths=256, training_stream=fo.RandomStream(seed=3, domain=0),
                         evaluation_stream=fo.RandomStream(seed=3, domain=1), polynomial_degree=1,
                         insufficient_exercise_support=fo.InsufficientExerciseSupportPolicy.CONTINUE)}


@pytest.mark.parametrize("price", [fo.price_lsm_call, fo.price_lsm_call_greeks], ids=["price", "greeks"])
def test_contracts_of_few_and_many_dates_side_by_side(price) -> None:
    wanted, done, failures = [], threading.Event(), []
    # 24 dates fit beside any kernel's own shared memory, 700 need more than the default limit.
    work = [market(24, fo.CudaExecutor(device=0)) for _ in range(4)] + [market(700, fo.CudaExecutor(device=0))]
    for kwargs in work:
        wanted.append(price(**kwargs))

    def run(k: int, calls: int) -> None:
        try:
            for _ in range(calls):
                if done.is_set():
                    return
                got = price(**work[k])
                assert got == wanted[k]
        except Exception as error:  # noqa: BLE001 - reported by the main thread
            failures.append(error)
        finally:
            if calls < 10**6:
                done.set()

    threads = [threading.Thread(target=run, args=(k, 300 if k == 4 else 10**6)) for k in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_a_smaller_launch_leaves_the_limit_of_a_larger_one() -> None:
    lib = BUILD / "libsmem_harness.so"
    src = HERE / "native" / "smem_harness.cu"
    deps = [src, CSRC / "lsm_kernels.h", CSRC / "lsm_device.cuh", CSRC / "fo_core.cuh"]
    if not lib.is_file() or lib.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        BUILD.mkdir(parents=True, exist_ok=True)
        subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17",
                        "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(lib)], check=True)
    h = ctypes.CDLL(str(lib))
    # What the first launch allows, what another allows before it is launched, what it takes.
    h.smem_check.argtypes = [ctypes.c_size_t] * 3
    for first, second in ((61440, 4096), (61440, 0), (200000, 61440), (4096, 200000)):
        assert h.smem_check(first, second, first) == 0
    assert h.smem_allow(ctypes.c_size_t(1 << 20)) == 1  # cudaErrorInvalidValue: more than a CTA has
