"""The backward kernel's waits: the exchange of the grid's sums gives up when a CTA's line never arrives,
wholly or in one half, every warp leaves and the status word says so; and the wait for a row's bulk copy
gives up when nothing completes it. The context stays usable. The failures are made without any fault, on
one CTA whose neighbours' lines the host lays out.
"""

from __future__ import annotations

import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
BUILD = HERE / "native" / "_build"
CSRC = HERE.parent / "finoptions-engine_b200" / "csrc"
SLOTS, USED, WARPS = 8, 6, 16
LIMIT = 300_000_000  # ns
OUTCOME = np.dtype([("total", "f8", (SLOTS, 2)), ("failed", "i4"), ("warps_left", "i4"), ("elapsed_ns", "u8")])


@pytest.fixture(scope="module")
def harness() -> ctypes.CDLL:
    lib = BUILD / "libexchange_harness.so"
    src = HERE / "native" / "exchange_harness.cu"
    deps = [src, *(CSRC / f for f in ("lsm_bulk_copy.cuh", "lsm_exchange.cuh", "lsm_sync.cuh", "lsm_common.cuh",
                                      "lsm_device.cuh", "lsm_kernels.h", "fo_core.cuh"))]
    if not lib.is_file() or lib.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        BUILD.mkdir(parents=True, exist_ok=True)
        subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17",
                        "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(lib)], check=True)
    dll = ctypes.CDLL(str(lib))
    assert dll.exchange_bytes() == OUTCOME.itemsize
    dll.exchange_check.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_uint,
                                   ctypes.c_ulonglong, ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    dll.copy_check.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong, ctypes.c_void_p,
                               ctypes.POINTER(ctypes.c_uint)]
    return dll


def exchange(h, red: np.ndarray, lines: np.ndarray, block: int, seq: int):
    out, flag = np.zeros(1, dtype=OUTCOME), ctypes.c_uint()
    assert h.exchange_check(red.ctypes.data, lines.ctypes.data, block, lines.shape[1], seq, LIMIT, out.ctypes.data,
                            ctypes.byref(flag)) == 0
    return out[0], flag.value


def grid_lines(h, sums: np.ndarray, block: int, seq: int) -> np.ndarray:
    """The two buffers [parity][CTA][slot][hi, lo] with every CTA's line of exchange `seq` but `block`'s, each
    written by the exchange itself: sums is [CTA][warp][slot]."""
    blocks = sums.shape[0]
    lines = np.zeros((2, blocks, SLOTS, 2))
    for b in range(blocks):
        if b == block:
            continue
        alone = np.zeros((2, blocks, SLOTS, 2))
        # Its neighbours' words carry the phase, so that it does not wait.
        alone.view(np.uint64)[seq & 1] = ((seq >> 1) & 1) ^ 1
        out, flag = exchange(h, sums[b], alone, b, seq)
        assert out["failed"] == 0 and flag == 0
        lines[seq & 1, b] = alone[seq & 1, b]
    return lines


@pytest.mark.parametrize("blocks, seq", [(2, 0), (5, 1), (33, 2), (161, 3)])
def test_the_grid_total_is_the_sum_of_the_lines(harness, blocks, seq) -> None:
    rng = np.random.default_rng(blocks)
    sums = rng.integers(1, 1 << 40, (blocks, WARPS, SLOTS)).astype(np.float64)
    out, flag = exchange(harness, sums[1], grid_lines(harness, sums, 1, seq), 1, seq)
    assert out["failed"] == 0 and flag == 0 and out["warps_left"] == WARPS
    np.testing.assert_array_equal(out["total"].sum(axis=1)[:USED], sums.sum(axis=(0, 1))[:USED])


@pytest.mark.parametrize("blocks, spread, signs", [(148, 2, False), (148, 30, False), (98, 2, True), (37, 20, True)])
def test_the_grid_total_rounds_to_the_exact_sum(harness, blocks, spread, signs) -> None:
    # Warp sums spread over 2 to 30 binary orders, of one sign or cancelling to a thousandth of their sum and
    # less: the exchanged total, of some 100 bits, rounds to the binary64 number nearest to the exact sum.
    rng = np.random.default_rng(spread + blocks)
    for seq in range(4):
        sums = np.exp2(rng.uniform(0.0, spread, (blocks, WARPS, SLOTS))) * rng.uniform(1.0, 2.0, (blocks, WARPS, SLOTS))
        if signs:
            sums[1::2] = -sums[0::2][: blocks // 2] * rng.uniform(0.999, 1.001, sums[1::2].shape)
        out, flag = exchange(harness, sums[0], grid_lines(harness, sums, 0, seq), 0, seq)
        assert out["failed"] == 0 and flag == 0
        got = out["total"].sum(axis=1)[:USED]
        assert got.tolist() == [math.fsum(sums[:, :, slot].ravel()) for slot in range(USED)]


@pytest.mark.parametrize("missing", ["all", "one", "high", "low"])
def test_a_line_that_never_arrives_ends_the_exchange(harness, missing) -> None:
    blocks, block, seq = 37, 0, 0
    sums = np.ones((blocks, WARPS, SLOTS))
    lines = grid_lines(harness, sums, block, seq)
    whole = lines.copy()
    if missing == "all":
        lines[:] = 0.0
    elif missing == "one":
        lines[0, 35] = 0.0
    else:  # half a word of one slot
        lines[0, 35, USED - 1, 0 if missing == "high" else 1] = 0.0
    out, flag = exchange(harness, sums[block], lines, block, seq)
    assert out["failed"] == 1 and flag == 1 and out["warps_left"] == WARPS
    assert 0.9 * LIMIT <= out["elapsed_ns"] < LIMIT + 1_000_000_000
    # Same device, next launch: with every line there the exchange passes.
    out, flag = exchange(harness, sums[block], whole, block, seq)
    assert out["failed"] == 0 and flag == 0 and out["elapsed_ns"] < LIMIT


def test_a_copy_that_nothing_completes_ends_its_wait(harness) -> None:
    src = np.arange(256, dtype=np.float64)

    def run(copy: int):
        out, flag = np.zeros(1, dtype=OUTCOME), ctypes.c_uint()
        assert harness.copy_check(src.ctypes.data, src.size, copy, LIMIT, out.ctypes.data, ctypes.byref(flag)) == 0
        return out[0], flag.value

    out, flag = run(0)
    assert out["failed"] == 1 and flag == 1
    assert 0.9 * LIMIT <= out["elapsed_ns"] < LIMIT + 1_000_000_000
    out, flag = run(1)
    assert out["failed"] == 0 and flag == 0 and out["total"][0, 0] == src.sum()
