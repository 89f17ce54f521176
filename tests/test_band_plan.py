"""The band kernel's launch shape (hy_debug_band_plan) for every alphabet and lane arithmetic: each pass has
a warp in some round, and a block's shared memory stays within the device's. No GPU."""
import ctypes as C

import numpy as np
import pytest

from hyalite_b200 import _abi

LIMIT = 227 * 1024  # a block's shared memory on sm_100
WORD_BYTES = {0: lambda al: 8 * (al + 1), 1: lambda al: 4 * (al + 1) ** 2, 2: lambda al: 4 * (al + 1)}
SW, NW = 0, 1


def plan(arith, mode, al, qlen):
    out = np.zeros(6, np.uint64)
    assert _abi.lib.hy_debug_band_plan(arith, mode, al, qlen, LIMIT, out.ctypes.data_as(C.POINTER(C.c_uint64))) == 0
    return [int(x) for x in out]


@pytest.mark.parametrize("mode", [SW, NW])
@pytest.mark.parametrize("arith", [0, 1, 2])
def test_every_pass_placed_within_a_blocks_shared_memory(arith, mode):
    for al in range(1, 256 if arith != 1 else 40):
        for qlen in (1, 64, 128, 129, 300, 600, 1025, 1100, 2000, 4096, 4097, 6200, 11300, 16384, 16385, 19500, 30000, 40000, 61000):
            rows, gprof, warps, blocks, rounds, smem = plan(arith, mode, al, qlen)
            passes = -(-qlen // (32 * rows))
            assert rows in (4, 8) and 1 <= blocks <= 8 and 1 <= warps <= 16 and (not gprof or blocks == 1)
            assert warps * blocks * rounds >= passes > warps * blocks * (rounds - 1)
            # At least the slices and two rings.
            slices = 0 if gprof else warps * 32 * rows * WORD_BYTES[arith](al)
            assert slices + 2048 < smem <= LIMIT, (al, qlen)
            # One warp: its slice, two rings of 64 pairs, 66 codes, the copied columns, barriers and words.
            one = 128 * WORD_BYTES[arith](al) + 2 * 1024 + 272 + 2048 + 80
            assert gprof == (one > LIMIT), al


def test_four_rows_on_as_few_rounds_as_fit():
    assert plan(0, SW, 20, 128)[:5] == [4, 0, 1, 1, 1]
    assert plan(0, SW, 20, 129)[:5] == [4, 0, 2, 1, 1]
    assert plan(2, SW, 20, 5000)[:5] == [4, 0, 5, 8, 1]  # 40 passes
    assert plan(2, SW, 4, 16384)[:5] == [4, 0, 16, 8, 1]  # 128 passes
    assert plan(2, SW, 4, 16385)[:5] == [4, 0, 9, 8, 2]  # 129: two rounds of 65
    assert plan(2, NW, 4, 16385)[:5] == [8, 0, 9, 8, 1]  # 65 passes of 256 rows
    assert plan(0, NW, 120, 1000)[:5] == [4, 0, 1, 8, 1]  # a slice of 124 KB: one warp a block
    assert plan(0, NW, 250, 1000)[:5] == [8, 1, 4, 1, 1]  # a slice that fits no block
