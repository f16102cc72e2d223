"""The tiles of a mini-batch (`Tiles`, gamma_b200/csrc/tiles.h, which the training
kernel's loop runs on), on the host through the test suite's self-test library:
every block ends, also where its last step would pass the largest 32-bit int."""
import ctypes
import os

import pytest

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gamma_b200", "lib",
                   "libgamma_selftest.so")
INT_MAX = 2**31 - 1


@pytest.mark.parametrize("n", [1, 64, 65, 9472, 9473, INT_MAX - 148 * 64, INT_MAX - 64, INT_MAX - 1, INT_MAX])
def test_blocks_take_every_tile_once(n):
    assert os.path.exists(LIB), "build the self-test library: make -C gamma_b200/csrc"
    f = ctypes.CDLL(LIB).gb_selftest_tiles
    f.argtypes, f.restype = [ctypes.c_int] * 4, ctypes.c_longlong
    tiles = -(-n // 64)
    for blocks in (1, 147, 148):
        for block in {0, 1, blocks // 2, blocks - 1}:
            want = len(range(block, tiles, blocks))
            assert f(n, 64, block, blocks) == want, (n, block, blocks)
