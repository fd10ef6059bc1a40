"""The radix sort's scratch: 2048 keys to a tile, or 1024 up to 147,456 keys, and no more tiles than a sort
of n keys or a smaller one has."""

import ctypes

import pytest

FEW = 144 * 1024


@pytest.fixture(scope="module")
def scratch():
    from galaxy_formation_gb300 import build

    fn = ctypes.CDLL(build.build())["_ZN2gf15os_scratch_intsEi"]
    fn.restype, fn.argtypes = ctypes.c_size_t, [ctypes.c_int]
    return fn


def _needed(n):
    tiles = -(-n // 1024) if n <= FEW else -(-n // 2048)
    return 8 * 256 + 64 + 8 * 256 * tiles


SIZES = [1, 2, 1023, 1024, 1025, 100000, FEW - 1, FEW, FEW + 1, 200000, 2 * FEW, 2 * FEW + 1, 1 << 20, 4000000]


@pytest.mark.parametrize("n", SIZES)
def test_scratch_is_what_sorts_up_to_n_use(scratch, n):
    smaller = [k for k in (1, 1024, FEW, FEW + 1, n) if k <= n]
    assert scratch(n) == max(_needed(k) for k in smaller)
