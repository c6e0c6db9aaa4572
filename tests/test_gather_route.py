"""Which gather a solve takes: bricks only where they were measured faster
than one thread per point (few points per brick copy too much, few bricks
leave the chip idle)."""
import ctypes

import numpy as np
import pytest


@pytest.fixture(scope="module")
def route(libsfac_path):
    f = ctypes.CDLL(libsfac_path).sfac_debug_gather_route
    f.argtypes = [np.ctypeslib.ndpointer(np.int32, shape=(3,), flags="C_CONTIGUOUS"), ctypes.c_int, ctypes.c_int]
    return lambda K, order, n: f(np.asarray(K, np.int32), order, n)


@pytest.mark.parametrize("K,order,n", [
    ((256,) * 3, 6, 70_000), ((256,) * 3, 8, 66_000), ((384,) * 3, 6, 1_000_000), ((384,) * 3, 8, 260_000),  # sparse
    ((48,) * 3, 6, 130_000), ((48,) * 3, 8, 130_000), ((72,) * 3, 6, 260_000), ((72,) * 3, 8, 520_000),  # few bricks
    ((96,) * 3, 6, 66_000), ((128,) * 3, 6, 512_000), ((104,) * 3, 8, 69_000), ((96,) * 3, 8, 260_000), ((9, 10, 12), 6, 66_000),
    ((195,) * 3, 6, 271_000), ((75,) * 3, 8, 520_000), ((195,) * 3, 8, 262_143),  # odd rows
    ((256,) * 3, 4, 1_000_000), ((256,) * 3, 2, 1_000_000),
    ((128,) * 3, 6, 100_000), ((256,) * 3, 6, 24_577),
])
def test_one_thread_per_point(route, K, order, n):
    assert route(K, order, n) == 0


@pytest.mark.parametrize("K,order,n", [
    ((256,) * 3, 6, 1_048_576), ((256,) * 3, 6, 520_000), ((160,) * 3, 6, 150_000), ((128,) * 3, 6, 128_000),
    ((120,) * 3, 6, 168_750), ((160,) * 3, 6, 1_600_000), ((256,) * 3, 8, 1_048_576), ((256,) * 3, 8, 130_000),
    ((192,) * 3, 8, 66_000), ((128,) * 3, 8, 512_000), ((96,) * 3, 8, 130_000),
    ((175,) * 3, 6, 327_110), ((225,) * 3, 8, 262_144),
])
def test_bricks(route, K, order, n):
    assert route(K, order, n) == 2


def test_lanes(route):
    assert route((40,) * 3, 6, 4000) == 1 and route((40,) * 3, 4, 4000) == 0
