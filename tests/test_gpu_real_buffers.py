"""Device allocations of a real-space call that needs new buffers: a call
waits for every one of them.  Counted with the library's test hook (the n-th
allocation from now on fails once; the call returns an error and the next one
starts over)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _allocations(lib, call):
    """Device allocations of a call that succeeds; those before it fail."""
    for nth in range(1, 40):
        lib.sfac_debug_fail_alloc(nth)
        try:
            call()
        except RuntimeError:
            continue
        finally:
            lib.sfac_debug_fail_alloc(0)
        return nth - 1
    raise AssertionError("the call never succeeded")


def test_allocations_of_new_buffers(libsfac_path):
    from ewaldcorrel_b200 import ewald as E

    lib = E.describe_sfac()[2]
    lib.sfac_debug_fail_alloc.argtypes = [ctypes.c_int]
    L = np.array([3.0, 3.1, 3.2, 0.1, 0.2, -0.3])
    rng = np.random.default_rng(1)
    x, q = rng.uniform(0, 3, size=(700, 3)), rng.normal(size=700)
    s = E.Sfac(L, np.array([16, 16, 16]), 4)
    want = E.Sfac(L, np.array([16, 16, 16]), 4).real_space(q, x, 3.0, 0.9)
    got = []
    assert _allocations(lib, lambda: got.append(s.real_space(q, x, 3.0, 0.9))) <= 5
    for a, b in zip(got[0], want):
        assert np.array_equal(a, b)
    assert _allocations(lib, lambda: s.real_space(q, x, 3.0, 0.9)) == 0  # kept
    assert _allocations(lib, lambda: s.real_space(q, x, 3.0, 0.5)) <= 5  # another coarse grid
    assert _allocations(lib, lambda: s.real_space(np.tile(q, 2), np.tile(x, (2, 1)), 3.0, 0.5)) <= 5  # more points
