"""Memory of the sort's slots: none where the sort does not take them (above
16 MB), for the spread's sort (whose slots lie on the real grid) and for the
real-space term's."""
import ctypes

import numpy as np
import pytest

MB = 1 << 20
ROW_IMAGE = 168  # bytes of a row's image table: 4 images of 4 doubles and 2 ints, 2 ints


def _footprint(lib, K, n):
    f = lib.sfac_footprint_bytes
    f.argtypes = [np.ctypeslib.ndpointer(np.int32, shape=(3,), flags="C_CONTIGUOUS"), ctypes.c_int]
    f.restype = ctypes.c_ulong
    return int(f(np.asarray(K, np.int32), n))


@pytest.mark.parametrize("K", [(1024, 1024, 1), (1024, 512, 4), (512, 512, 33)])
def test_footprint_without_slots(libsfac_path, K):
    """Grids of more than 131,072 buckets: what a handle holds on the device
    and in pinned memory, without 128 bytes per bucket for slots."""
    lib = ctypes.CDLL(libsfac_path)
    rows, ldim, nb = K[0] * K[1], K[2] // 2 + 1, K[0] * K[1] * ((K[2] + 31) // 32)
    grids = 4 * rows * K[2] + 8 * rows * ldim
    counts = 4 * (3 * nb + 4096)
    tables = 16 * sum(K) + ROW_IMAGE * rows + 8 * 8 * (K[1] * ldim // 8 + 592)  # moduli, twiddles, row images, partials
    host = 16 * rows * ldim + 4 * rows * K[2]
    atoms = 160 * (1000 * 3 // 2 + 64)  # sort buffers and gather staging of 1000 atoms
    assert _footprint(lib, K, 1000) <= grids + counts + tables + host + atoms


def _device_bytes(make):
    import torch

    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    keep = make()
    torch.cuda.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    return free0 - free1, keep


@pytest.mark.gpu
def test_device_memory_without_slots(libsfac_path):
    from ewaldcorrel_b200 import ewald as E

    L = np.array([10.0, 10.0, 10.0, 0, 0, 0])
    warm = E.Sfac(L, np.array([16, 16, 16]), 4)  # context, modules
    x, q = np.random.default_rng(0).uniform(0, 10, size=(500, 3)), np.ones(500)
    warm.real_space(q, x, 3.0, 1.0)
    # a thin grid: 1M buckets, 128 MB of slots, 16 MB of grid
    K = np.array([1024, 1024, 4])
    used, s = _device_bytes(lambda: E.Sfac(L, K, 4))
    assert used < _footprint(s._libsfac, K, 1)
    del s
    # a fine coarse grid: 2.1M cells, 134 MB of slots, 25 MB of counts
    used, _ = _device_bytes(lambda: warm.real_space(q, x, 3.0, 2.0 * 10.0 / 128))
    assert used < 64 * MB


@pytest.mark.gpu
def test_real_space_count_words(libsfac_path):
    """The real-space sort keeps, and zeroes on every call, one count word per
    coarse cell: 16.8M cells here, 67 MB; head and tail counts are the spread's."""
    from ewaldcorrel_b200 import ewald as E

    L = np.array([10.0, 10.0, 10.0, 0, 0, 0])
    s = E.Sfac(L, np.array([16, 16, 16]), 4)
    x, q = np.random.default_rng(0).uniform(0, 10, size=(500, 3)), np.ones(500)
    s.real_space(q, x, 3.0, 1.0)
    used, _ = _device_bytes(lambda: s.real_space(q, x, 3.0, 2.0 * 10.0 / 256))
    assert used < 2 * 4 * 256**3
