"""The brick gather at the edges of its tiles, copies and grids, against the
thread-per-point gather of the same solve with dE/dL (which never takes
bricks): the same FP32 sums, term by term, so the same potentials; the
gradients' few FP64 products and sums may round differently."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs

pytestmark = pytest.mark.gpu

TRI = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])


def both(K, order, n, s):
    """(phi, dx) of the plain solve and of the one with dE/dL."""
    import ctypes

    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    rng = np.random.default_rng(7)
    x = torch.tensor(s(rng) @ configs.LofS(TRI), device="cuda")
    q = torch.tensor(rng.normal(0, 0.5, size=n), device="cuda")
    sv = SpmeSolver(TRI, K, order, 3.2, configs.MAX_M_FACTOR * 3.2)
    route = sv.lib.sfac_debug_gather_route
    route.argtypes = [np.ctypeslib.ndpointer(np.int32, shape=(3,), flags="C_CONTIGUOUS"), ctypes.c_int, ctypes.c_int]
    assert route(np.asarray(K, np.int32), order, n) == 2
    out = [[torch.full_like(q, np.nan), torch.full_like(x, np.nan)] for _ in range(2)]
    ev, dEdL = torch.zeros(7, dtype=torch.float64, device="cuda"), torch.zeros(6, dtype=torch.float64, device="cuda")
    cell = sv.lib.sfac_solve_device_cell
    cell.argtypes, cell.restype = [ctypes.c_void_p, ctypes.c_int] + [ctypes.c_void_p] * 6, ctypes.c_int
    torch.cuda.synchronize()
    sv.solve(x, q, out[0][1], out[0][0])
    assert cell(sv.handle, n, x.data_ptr(), q.data_ptr(), out[1][1].data_ptr(), out[1][0].data_ptr(), ev.data_ptr(),
                dEdL.data_ptr()) == 0
    torch.cuda.synchronize()
    return out


def check(out):
    import torch

    (phi, dx), (phi1, dx1) = out
    assert torch.equal(phi, phi1)
    # three products and two sums of terms below 3 max |dx| / min |cos| of this box: 8 roundings of 2^-53 each
    assert (dx - dx1).abs().max() <= 8 * 2.0**-53 * 4 * dx1.abs().max()


@pytest.mark.parametrize("K,order,n", [
    ((130, 129, 100), 6, 122880),  # ragged in x and y, a z brick of 4 cells, 16-byte copies; the smallest count
    ((130, 129, 102), 8, 70001),   # 8-byte copies
    ((200, 129, 101), 6, 262144),  # odd rows: 4-byte copies
    ((200, 129, 101), 8, 262144),
    ((9, 700, 384), 6, 122880),    # x shorter than a tile
    ((300, 5, 700), 8, 70000),     # y shorter than the stencil
    ((300, 300, 20), 6, 122880),   # rows shorter than a tile's
    ((400, 300, 6), 8, 70000),     # rows shorter than the stencil
    ((192, 192, 192), 8, 65536),   # few points per brick
    ((160, 160, 160), 6, 1500000), # more points per brick than one list holds
])
def test_bricks_against_one_thread_per_point(libsfac_path, K, order, n):
    check(both(K, order, n, lambda rng: rng.uniform(0, 1, size=(n, 3))))


def test_empty_bricks(libsfac_path):
    n, part = 200000, np.array([1.0, 0.5, 0.7])
    check(both((144, 160, 160), 6, n, lambda rng: part * rng.uniform(0, 1, size=(n, 3))))


def _clusters(n, *parts):
    """Shares of the points (the rest: the whole box) in cubes (share, corner, side) of the box."""
    def s(rng):
        u, a = rng.uniform(0, 1, size=(n, 3)), 0
        for share, corner, side in parts:
            b = a + int(share * n)
            u[a:b] = corner + side * u[a:b]
            a = b
        return u[rng.permutation(n)]

    return s


@pytest.mark.parametrize("K,order,n,parts", [
    ((144, 160, 160), 6, 200000, [(1.0, 0.45, 0.45)]),            # a droplet in a tenth of the box
    ((160, 160, 160), 8, 70000, [(1.0, 0.98, 0.1)]),              # across the boundaries
    ((130, 129, 100), 6, 122880, [(0.5, 0.1, 0.001)]),            # one bucket with half of the points
    ((200, 129, 101), 8, 262144, [(0.3, 0.5, 0.2), (0.2, 0.1, 0.02)]),
    ((9, 700, 384), 6, 122880, [(0.9, 0.3, 0.3)]),
    ((300, 300, 20), 6, 122880, [(0.2, 0.7, 0.05)]),
    ((160, 160, 160), 6, 1000000, [(0.00003, 0.2, 1e-4)]),        # 30 points more in one of evenly filled buckets
])
def test_crowded_buckets(libsfac_path, K, order, n, parts):
    """Clusters of every size: by bricks or, where the sort finds a bucket
    above the limit, by one thread per point."""
    check(both(K, order, n, _clusters(n, *parts)))


def test_every_solve_decides_anew(libsfac_path):
    """Evenly filled and crowded systems in turn on one handle, through its
    graph: each has the bits of a handle of its own."""
    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    K, order, n = (160, 160, 160), 6, 150000
    rng = np.random.default_rng(3)
    x = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    q = torch.tensor(rng.normal(size=n), device="cuda")
    out = [torch.empty_like(x), torch.empty_like(q)]
    sets = [torch.tensor(side * rng.uniform(0, 1, size=(n, 3)) @ configs.LofS(TRI), device="cuda") for side in (1, 0.1)]

    def solve(s, k):
        x.copy_(sets[k])
        torch.cuda.synchronize()
        s.solve(x, q, *out)
        torch.cuda.synchronize()
        return [a.clone() for a in out]

    new = lambda: SpmeSolver(TRI, K, order, 3.2, configs.MAX_M_FACTOR * 3.2)  # noqa: E731
    want = [solve(new(), k) for k in (0, 1)]
    one = new()
    for k in (0, 1, 0, 0, 1, 1, 0):
        for a, b in zip(solve(one, k), want[k]):
            assert torch.equal(a, b)
