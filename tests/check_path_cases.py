"""Solves through the index-checking library (libsfac_check.so, loaded because
EWALDCORREL_LIBSFAC names it) on the paths that tests/check_cases.py does not
reach: the gathers by bricks, by lanes and of crowded systems, the FFT passes
by groups of stages, the sort's routes, the real-space sort, a batch, and the
calls after a failed launch.  Prints one JSON line; run as a child process by
tests/test_gpu_check_paths.py.
"""
from __future__ import annotations

import ctypes
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

from ewaldcorrel_b200 import configs  # noqa: E402
from ewaldcorrel_b200 import ewald as E  # noqa: E402
from tests import spme_testlib as T  # noqa: E402

L = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])
BETA, MAX_M = 3.2, configs.MAX_M_FACTOR * 3.2

# (name, K, order, atoms, side of the cube of the box that holds them, route of the gather)
CASES = [
    ("bricks_p6", (130, 129, 100), 6, 122880, 1.0, 2),
    ("bricks_p8_8_byte_copies", (130, 129, 102), 8, 70001, 1.0, 2),
    ("bricks_p8_odd_rows", (200, 129, 101), 8, 262144, 1.0, 2),
    ("bricks_p6_x_below_a_tile", (9, 700, 384), 6, 122880, 1.0, 2),
    ("crowded_p6", (130, 129, 100), 6, 122880, 0.3, 2),
    ("crowded_p8", (130, 129, 102), 8, 70001, 0.2, 2),
    ("lanes_p6", (40, 36, 64), 6, 4000, 1.0, 1),
    ("lanes_p8", (24, 24, 75), 8, 3000, 1.0, 1),
    ("groups_x", (216, 24, 20), 4, 3000, 1.0, 0),
    ("groups_y_odd_planes", (8, 125, 64), 4, 2000, 1.0, 0),
    ("groups_z", (12, 24, 125), 6, 2000, 1.0, 1),
    ("groups_xyz", (125, 162, 200), 4, 30000, 1.0, 0),
    ("slots_chain", (64, 64, 64), 4, 9000, 0.12, 0),
    ("slots_merge_sort", (64, 64, 64), 4, 9000, 0.02, 0),
    ("scatter_merge_sort", (64, 64, 64), 4, 60000, 0.02, 0),
    ("one_cta_sort", (32, 32, 32), 4, 1024, 1.0, 0),
    ("one_cta_merge_sort", (32, 32, 32), 4, 1024, 0.02, 0),
]


def main():
    import torch

    from ewaldcorrel_b200.autograd import SpmeBatch
    from ewaldcorrel_b200.device import SpmeSolver

    _, _, lib = E.describe_sfac()
    lib.sfac_check_take.argtypes = [ctypes.POINTER(ctypes.c_ulonglong)]
    lib.sfac_debug_gather_route.argtypes = [np.ctypeslib.ndpointer(np.int32, shape=(3,), flags="C_CONTIGUOUS"),
                                            ctypes.c_int, ctypes.c_int]

    def take():
        w = ctypes.c_ulonglong(0)
        return lib.sfac_check_take(ctypes.byref(w)), hex(w.value)

    out = {"library": os.environ.get("EWALDCORREL_LIBSFAC", ""), "enabled": lib.sfac_check_enabled(), "start": take(),
           "cases": []}

    def add(name, **more):
        m, w = take()
        out["cases"].append(dict(case=name, module=m, word=w, **more))

    for i, (name, K, order, n, side, route) in enumerate(CASES):
        rng = np.random.default_rng(200 + i)
        x = (0.4 + side * (rng.uniform(0, 1, size=(n, 3)) - 0.4)) @ configs.LofS(L)
        # like charges in a cluster: no FP32 cancellation on the few grid points they reach
        q = np.ones(n) if side < 1.0 else np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
        assert lib.sfac_debug_gather_route(np.asarray(K, np.int32), order, n) == route, name
        s = SpmeSolver(L, K, order, BETA, MAX_M)
        xd, qd = torch.tensor(x, device=s.device), torch.tensor(q, device=s.device)
        dx, phi = torch.empty_like(xd), torch.empty_like(qd)
        torch.cuda.synchronize()
        for a, b in ((dx, phi), (dx, None), (None, phi), (dx, phi)):
            ev = s.solve(xd, qd, a, b)
        torch.cuda.synchronize()
        o = T.solve("oracle", L, K, order, x, q, beta=BETA, max_m=MAX_M)
        add(name, energy_rel=abs(float(ev[0]) - o["en"]) / abs(o["en"]),
            force_rrms=T.rel_rms(dx.cpu().numpy(), o["dx"]), pot_rrms=T.rel_rms(phi.cpu().numpy(), o["phi"]))
        del s

    rng = np.random.default_rng(1)
    x, q = rng.uniform(0, 1, size=(20000, 3)) @ configs.LofS(L), rng.normal(size=20000)
    s = E.Sfac(L, np.array([16, 16, 16]), 4)
    for n, rcut in ((20000, 0.9), (20000, 0.05), (700, 0.9), (700, 0.05)):  # slots, many cells, one CTA, scatter
        s.real_space(q[:n], x[:n], 3.0, rcut)
    add("real_space")

    shapes = [(3, (24, 24, 24), 4), (0, (24, 25, 27), 4), (700, (32, 30, 36), 6), (30000, (48, 45, 40), 8)]
    N = sum(t[0] for t in shapes)
    batch = SpmeBatch(shapes)
    xt, qt = torch.tensor(rng.uniform(0, 2.8, size=(N, 3)), device="cuda"), torch.tensor(rng.normal(size=N), device="cuda")
    for _ in range(2):
        batch(xt, qt, torch.tensor(np.stack([L] * 4)))
    torch.cuda.synchronize()
    add("batch")

    # the launch of z rows longer than an SM's shared memory fails; the calls after it begin from clean counts
    s = E.Sfac(L, np.array([4, 4, 6000]), 4)
    for _ in range(3):
        s.sfac(q[:2000], x[:2000])
    add("failed_launches", failed=int(s.last_error()[0] != 0))
    print(json.dumps(out))


if __name__ == "__main__":
    main()
