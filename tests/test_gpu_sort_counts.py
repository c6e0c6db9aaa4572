"""The cell sort's count words stay zero between calls (no memset heads a
sort): calls of every route on one handle, in any order, through graphs and
without, match fresh handles bit for bit."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,order", [((40, 36, 64), 6), ((24, 24, 75), 8), ((16, 125, 24), 4), ((11, 13, 34), 6)])
def test_calls_in_any_order_match_fresh_handles(libsfac_path, K, order):
    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    L = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])
    beta, max_m = 3.2, configs.MAX_M_FACTOR * 3.2
    rng = np.random.default_rng(2)
    # one CTA; slots; scatter and fix-up; the brick gather (which reads the buckets last); no atoms
    sizes = [600, 5000, 60000, 70000, 5000, 0, 70000, 600, 60000]
    xs, qs = {}, {}
    for n in set(sizes):
        xs[n] = torch.tensor(rng.uniform(0, 1, size=(n, 3)) @ configs.LofS(L), device="cuda")
        qs[n] = torch.tensor(rng.normal(0, 0.5, size=n), device="cuda")

    def solve(s, n):
        dx, phi = torch.zeros_like(xs[n]), torch.zeros_like(qs[n])
        torch.cuda.synchronize()
        ev = s.solve(xs[n], qs[n], dx, phi)
        torch.cuda.synchronize()
        return ev, dx, phi

    want = {n: solve(SpmeSolver(L, K, order, beta, max_m), n) for n in set(sizes)}
    s = SpmeSolver(L, K, order, beta, max_m)
    for graphs in (1, 0, 1):
        s.lib.sfac_set_graphs(s.handle, graphs)
        for n in sizes:
            for a, b in zip(solve(s, n), want[n]):
                assert torch.equal(a, b)
            if n == 5000:  # the host interface and an energy-only solve in between
                s.sf.sfac(qs[n].cpu().numpy(), xs[n].cpu().numpy())
                s.sf.en()
                s.solve(xs[n], qs[n])
