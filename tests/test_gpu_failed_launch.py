"""Calls whose FFT launches fail (z rows longer than the shared memory of an
SM holds; the launch itself returns the error, nothing runs with it): each
returns its error, and the sort of the next call begins from zeroed count
words, not from the offsets that the failed call left in them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = (4, 4, 6000)  # 3008 buckets; 2000 atoms take the sort's passes, not its one-CTA form
L = np.array([2.0, 2.1, 30.0, 0.1, 0.0, -0.2])


def test_calls_after_a_failed_launch(libsfac_path):
    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    rng = np.random.default_rng(4)
    x = rng.uniform(0, 2, size=(2000, 3))
    x[:, 2] *= 15.0
    q = rng.normal(size=2000)
    xd, qd = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
    dx, phi = torch.zeros_like(xd), torch.zeros_like(qd)
    torch.cuda.synchronize()
    s = SpmeSolver(L, K, 4, 3.0, 1.0)
    good = SpmeSolver(L, (24, 24, 96), 4, 3.0, 1.0)

    def energy():
        ev = good.solve(xd, qd)
        torch.cuda.synchronize()
        return ev.cpu().numpy()

    want = energy()
    for graphs in (0, 1, 0):
        s.lib.sfac_set_graphs(s.handle, graphs)
        for _ in range(2):
            s.sf.sfac(q, x)
            assert s.sf.last_error()[0] != 0
            with pytest.raises(RuntimeError, match="sfac_solve_device failed"):
                s.solve(xd, qd, dx, phi)
        torch.cuda.synchronize()  # no kernel faulted
    assert np.array_equal(energy(), want)
    # what needs no FFT works on the handle as on any other
    assert s.sf.real_space(q, x, 3.0, 0.5)[0] == good.sf.real_space(q, x, 3.0, 0.5)[0]
