"""SpmeBatch's common buffers under calls from several streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_on_alternating_streams(libsfac_path):
    """A batch called from two streams in turn, without a wait between: the
    common buffers of the first call are not overwritten by the second."""
    import torch

    from ewaldcorrel_b200.autograd import SpmeBatch

    rng = np.random.default_rng(3)
    shapes = [(3, (24, 24, 24), 4), (0, (24, 25, 27), 4), (700, (32, 30, 36), 6), (64, (24, 24, 24), 4)]
    N = sum(s[0] for s in shapes)
    batch = SpmeBatch(shapes)
    L = torch.tensor([[2.5, 2.4, 2.6, 0.2, -0.1, 0.3]] * len(shapes), dtype=torch.float64)
    sets = [(torch.tensor(rng.uniform(0, 2.4, size=(N, 3)), device="cuda"), torch.tensor(rng.normal(size=N), device="cuda"))
            for _ in range(2)]

    def grads(x, q):
        x, q = x.clone().requires_grad_(), q.clone().requires_grad_()
        E = batch(x, q, L)
        return (E.detach(),) + torch.autograd.grad(E.sum(), (x, q))

    want = []
    for s in sets:
        want.append([t.clone() for t in grads(*s)])
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for k in range(6):
        with torch.cuda.stream(streams[k % 2]):
            got.append(grads(*sets[k % 2]))
    torch.cuda.synchronize()
    for k in range(6):
        for a, b in zip(got[k], want[k % 2]):
            assert torch.equal(a, b)
