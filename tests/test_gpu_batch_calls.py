"""SpmeBatch calls: boxes changed through a plan, arguments of other shapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(40, (24, 24, 24), 4), (60, (24, 25, 27), 6)]
L0 = np.array([[2.5, 2.4, 2.6, 0.2, -0.1, 0.3], [2.2, 2.3, 2.6, 0.0, 0.1, -0.3]])


def _inputs():
    import torch

    rng = np.random.default_rng(5)
    N = sum(s[0] for s in SHAPES)
    return (torch.tensor(rng.uniform(0, 2.2, size=(N, 3)), device="cuda"),
            torch.tensor(rng.normal(size=N), device="cuda"))


def test_box_set_through_a_plan(libsfac_path):
    """A plan's box set between two calls of its batch is not taken for the
    box of the calls: every call solves in the boxes that it is given."""
    import torch

    from ewaldcorrel_b200.autograd import SpmeBatch

    batch = SpmeBatch(SHAPES)
    x, q = _inputs()
    L1 = 1.1 * L0
    want0, want1 = batch(x, q, torch.tensor(L0)).clone(), batch(x, q, torch.tensor(L1)).clone()
    assert not torch.equal(want0, want1)
    batch.plans[0].set_box(L0[0])
    assert torch.equal(batch(x, q, torch.tensor(L1)), want1)
    batch.plans[1].set_box(L0[1])
    assert torch.equal(batch(x, q, torch.tensor(L0)), want0)


def test_shapes_of_the_arguments(libsfac_path):
    """Fewer rows than charges, or fewer boxes than systems, are refused, not
    broadcast over the systems; rows past the charges are not read."""
    import torch

    from ewaldcorrel_b200.autograd import SpmeBatch, spme_energy

    x, q = _inputs()
    L = torch.tensor(L0)
    batch, one = SpmeBatch(SHAPES), SpmeBatch(SHAPES[:1])
    n = SHAPES[0][0]
    want, want1 = batch(x, q, L).clone(), one(x[:n], q[:n], L[:1]).clone()
    for a, b in ((x[:1], q[:n]), (x[:n], q[:1]), (x[0], q[:n]), (x[: n - 1], q[:n]), (x[:n], q[: n - 1]),
                 (x[:n, :1], q[:n]), (x[:n], q[:n, None]), (x[:n], q[0])):
        with pytest.raises((RuntimeError, IndexError)):
            one(a, b, L[:1])
    with pytest.raises(RuntimeError):
        spme_energy(x[:1], q[:n], L[0], *SHAPES[0][1:])
    same = torch.tensor(np.stack([L0[0], L0[0]]))
    batch(x, q, same)
    for boxes in (L[:1], same[:1]):  # whatever the boxes of the call before
        with pytest.raises(IndexError):
            batch(x, q, boxes)
    more = torch.cat([x, x]), torch.cat([q, q]), torch.cat([L, L])
    assert torch.equal(batch(*more), want)
    assert torch.equal(one(x, q, L), want1)
