"""The brick gather (k_gather.cu: orders 6 and 8, many points) against the FP64
oracle, at the sizes where its tiles, copies and point lists have edges."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs
from oracle import oracle as O
from tests.spme_testlib import FORCE_RRMS, POT_RRMS, rel_rms

pytestmark = pytest.mark.gpu

TRI = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])


@pytest.mark.parametrize("K,order,n,part", [
    ((33, 17, 96), 6, 65536, 1.0),   # ragged bricks, 16-byte copies; the smallest count that takes them
    ((24, 40, 50), 8, 70001, 1.0),   # 8-byte copies, a partial z brick
    ((9, 10, 12), 6, 66000, 1.0),    # axes shorter than a tile, more points per brick than one list holds
    ((40, 36, 75), 6, 262144, 1.0),  # odd rows: 4-byte copies
    ((48, 64, 128), 8, 66000, 0.3),  # points in a corner: empty bricks beside full ones
])
def test_brick_gather_against_oracle(libsfac_path, oracle_built, K, order, n, part):
    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    rng = np.random.default_rng(7)
    x = (part * rng.uniform(0, 1, size=(n, 3))) @ configs.LofS(TRI)
    q = rng.normal(0, 0.5, size=n)
    beta, max_m = 3.2, configs.MAX_M_FACTOR * 3.2
    s = SpmeSolver(TRI, K, order, beta, max_m)
    dev = s.device
    xd, qd = torch.tensor(x, device=dev), torch.tensor(q, device=dev)
    torch.cuda.synchronize(dev)
    dx, phi = torch.full_like(xd, np.nan), torch.full_like(qd, np.nan)
    dx1, phi1 = torch.full_like(xd, np.nan), torch.full_like(qd, np.nan)
    torch.cuda.synchronize(dev)
    s.solve(xd, qd, dx, phi)
    s.solve(xd, qd, dx1, None)
    s.solve(xd, qd, None, phi1)
    torch.cuda.synchronize(dev)
    assert torch.equal(dx, dx1) and torch.equal(phi, phi1)  # each output alone: the same bits
    o = O.OracleSfac(TRI, np.array(K), order)
    o.set_ewald(beta, max_m)
    o.sfac(q, x)
    o.de1(np.zeros(6))
    dxo, phio = np.zeros((n, 3)), np.zeros(n)
    o.de2(n, q, x, dxo)
    o.potl(n, x, phio)
    assert rel_rms(dx.cpu().numpy(), dxo) <= FORCE_RRMS
    assert rel_rms(phi.cpu().numpy(), phio) <= POT_RRMS
