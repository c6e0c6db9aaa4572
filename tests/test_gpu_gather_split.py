"""The gather with 8 lanes per point (k_gather.cu: orders 6 and 8, few points)
against the FP64 oracle, sorted (device solve) and in input order (de2, potl)."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs
from oracle import oracle as O
from tests.spme_testlib import FORCE_RRMS, POT_RRMS, rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,order,n", [
    ((16, 18, 20), 6, 1),          # a single point
    ((5, 4, 7), 6, 17),            # axes shorter than the stencil, odd rows, one point past a CTA
    ((24, 20, 22), 8, 1000),       # z runs that wrap beside ones that do not
    ((40, 36, 33), 8, 24576),      # the most points
    ((40, 36, 33), 6, 24577),      # one more: thread per point
])
def test_split_gather_against_oracle(libsfac_path, oracle_built, K, order, n):
    import torch

    from ewaldcorrel_b200.device import SpmeSolver

    L = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])
    rng = np.random.default_rng(4)
    x = rng.uniform(-0.5, 1.5, size=(n, 3)) @ configs.LofS(L)
    q = rng.normal(0, 0.5, size=n)
    beta, max_m = 3.2, configs.MAX_M_FACTOR * 3.2
    o = O.OracleSfac(L, np.array(K), order)
    o.set_ewald(beta, max_m)
    o.sfac(q, x)
    o.de1(np.zeros(6))
    dxo, phio = np.zeros((n, 3)), np.zeros(n)
    o.de2(n, q, x, dxo)
    o.potl(n, x, phio)
    scale = np.sqrt(np.mean(phio**2)) * np.sqrt(np.mean(q**2)) * beta  # a lone point's force is a rounding residue

    s = SpmeSolver(L, K, order, beta, max_m)
    xd, qd = torch.tensor(x, device=s.device), torch.tensor(q, device=s.device)
    dx, phi = torch.full_like(xd, np.nan), torch.full_like(qd, np.nan)
    dx1, phi1 = torch.full_like(xd, np.nan), torch.full_like(qd, np.nan)
    torch.cuda.synchronize()
    s.solve(xd, qd, dx, phi)
    s.solve(xd, qd, dx1, None)
    s.solve(xd, qd, None, phi1)
    torch.cuda.synchronize()
    assert torch.equal(dx, dx1) and torch.equal(phi, phi1)
    s.sf.sfac(q, x)
    s.sf.de1(np.zeros(6))
    dxh, phih = np.full((n, 3), np.nan), np.full(n, np.nan)
    s.sf.de2(n, q, x, dxh)
    s.sf.potl(n, x, phih)
    for d, p in ((dx.cpu().numpy(), phi.cpu().numpy()), (dxh, phih)):
        assert rel_rms(d, dxo, floor=scale) <= FORCE_RRMS
        assert rel_rms(p, phio) <= POT_RRMS
