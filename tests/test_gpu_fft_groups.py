"""The FFT passes by groups of stages (k_fft_groups.cu) against the FP64 oracle:
every compiled group in either place, odd planes (rows paired per plane), one
line more than a CTA holds, and each axis alone."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs
from oracle import oracle as O
from tests.spme_testlib import ENERGY_RTOL, VIRIAL_RTOL

pytestmark = pytest.mark.gpu

L = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])


@pytest.mark.parametrize("K", [
    (125, 9, 8),      # x alone: [5,5] [5]
    (162, 5, 6),      # [2,3,3] [3,3]
    (200, 7, 5),      # [4,2] [5,5]
    (216, 3, 4),      # [4,2] [3,3,3]
    (243, 1, 9),      # [3,3] [3,3,3]
    (250, 2, 2),      # [2,5] [5,5]
    (147, 3, 5),      # [3,7] [7]
    (189, 4, 3),      # [3,3,3] [7]
    (252, 3, 3),      # [4,3] [3,7]
    (8, 125, 64),     # y and z: [4,4] [4]; 125 odd rows per plane
    (5, 32, 125),     # [4] [4,2]
    (3, 162, 21),     # [3] [7]
    (3, 20, 125),     # [4] [5]
    (2, 243, 35),     # [5] [7], odd planes
    (2, 216, 30),     # [2,3] [5]
    (2, 45, 200),     # [3,3] [5], odd planes
    (3, 60, 189),     # [4,3] [5], odd z
    (1, 162, 75),     # [3,5] [5], odd z
    (4, 125, 100),    # [4,5] [5]
    (2, 256, 162),    # planes too large for one CTA: rows paired over all planes
    (1, 225, 250),    # the same, odd planes
    (125, 128, 162),  # all three axes
])
def test_group_passes_against_oracle(libsfac_path, oracle_built, K):
    from ewaldcorrel_b200 import ewald as E

    rng = np.random.default_rng(5)
    n = 500
    x = rng.uniform(0, 1, size=(n, 3)) @ configs.LofS(L)
    q = rng.normal(0, 0.5, size=n)
    out = []
    for cls in (E.Sfac, O.OracleSfac):
        s = cls(L, np.array(K), 4)
        s.set_ewald(3.2, configs.MAX_M_FACTOR * 3.2)
        s.sfac(q, x)
        S = np.array(s.get_S())
        e0 = s.en()
        vir = np.zeros(6)
        e1 = s.de1(vir)
        out.append((S, e0, e1, vir, s.get_grid()))
    (S, e0, e1, vir, grid), (So, _, eo, viro, grido) = out
    # FP32 spreading and transforms: as the parity tests of the other lengths
    assert np.abs(S - So).max() <= 5e-6 * np.abs(So).max()
    assert e0 == e1
    assert abs(e1 - eo) <= ENERGY_RTOL * abs(eo)
    assert np.abs(vir - viro).max() <= VIRIAL_RTOL * np.abs(viro).max()
    assert np.abs(grid - grido).max() <= 1e-5 * np.abs(grido).max()
