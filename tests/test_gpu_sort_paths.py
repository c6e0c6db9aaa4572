"""The cell sort's three routes (one CTA, slots, scatter and fix-up; k_sort.cu)
against the oracle's stable sort, bit for bit, at the sizes where each begins
and where its buckets overflow."""
import numpy as np
import pytest

from ewaldcorrel_b200 import configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

L = np.array([3.0, 3.2, 2.9, 0.3, -0.2, 0.5])


@pytest.mark.parametrize("K,order,n,spread", [
    ((24, 24, 24), 4, 1, 1.0),           # one CTA: a single atom
    ((32, 32, 32), 4, 1024, 1.0),        # one CTA: full
    ((32, 32, 32), 4, 1024, 0.02),       # one CTA: buckets above the merge limit
    ((128, 64, 20), 6, 1000, 1.0),       # one CTA: the most buckets
    ((129, 64, 20), 6, 1000, 1.0),       # slots: one bucket more
    ((32, 32, 32), 4, 1025, 1.0),        # slots: one atom more
    ((40, 36, 75), 8, 9000, 0.35),       # slots: some buckets spill past their 16
    ((64, 64, 64), 4, 9000, 0.12),       # slots: long chains
    ((64, 64, 64), 4, 9000, 0.02),       # slots: buckets above the merge limit
    ((64, 64, 64), 4, 20480, 1.0),       # slots: a mean of 5, the last that takes them
    ((64, 64, 64), 4, 20481, 1.0),       # scatter and fix-up: one atom more
    ((64, 64, 64), 4, 60000, 0.02),      # scatter and fix-up: buckets above the merge limit
    ((512, 256, 31), 4, 3000, 1.0),      # slots: 131,072 buckets, the last that take them; tile sums while counting
    ((513, 256, 31), 4, 3000, 1.0),      # scatter and fix-up
])
def test_sort_routes_bit_exact(libsfac_path, oracle_built, K, order, n, spread):
    from ewaldcorrel_b200 import ewald as E

    rng = np.random.default_rng(11)
    s = 0.4 + spread * (rng.uniform(0, 1, size=(n, 3)) - 0.4)
    s[::7] = s[0]  # ties: equal cells keep the input order
    x = s @ configs.LofS(L)
    q = rng.normal(0, 0.5, size=n)
    sf = E.Sfac(L, np.array(K), order)
    sf.sfac(q, x)
    keys, perm = sf.debug_sort(n)
    okeys, operm, _ = O.OracleSfac(L, np.array(K), order).sort(x)
    assert np.array_equal(keys, okeys)
    assert np.array_equal(perm, operm)
