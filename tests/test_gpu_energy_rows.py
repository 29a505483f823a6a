"""Correlation energy from packed rows of t2: odd and even numbers of pairs, one pair, fewer and more rows
than the grid's blocks, against the oracle."""

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v", [(1, 1), (1, 2), (3, 5), (4, 33), (2, 128), (16, 149), (23, 105)])
def test_energy(n_o, n_v):
    from et_b200 import CCSD
    s = make_system(n_o, n_v, 9, seed=n_v)
    rng = np.random.default_rng(n_o)
    n1 = n_o * n_v
    t = 0.05 * rng.standard_normal(n1 + n1 * (n1 + 1) // 2)
    ref = oc.CCSDSystem(s.L_mo, s.h_mo, s.eps, s.n_o)
    ref.set_amplitudes(t)
    e_ref = ref.energy()
    with CCSD(n_o, n_v, 9) as gpu:
        gpu.set_system(s.L_mo, s.h_mo, s.eps)
        gpu.set_amplitudes(t)
        # a sum of nov^2 products, rounded in another order
        assert abs(gpu.calculate_energy() - e_ref) <= 1e-14 * n1 * max(1.0, abs(e_ref))
