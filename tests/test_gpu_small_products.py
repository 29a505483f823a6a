"""Small products in one launch: summed lengths N_J n_o, N_J n_v and n_o n_v around 64 and 1024 (one thread, a
warp, a block per element; one or more tables), against the oracle."""

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v,n_J", [(1, 2, 64), (2, 3, 32), (1, 5, 65), (3, 4, 341), (4, 4, 256), (5, 5, 205), (2, 7, 600)])
def test_lengths(n_o, n_v, n_J):
    from et_b200 import CCSD
    s = make_system(n_o, n_v, n_J, seed=n_J)
    ref = oc.CCSDSystem(s.L_mo, s.h_mo, s.eps, s.n_o)
    rng = np.random.default_rng(n_J)
    ref.set_amplitudes(0.05 * rng.standard_normal(ref.n_amp))
    C = rng.standard_normal((ref.n_amp, 2))
    with CCSD(n_o, n_v, n_J) as gpu:
        gpu.set_system(s.L_mo, s.h_mo, s.eps)
        gpu.set_amplitudes(ref.get_amplitudes())
        om, om_ref = gpu.construct_omega(), ref.omega()
        # FP64 sums of at most N_J n_v terms in another order
        assert np.abs(om - om_ref).max() <= 1e-13 * max(1.0, np.abs(om_ref).max())
        rho, sig = gpu.jacobian_transformation(C), gpu.jacobian_transpose_transformation(C)
        for k in range(2):
            r = ref.jacobian_transformation(C[:, k])
            assert np.abs(rho[:, k] - r).max() <= 1e-12 * max(1.0, np.abs(r).max())
        dots = C.T @ rho
        assert np.abs(dots - sig.T @ C).max() <= 1e-11 * max(1.0, np.abs(dots).max())
