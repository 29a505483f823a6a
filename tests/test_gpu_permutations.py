"""Index permutations around their kernels' edges: dimensions below and above 8 and 16, runs that merge into rows
longer than a segment (1024), and tiles with remainders, through the residual and both transformations."""

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v,n_J,n_vec", [(7, 41, 9, 1), (8, 33, 130, 3), (9, 8, 40, 2), (15, 16, 33, 2), (17, 36, 8, 1)])
def test_edges(n_o, n_v, n_J, n_vec):
    from et_b200 import CCSD
    s = make_system(n_o, n_v, n_J, seed=n_o)
    ref = oc.CCSDSystem(s.L_mo, s.h_mo, s.eps, s.n_o)
    rng = np.random.default_rng(n_v)
    ref.set_amplitudes(0.05 * rng.standard_normal(ref.n_amp))
    C = rng.standard_normal((ref.n_amp, n_vec))
    with CCSD(n_o, n_v, n_J) as gpu:
        gpu.set_system(s.L_mo, s.h_mo, s.eps)
        gpu.set_amplitudes(ref.get_amplitudes())
        om, om_ref = gpu.construct_omega(), ref.omega()
        # FP64 sums in another order
        assert np.abs(om - om_ref).max() <= 1e-13 * max(1.0, np.abs(om_ref).max()) * np.sqrt(n_v)
        rho, sig = gpu.jacobian_transformation(C), gpu.jacobian_transpose_transformation(C)
        for k in range(n_vec):
            r = ref.jacobian_transformation(C[:, k])
            assert np.abs(rho[:, k] - r).max() <= 1e-12 * max(1.0, np.abs(r).max())
        dots = C.T @ rho
        assert np.abs(dots - sig.T @ C).max() <= 1e-11 * max(1.0, np.abs(dots).max())
