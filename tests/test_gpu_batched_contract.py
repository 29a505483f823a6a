"""Products that run as strided batches of GEMMs over an output index (the trial index, or one between
the others) against the oracle: blocks of several trial vectors at sizes where the batched index is the
smallest, the largest or one of the orbital ranges, and where it has no second element."""

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v,n_J,n_vec", [(8, 9, 20, 2), (9, 8, 31, 5), (8, 24, 16, 1), (11, 17, 8, 3), (3, 40, 50, 4)])
def test_block_matches_single_vectors_and_oracle(n_o, n_v, n_J, n_vec):
    from et_b200 import CCSD
    s = make_system(n_o, n_v, n_J, seed=n_vec)
    ref = oc.CCSDSystem(s.L_mo, s.h_mo, s.eps, s.n_o)
    rng = np.random.default_rng(n_J)
    ref.set_amplitudes(0.05 * rng.standard_normal(ref.n_amp))
    C = rng.standard_normal((ref.n_amp, n_vec))
    with CCSD(n_o, n_v, n_J) as gpu:
        gpu.set_system(s.L_mo, s.h_mo, s.eps)
        gpu.set_amplitudes(ref.get_amplitudes())
        rho = gpu.jacobian_transformation(C)
        sig = gpu.jacobian_transpose_transformation(C)
        for k in range(n_vec):
            r = ref.jacobian_transformation(C[:, k])
            # FP64 sums of a few thousand terms in another order
            assert np.abs(rho[:, k] - r).max() <= 1e-12 * max(1.0, np.abs(r).max())
            one = gpu.jacobian_transpose_transformation(C[:, k])
            assert np.abs(sig[:, k] - one).max() <= 1e-12 * max(1.0, np.abs(one).max())
        dots = C.T @ rho
        assert np.abs(dots - sig.T @ C).max() <= 1e-11 * max(1.0, np.abs(dots).max())
