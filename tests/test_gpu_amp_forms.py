"""Packed doubles <-> full arrays around the 32 x 32 tiles of (a, b): every element of the residual and
of both transformations of a block of vectors against the oracle."""

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v", [(1, 1), (2, 31), (2, 32), (1, 33), (3, 34), (1, 65)])
def test_tile_edges(n_o, n_v):
    from et_b200 import CCSD
    n_J = 17
    s = make_system(n_o, n_v, n_J, seed=n_v)
    ref = oc.CCSDSystem(s.L_mo, s.h_mo, s.eps, s.n_o)
    rng = np.random.default_rng(n_o)
    ref.set_amplitudes(0.05 * rng.standard_normal(ref.n_amp))
    C = rng.standard_normal((ref.n_amp, 2))
    with CCSD(n_o, n_v, n_J) as gpu:
        gpu.set_system(s.L_mo, s.h_mo, s.eps)
        gpu.set_amplitudes(ref.get_amplitudes())
        om, om_ref = gpu.construct_omega(), ref.omega()
        # FP64 sums in another order: a few hundred terms of the size of the largest output
        assert np.abs(om - om_ref).max() <= 1e-13 * max(1.0, np.abs(om_ref).max())
        rho = gpu.jacobian_transformation(C)
        for k in range(2):
            r = ref.jacobian_transformation(C[:, k])
            assert np.abs(rho[:, k] - r).max() <= 1e-12 * max(1.0, np.abs(r).max())
        sig = gpu.jacobian_transpose_transformation(C)
        # <b_j, A c_k> = <A^T b_j, c_k>
        assert np.abs(C.T @ rho - sig.T @ C).max() <= 1e-11 * max(1.0, np.abs(C.T @ rho).max())
