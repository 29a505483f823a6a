"""Small products in one launch: summed lengths N_J n_o, N_J n_v and n_o n_v around 64 and 1024 (one thread, a
warp, a block per element; one or more tables), against the oracle."""

import os
import subprocess
import sys

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


SIZES = [(1, 2, 64), (2, 3, 32), (1, 5, 65), (3, 4, 341), (4, 4, 256), (5, 5, 205), (2, 7, 600)]


@pytest.mark.parametrize("n_o,n_v,n_J", SIZES)
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


def test_lengths_reach_every_form():
    """The sizes above make products of one thread, one warp and one block per element, at lengths on both sides of
    64 and 1024."""
    code = f"import sys; sys.path.insert(0, 'tests'); import test_gpu_small_products as t; " \
           f"[t.test_lengths(*n) for n in t.SIZES]"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, CCSD_GPU_TRACE="2"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    products = []
    for line in r.stderr.splitlines():
        if " fp64 small " in line:
            w = line.split()
            products.append(tuple(int(w[w.index(x, w.index("small")) + 1]) for x in "mnk"))
    lengths = {k for _, _, k in products}
    assert {64, 65, 1024, 1025} <= lengths
    assert any(k >= 1024 and m * n <= 1024 for m, n, k in products)
