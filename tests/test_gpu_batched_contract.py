"""Products that run as strided batches of GEMMs over an output index (the trial index, or one between
the others) against the oracle: blocks of several trial vectors at sizes where the batched index is the
smallest, the largest or one of the orbital ranges, and where it has no second element."""

import os
import subprocess
import sys

import numpy as np
import pytest

from et_b200.synthetic import make_system
from oracle import ccsd as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v,n_J,n_vec", [(8, 9, 20, 2), (9, 8, 31, 5), (8, 24, 16, 1), (11, 17, 8, 3), (3, 40, 50, 4), (5, 70, 90, 2)])
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


PLANS = """
import numpy as np
from et_b200 import CCSD
from et_b200.synthetic import make_system
s = make_system(5, 70, 90, seed=2)
with CCSD(5, 70, 90) as g:
    g.set_system(s.L_mo, s.h_mo, s.eps)
    g.set_amplitudes(0.05 * np.random.default_rng(1).standard_normal(g.n_amp))
    c = np.random.default_rng(2).standard_normal((g.n_amp, 2))
    g.jacobian_transformation(c)
    g.jacobian_transpose_transformation(c)
"""


def test_plans_of_two_vectors():
    """What the products of the case n_o = 5, n_v = 70, n_J = 90 with two vectors above run as: a batch over an
    orbital with the operands in place and exchanged, over the trial index alone and merged with an orbital, and
    with the operand that has no batch index copied."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PLANS], cwd=root, env=dict(os.environ, CCSD_GPU_TRACE="2"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    plans = set()
    for line in r.stderr.splitlines():
        if " fp64 batch " in line:
            w = line.split()
            plans.add((w[2].strip("[]"), int(w[w.index("batch") + 3]), " ".join(w[w.index("k") + 2:])))
    assert {("al,bjli->aibj", 5, ""), ("al,lckj->ckaj", 5, "swap"), ("aibk#,kj->aibj#", 2, ""),
            ("al,lckj#->ckaj#", 10, "swap"), ("ai#,kbji->ajbk#", 2, "copyB")} <= plans
