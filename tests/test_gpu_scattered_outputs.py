"""Tensor-core products whose outputs lie in tensors of interleaved indices, on single CTAs and, in a process of its
own (the choice is read once), on CTA pairs."""

import os
import subprocess
import sys

import numpy as np
import pytest

from et_b200.synthetic import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v,n_J,n_vec", [(2, 33, 20, 3), (5, 19, 33, 1), (7, 40, 65, 2)])
def test_scattered_outputs(n_o, n_v, n_J, n_vec):
    """Every product on the tensor cores (mixed_min_flops = 1): transformations and residual against FP64."""
    from et_b200 import CCSD, FP64, MIXED
    s = make_system(n_o, n_v, n_J, seed=2)
    out = {}
    for prec in (FP64, MIXED):
        with CCSD(n_o, n_v, n_J, precision=prec, mixed_min_flops=1) as g:
            g.set_system(s.L_mo, s.h_mo, s.eps)
            rng = np.random.default_rng(3)
            g.set_amplitudes(0.05 * rng.standard_normal(g.n_amp))
            C = rng.standard_normal((g.n_amp, n_vec))
            out[prec] = (g.construct_omega(), g.jacobian_transformation(C), g.jacobian_transpose_transformation(C))
    for ref, mix in zip(out[FP64], out[MIXED]):
        assert np.linalg.norm(mix - ref) <= 1e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("n_o,n_v,n_J,n_vec", [(7, 40, 65, 2), (9, 37, 130, 3)])
def test_scattered_outputs_on_pairs(n_o, n_v, n_J, n_vec):
    """The same comparison with every product of at least 256 rows on CTA pairs: n_o n_v (or n_J n_v) rows."""
    code = f"import sys; sys.path.insert(0, 'tests'); import test_gpu_scattered_outputs as t; " \
           f"t.test_scattered_outputs({n_o}, {n_v}, {n_J}, {n_vec})"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, CCSD_GPU_PAIR_GEMM="1"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
