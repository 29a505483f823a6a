"""Ladder integrals formed block by block of a: lengths around the line where blocks start (n_v = 48) and a
short last block, against explicit batches, which are contracted one by one, and against one block."""

import numpy as np
import pytest

from et_b200.synthetic import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_o,n_v", [(2, 47), (3, 48), (1, 50), (2, 61), (2, 97)])
def test_blocks(n_o, n_v):
    from et_b200 import CCSD, FP64, MIXED
    n_J = 21
    s = make_system(n_o, n_v, n_J, seed=n_v)
    rng = np.random.default_rng(n_o)
    t = C = None
    out = {}
    for prec, batch in ((FP64, 0), (FP64, n_v), (FP64, 7), (MIXED, 0), (MIXED, 7)):
        with CCSD(n_o, n_v, n_J, precision=prec, ladder_batch=batch, mixed_min_flops=1) as g:
            g.set_system(s.L_mo, s.h_mo, s.eps)
            if t is None:
                t, C = 0.05 * rng.standard_normal(g.n_amp), rng.standard_normal((g.n_amp, 2))
            g.set_amplitudes(t)
            out[prec, batch] = (g.construct_omega(), g.jacobian_transformation(C), g.jacobian_transpose_transformation(C))
    for (prec, batch), res in out.items():
        for x, ref in zip(res, out[FP64, n_v]):
            # FP64: the same sums in another order; mixed: the bound of the other split-bf16 tests
            assert np.linalg.norm(x - ref) <= (1e-12 if prec == FP64 else 1e-4) * np.linalg.norm(ref)
