"""Tensor-core GEMM around the edges of its tiles: N tiles of every width class, on single CTAs and, in a process
of its own (the choice is read once), on CTA pairs."""

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from et_b200 import CCSD
    with CCSD(2, 3, 4) as c:
        yield c


@pytest.mark.parametrize("m,k", [(1, 64), (129, 130), (700, 4200)])
@pytest.mark.parametrize("n", [1, 16, 17, 33, 96, 169, 176, 255, 257, 300, 528])
def test_n_tile_widths(ctx, m, n, k):
    rng = np.random.default_rng(m + 7 * n)
    A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    out = ctx.selftest_gemm(A, B, C0, alpha=0.7, beta=-0.3, mixed=True)
    ref = 0.7 * (A @ B) - 0.3 * C0
    # 16 significant bits per operand (the bound of the other split-bf16 tests)
    assert np.abs(out - ref).max() <= 1e-4 * np.abs(A).max() * np.abs(B).max() * np.sqrt(k)


PAIRS = """
import numpy as np
from et_b200 import CCSD
with CCSD(2, 3, 4) as c:
    # partial and whole tiles of 256 rows; one K block, several, and K splits
    for m, k in ((257, 64), (300, 1000), (512, 130), (700, 4200)):
        for n in (1, 16, 17, 33, 96, 169, 176, 255, 257, 300, 528):
            rng = np.random.default_rng(m + 7 * n)
            A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
            out = c.selftest_gemm(A, B, C0, alpha=0.7, beta=-0.3, mixed=True)
            ref = 0.7 * (A @ B) - 0.3 * C0
            err = np.abs(out - ref).max()
            assert err <= 1e-4 * np.abs(A).max() * np.abs(B).max() * np.sqrt(k), (m, n, k, err)
"""


def test_n_tile_widths_on_pairs():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PAIRS], cwd=root, env=dict(os.environ, CCSD_GPU_PAIR_GEMM="1"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
