"""Tensor-core GEMM around the edges of its tiles: N tiles of every width class, on single CTAs and CTA pairs."""

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
