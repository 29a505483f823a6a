"""Digit GEMM on CTA pairs at the edges of its 256-row tiles, N tiles of 32..256 columns, K blocks and exact
int32 chunks, for every digit count, against FP64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from et_b200 import CCSD
    with CCSD(2, 3, 4) as c:
        yield c


@pytest.mark.parametrize("digits", [4, 5, 6, 7])
@pytest.mark.parametrize("m,n,k", [(128, 40, 70), (129, 1, 64), (256, 33, 65), (257, 255, 130), (300, 257, 1000),
                                   (520, 300, 200), (150, 96, 16384 + 72)])
def test_pair_tiles(ctx, m, n, k, digits):
    rng = np.random.default_rng(m + n + k)
    # rows and columns of very different scale, one of each all zero
    A = rng.standard_normal((m, k)) * np.exp2(rng.integers(-20, 20, (m, 1)))
    B = rng.standard_normal((k, n)) * np.exp2(rng.integers(-20, 20, (1, n)))
    A[m // 2] = 0.0
    B[:, n // 2] = 0.0
    C0 = rng.standard_normal((m, n))
    ref = 0.7 * (A @ B) - 0.3 * C0
    out = ctx.selftest_gemm(A, B, C0, alpha=0.7, beta=-0.3, mixed=digits)
    # each operand is cut 2^-7 digits below the largest element of its row or column; the dropped digit
    # products add as much again for every diagonal
    bound = 0.7 * (digits + 3) * 2.0 ** (-7 * digits) * k * np.abs(A).max(1, keepdims=True) * np.abs(B).max(0, keepdims=True)
    assert np.all(np.abs(out - ref) <= bound + 1e-14 * (np.abs(ref) + np.abs(A) @ np.abs(B)))
