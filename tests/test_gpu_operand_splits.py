"""FP64 operands split into bf16 planes from either unit stride: runs that are no multiple of the vector width or
of a tile, one row, one K position, and padding next to real values."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from et_b200 import CCSD
    with CCSD(2, 3, 4) as c:
        yield c


@pytest.mark.parametrize("transA,transB", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 2), (33, 31, 63), (34, 32, 65), (129, 66, 130), (64, 40, 4099)])
def test_layouts(ctx, m, n, k, transA, transB):
    rng = np.random.default_rng(m + n + k)
    A, B = rng.standard_normal((k, m) if transA else (m, k)), rng.standard_normal((n, k) if transB else (k, n))
    out = ctx.selftest_gemm(A, B, transA=transA, transB=transB, mixed=True)
    ref = (A.T if transA else A) @ (B.T if transB else B)
    # 16 significant bits per operand (the bound of the other split-bf16 tests)
    assert np.abs(out - ref).max() <= 1e-4 * np.abs(A).max() * np.abs(B).max() * np.sqrt(k)


def _bf16(x):
    m, e = np.frexp(x)
    return np.ldexp(np.rint(m * 256.0), e - 8)   # eight bits, ties to even


@pytest.mark.parametrize("transA", [False, True])
def test_ties_round_once(ctx, transA):
    """Values a little above and below the tie of two bf16 neighbours go to the nearer one in either split."""
    tie = 1.0 + np.arange(64.0) * 2.0 ** -7 + 2.0 ** -8
    x = np.diag(np.concatenate([tie * (1 + 2.0 ** -40), tie * (1 - 2.0 ** -40)]))
    b = 1.0 + 2.0 ** -9   # planes 1 and 2^-9; the product of the two low planes is left out
    out = ctx.selftest_gemm(x.T if transA else x, b * np.eye(128), transA=transA, mixed=True)
    hi = _bf16(np.diag(x))
    assert np.array_equal(np.diag(out), hi * b + _bf16(np.diag(x) - hi))
