"""Arithmetic of Q_kilj = sum_cd g_kcld t_cidj and of the t part of X_klij, on systems whose other products are
exact: every Cholesky block but L_ov is zero and the integrals and amplitudes are small integers."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n_o, n_v, n_J, seed):
    """L, h, eps, t with L = 0, h = 0 and integer amplitudes; the caller fills L[:, :n_o, n_o:]."""
    rng = np.random.default_rng(seed)
    nov = n_o * n_v
    t = np.zeros(nov + nov * (nov + 1) // 2)
    t[nov:] = rng.integers(-1, 2, t.size - nov)
    n = n_o + n_v
    return rng, np.zeros((n_J, n, n)), np.zeros((n, n)), np.linspace(-1.0, 1.0, n), t


def _omega(system, t, n_o, n_v, n_J, digits=0, min_flops=0.0, **kw):
    from et_b200 import CCSD
    with CCSD(n_o, n_v, n_J, **kw) as g:
        if digits:
            g.set_fp64_digits(digits, min_flops)
        g.set_system(*system)
        g.set_amplitudes(t)
        return g.construct_omega()


@pytest.mark.parametrize("n_o,n_v", [(4, 20), (5, 33)])
def test_integrals_split_from_fp64(n_o, n_v):
    """Mixed precision holds g_kcld as bf16 planes of the FP64 integrals.  Here g_kcld is an integer to rounding
    while the two vectors that form it (cos and sin of one direction) need all their bits."""
    from et_b200 import FP64, MIXED
    rng, L, h, eps, t = _system(n_o, n_v, 2, n_v)
    a = rng.integers(-1, 2, (n_o, n_v))
    L[0, :n_o, n_o:], L[1, :n_o, n_o:] = np.cos(0.7) * a, np.sin(0.7) * a
    ref = _omega((L, h, eps), t, n_o, n_v, 2, precision=FP64)
    out = _omega((L, h, eps), t, n_o, n_v, 2, precision=MIXED, mixed_min_flops=1)
    # integers below 2^16 are exact in two planes, their sums below 2^24 exact in FP32
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("n_o,n_v", [(2, 9), (8, 64)])
def test_small_products_stay_fp64(n_o, n_v):
    """Products below mixed_min_flops stay FP64, Q and X_klij among them."""
    from et_b200 import FP64, MIXED
    rng, L, h, eps, t = _system(n_o, n_v, 7, n_v)
    L[:, :n_o, n_o:] = rng.standard_normal((7, n_o, n_v))
    t = rng.standard_normal(t.size)
    t[:n_o * n_v] *= 0.1
    ref = _omega((L, h, eps), t, n_o, n_v, 7, precision=FP64)
    out = _omega((L, h, eps), t, n_o, n_v, 7, precision=MIXED, mixed_min_flops=10 ** 15)
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)


def test_small_products_stay_on_dgemm():
    """Products below the line of set_fp64_digits stay on DGEMM, Q and X_klij among them.  A virtual pair of two
    odd orbitals has integrals of 2^-40, one of two even orbitals integrals of 1, and only the former meet
    amplitudes: in the rows of every other product a row's integrals have one size, in those of Q (k, l) both
    occur and four digits keep the larger only."""
    n_o, n_v = 16, 48
    rng, L, h, eps, t = _system(n_o, n_v, 2, 5)
    odd = np.arange(n_v) % 2 == 1
    a = rng.integers(0, 2, (n_o, n_v)) * 2.0 - 1.0
    L[0, :n_o, n_o:], L[1, :n_o, n_o:] = np.where(odd, 0.0, a), np.where(odd, 2.0 ** -20 * a, 0.0)
    M, m = np.tril_indices(n_o * n_v)
    t[n_o * n_v:] *= odd[M % n_v] & odd[m % n_v]
    # the line lies between Q (3.0e8 flops) and the products over n_o n_v (9.1e8)
    out = _omega((L, h, eps), t, n_o, n_v, 2, digits=4, min_flops=5e8)
    ref = _omega((L, h, eps), t, n_o, n_v, 2)
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)
