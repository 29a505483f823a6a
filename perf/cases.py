"""Workloads whose speed is tracked, each through the public entry points of ``et_b200.CCSD``.

A case names a closed-shell CCSD system (n_o occupied and n_v virtual orbitals, n_J Cholesky vectors),
an arithmetic (plain FP64, FP64 with the large products on the int8 digit GEMM, or mixed precision)
and one call of a coupled-cluster program on it:

* ``omega``      one residual at the current amplitudes, written to device memory;
* ``iteration``  what a ground-state solver on the host calls per iteration: set_amplitudes from a
                 host array, calculate_energy, construct_omega into a host array;
* ``jacobian`` / ``transpose``  rho = A c or sigma = b^T A for a block of trial vectors on the device,
                 after prepare_for_jacobian (a Davidson run) or without it (a single transformation);
* ``vjp``        the adjoint of the residual into amplitudes, Cholesky vectors and h (host arrays);
* ``solve``      a whole ground-state solve from the integrals on the host to the amplitudes on the
                 host, context creation included.

The integrals follow the recipe of ``et_b200/synthetic.py`` (s_J-weighted random symmetric vectors,
orbital energies in [-1.2, -0.4] and [0.1, 2.5] Eh), the amplitudes are the MP2 doubles times
(1 + 0.1 N(0,1)) with small singles: the values met along a solve.  Everything is drawn from the seed.
A system that is evaluated repeatedly has had its first residual (a solver's first iteration), so the
integrals that the library keeps per set of Cholesky vectors exist, as they do for every later
iteration; ``solve`` starts from nothing.

``exact`` restates the residual in plain torch FP64 and differentiates it with torch's autograd.
"""

from __future__ import annotations

import math

import torch

from et_b200 import CCSD, FP64, MIXED

COUPLING = 0.15


def _case(name, call, n_o, n_v, n_J, precision, **kw):
    c = {"name": name, "call": call, "n_o": n_o, "n_v": n_v, "n_J": n_J, "precision": precision,
         "digits": 0, "resident": True, "n_vec": 1, "prepared": True}
    c.update(kw)
    return c


def listed():
    return [
        # the benchmark's ground state: one mixed residual of the largest system
        _case("omega_mixed_large", "omega", 32, 320, 1200, "mixed"),
        # a Davidson run on the EOM workload: a block of trial vectors per iteration, prepared once
        _case("jacobian_block_mixed", "jacobian", 24, 240, 792, "mixed", n_vec=6),
        # the largest system of the uneven batch, driven by a host solver (eT's calls)
        _case("iteration_mixed", "iteration", 24, 192, 648, "mixed"),
        # the FP64 refresh of a mixed solve: six int8 digits per operand
        _case("omega_digits", "omega", 20, 200, 660, "fp64", digits=6),
        # left states or multipliers of the adjoint workload's system
        _case("transpose_block_mixed", "transpose", 16, 128, 432, "mixed", n_vec=4),
        # a ragged molecule-sized system of the batch in mixed precision
        _case("omega_mixed_ragged", "omega", 13, 107, 361, "mixed"),
        # plain FP64 residual, integrals kept per set of Cholesky vectors (the library's default)
        _case("omega_fp64", "omega", 16, 128, 432, "fp64"),
        # gradient contributions: the adjoint into amplitudes, Cholesky vectors and h
        _case("vjp_fp64", "vjp", 11, 93, 317, "fp64"),
        # one unprepared FP64 transformation (a property or a check of one vector)
        _case("jacobian_single_fp64", "jacobian", 12, 96, 324, "fp64", prepared=False),
        # T1-transformed integrals formed in every call, as when they do not fit in memory
        _case("omega_fp64_per_call", "omega", 9, 71, 241, "fp64", resident=False),
        # a member of the uneven batch from integrals to converged amplitudes
        _case("solve_mixed", "solve", 10, 80, 270, "mixed"),
        # H2O in cc-pVDZ (5 occupied, 19 virtual, 279 vectors): latency and launches count
        _case("iteration_water", "iteration", 5, 19, 279, "fp64"),
    ]


def draw(rng):
    call = rng.choice(["omega", "omega", "omega", "iteration", "iteration", "jacobian", "transpose", "vjp", "solve"])
    largest = {"omega": 28, "iteration": 24, "jacobian": 20, "transpose": 16, "vjp": 12, "solve": 12}[call]
    n_o = int(round(math.exp(rng.uniform(math.log(4.0), math.log(largest + 0.49)))))
    n_v = int(round(n_o * rng.uniform(4.0, 9.5)))
    n_J = int(round((n_o + n_v) * rng.uniform(2.5, 4.0)))
    precision = "fp64" if call == "vjp" else rng.choice(["mixed", "mixed", "fp64"])
    kw = {}
    if precision == "fp64" and call == "omega":
        kw["digits"] = rng.choice([0, 6])
        kw["resident"] = kw["digits"] == 6 or rng.random() < 0.5
    if call in ("jacobian", "transpose"):
        kw["n_vec"] = rng.randint(1, 5)
        kw["prepared"] = rng.random() < 0.7
    c = _case("", call, n_o, n_v, n_J, precision, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _packed_index(nov, device):
    """(M, m) of the packed doubles, M >= m, packed index M (M + 1) / 2 + m."""
    ij = torch.tril_indices(nov, nov, device=device)
    return ij[0], ij[1]


class _Inputs:
    """Integrals and amplitudes of one case: L[q, p, J] (the memory order of the library's L(J, p, q)),
    h, eps, and t = [t1 | packed t2] with ai = a + n_v i."""

    def __init__(self, case, seed, device="cuda", amplitudes=True):
        o, v, J = case["n_o"], case["n_v"], case["n_J"]
        n = o + v
        self.o, self.v, self.J, self.nov = o, v, J, o * v
        self.n_amp = self.nov + self.nov * (self.nov + 1) // 2
        g = torch.Generator(device=device)
        g.manual_seed(int(seed) * 7919 + 17)
        self.gen, self.device = g, device
        kw = {"dtype": torch.float64, "device": device}
        s = torch.exp(-8.0 * torch.arange(J, **kw) / J) * (0.5 * COUPLING / math.sqrt(n))
        X = torch.randn(n, n, J, generator=g, **kw)
        self.L = (X + X.transpose(0, 1)) * s
        del X
        e_o = torch.sort(-1.2 + 0.8 * torch.rand(o, generator=g, **kw)).values
        e_v = torch.sort(0.1 + 2.4 * torch.rand(v, generator=g, **kw)).values
        self.eps = torch.cat([e_o, e_v])
        Lk = torch.einsum("kkJ->J", self.L[:o, :o])
        Lo = self.L[:, :o].reshape(n, o * J)
        self.h = torch.diag(self.eps) - 2.0 * torch.einsum("qpJ,J->pq", self.L, Lk) + Lo @ Lo.T
        self.t = self._amplitudes() if amplitudes else None

    def _amplitudes(self):
        o, nov = self.o, self.nov
        Lai = self.L[:o, o:].reshape(nov, self.J)              # [i, a, J], row ai = a + n_v i
        d = (self.eps[None, o:] - self.eps[:o, None]).reshape(nov)
        g = Lai @ Lai.T
        g /= -(d[:, None] + d[None, :])
        M, m = _packed_index(nov, self.device)
        t = torch.empty(self.n_amp, dtype=torch.float64, device=self.device)
        t[nov:] = g[M, m]
        del g, M, m
        for lo in range(nov, self.n_amp, 1 << 24):
            part = t[lo:lo + (1 << 24)]
            part *= 1.0 + 0.1 * torch.randn(part.numel(), generator=self.gen, dtype=torch.float64, device=self.device)
        t[:nov] = 0.01 * torch.randn(nov, generator=self.gen, dtype=torch.float64, device=self.device)
        return t

    def vectors(self, k):
        """k vectors of unit norm as rows (the library's column-major columns)."""
        c = torch.randn(k, self.n_amp, generator=self.gen, dtype=torch.float64, device=self.device)
        return c / torch.linalg.vector_norm(c, dim=1, keepdim=True)

    def L_host(self):
        """L[J, p, q] in eT's memory order, in pinned host memory."""
        return _pinned(self.L).transpose(2, 1, 0)


def _pinned(x):
    y = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    y.copy_(x)
    return y.numpy()


class _State:
    pass


def _precision(case):
    return MIXED if case["precision"] == "mixed" else FP64


def prepare(case, seed):
    call = case["call"]
    x = _Inputs(case, seed, amplitudes=call != "solve")
    st = _State()
    st.case = case
    if call == "solve":
        st.system = (x.L_host(), _pinned(x.h), _pinned(x.eps))
        return st
    st.gpu = gpu = CCSD(case["n_o"], case["n_v"], case["n_J"], precision=_precision(case))
    if case["digits"]:
        gpu.set_fp64_digits(case["digits"])
    if not case["resident"]:
        gpu.set_fp64_integrals(False)
    gpu.set_system(x.L_host(), _pinned(x.h), _pinned(x.eps))
    x.L = None
    st.t = _pinned(x.t)
    gpu.set_amplitudes(st.t)
    if call == "omega":
        st.out = torch.empty(x.n_amp, dtype=torch.float64, device="cuda")
    elif call == "iteration":
        st.out = torch.empty(x.n_amp, dtype=torch.float64, pin_memory=True).numpy()
    elif call == "vjp":
        st.b = _pinned(x.vectors(1)[0])
    else:
        st.c = x.vectors(case["n_vec"])
        st.out = torch.empty_like(st.c)
        if case["prepared"]:
            gpu.prepare_for_jacobian(1 if call == "transpose" else 0)
    torch.cuda.synchronize()
    run(st)
    return st


def run(st):
    case = st.case
    call = case["call"]
    if call == "solve":
        L, h, eps = st.system
        with CCSD(case["n_o"], case["n_v"], case["n_J"], precision=_precision(case)) as gpu:
            gpu.set_system(L, h, eps)
            gpu.set_initial_amplitudes_guess()
            energy = gpu.solve_ground_state(omega_threshold=5e-7, energy_threshold=5e-9)[0]
            return {"energy": energy, "t": gpu.get_amplitudes()}
    gpu = st.gpu
    if call == "omega":
        gpu.construct_omega_device(st.out.data_ptr())
        return st.out
    if call == "iteration":
        gpu.set_amplitudes(st.t)
        energy = gpu.calculate_energy()
        return {"energy": energy, "omega": gpu.construct_omega(st.out)}
    if call == "vjp":
        dt, dL, dh = gpu.vjp(st.b, want_L=True, want_h=True)
        return {"dt": dt, "dL": dL, "dh": dh}
    gpu.jacobian_device(case["n_vec"], st.c.data_ptr(), st.out.data_ptr(), transpose=call == "transpose")
    return st.out


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------


def _residual_flops(o, v, J):
    """2mnk of the residual's contractions: the ladder in its +/- form, from integrals of the
    untransformed vectors."""
    ov = float(o * v)
    nop, nom, nvp, nvm = o * (o + 1) / 2, o * (o - 1) / 2, v * (v + 1) / 2, v * (v - 1) / 2
    f = 2 * nop * nvp * nvp + 2 * nom * nvm * nvm                       # ladder
    f += 4 * 2 * ov ** 3                                                # C and D terms
    f += 2 * J * ov * ov * 2 + 2 * J * (o * v * v * o)                  # g_aibj, g_aikc, g_ackj
    f += 2 * (o * v * v * v * o * o)                                    # t1 part of the ladder
    f += 4 * (2.0 * o ** 4 * v * v) + 2 * 2.0 * o * o * v ** 3 + 2 * 2.0 * o ** 3 * v * v
    return f


def work(case):
    o, v, J = case["n_o"], case["n_v"], case["n_J"]
    n, ov = o + v, o * v
    amp = 8.0 * (ov + ov * (ov + 1) / 2)
    L = 8.0 * J * n * n
    res, call = _residual_flops(o, v, J), case["call"]
    pairs = float(v) ** 4 * J                                           # forming the ladder integrals
    if not case["resident"]:
        res += pairs
    t1_part = 2.0 * J * o * (v * v + v * n + 2 * o * n) * 2             # T1 transformation and Fock matrix
    if call == "omega":
        return {"bytes": L + 2 * amp, "flops": res}
    if call == "iteration":
        return {"bytes": L + 2 * amp, "flops": res + t1_part}
    if call == "vjp":
        return {"bytes": 2 * L + 3 * amp, "flops": 3 * res + 3 * pairs}
    if call == "solve":
        return {"bytes": L + amp, "flops": 10 * (res + t1_part) + pairs}
    # a product of two amplitude-dependent factors has two derivative terms
    once = 0.0 if case["prepared"] else res + pairs
    return {"bytes": L + amp * (1 + 2 * case["n_vec"]), "flops": case["n_vec"] * 2 * res + once}


def tolerance(case):
    # About four times the relative error seen against the FP64 reference: DGEMM sums in another order
    # (up to 1e-15), six-digit products of the int8 digit GEMM (5e-12), split-bf16 products (16 significant
    # bits per operand, FP32 accumulation; 1.4e-6 at the largest size), and the thresholds of a converged
    # solve (5e-7).
    if case["call"] == "solve":
        return {"rel": 2e-6, "max": 1e-3}
    if case["precision"] == "mixed":
        return {"rel": 6e-6, "max": 1e-3}
    if case["digits"]:
        return {"rel": 4e-11, "max": 4e-9}
    return {"rel": 1e-14, "max": 1e-12}


# ---------------------------------------------------------------------------
# the residual in plain torch FP64
# ---------------------------------------------------------------------------


def _square(t2, o, v):
    """packed doubles -> t[i, a, j, b] (row ai = a + n_v i)."""
    nov = o * v
    M, m = _packed_index(nov, t2.device)
    low = torch.zeros(nov, nov, dtype=t2.dtype, device=t2.device).index_put((M, m), t2)
    return (low + low.T - torch.diag(torch.diagonal(low))).reshape(o, v, o, v)


def _pack_half(x, o, v):
    """packed lower triangle with the diagonal halved."""
    x = x.reshape(o * v, o * v)
    x = x - 0.5 * torch.diag(torch.diagonal(x))
    M, m = _packed_index(o * v, x.device)
    return x[M, m]


def _t1_blocks(L, h, t1, o):
    """T1-transformed Cholesky vectors [q, p, J] and Fock matrix, X M Y^T with X = 1 - t1, Y = 1 + t1^T."""
    n = L.shape[0]
    v = n - o
    kw = {"dtype": L.dtype, "device": L.device}
    low = torch.cat([torch.zeros(o, n, **kw), torch.cat([t1.T, torch.zeros(v, v, **kw)], 1)], 0)
    X, Y = torch.eye(n, **kw) - low, torch.eye(n, **kw) + low.T
    Lt = torch.einsum("pr,srJ->spJ", X, L)
    Lt = torch.einsum("spJ,qs->qpJ", Lt, Y)
    F = X @ h @ Y.T
    tr = torch.einsum("kkJ->J", Lt[:o, :o])
    F = F + 2.0 * torch.einsum("qpJ,J->pq", Lt, tr) - torch.einsum("kpJ,qkJ->pq", Lt[:o], Lt[:, :o])
    return Lt, F


def _energy(t1, t2, L, o):
    v = L.shape[0] - o
    Lov = L[o:, :o]                                                        # [a, i, J]
    g = torch.einsum("aiJ,bjJ->iajb", Lov, Lov)
    T = _square(t2, o, v) + torch.einsum("ia,jb->iajb", t1, t1)
    return (T * (2.0 * g - g.permute(0, 3, 2, 1))).sum()


def _omega(t1, t2, L, h, o):
    """[Omega_1 | packed Omega_2] of closed-shell CCSD with T1-transformed integrals; t1[i, a]."""
    v = L.shape[0] - o
    Lt, F = _t1_blocks(L, h, t1, o)
    # blocks as [p, q, J]
    oo, ov = Lt[:o, :o].transpose(0, 1), Lt[o:, :o].transpose(0, 1)
    vo, vv = Lt[:o, o:].transpose(0, 1), Lt[o:, o:].transpose(0, 1)
    Foo, Fov, Fvo, Fvv = F[:o, :o], F[:o, o:], F[o:, :o], F[o:, o:]
    t = _square(t2, o, v)                                                   # [i, a, j, b]
    u = 2.0 * t - t.permute(2, 1, 0, 3)
    L_vo = L[:o, o:].transpose(0, 1)                                        # untransformed [a, i, J]
    om1 = Fvo + torch.einsum("abJ,biJ->ai", vv, torch.einsum("cjJ,jcib->biJ", L_vo, u))
    om1 = om1 - torch.einsum("jakb,kbji->ai", u, torch.einsum("kbJ,jiJ->kbji", ov, oo))
    om1 = om1 + torch.einsum("iajb,jb->ai", u, Fov)
    g = torch.einsum("iaJ,jbJ->iajb", ov, ov)
    Xbc = Fvv - torch.einsum("kbld,ldkc->bc", u, g)
    Ykj = Foo + torch.einsum("kdlc,jdlc->kj", g, u)
    om = torch.einsum("bc,jcia->jbia", Xbc, t) - torch.einsum("iakb,kj->iajb", t, Ykj)
    om = om + 0.5 * torch.einsum("aiJ,bjJ->iajb", vo, vo)
    W = torch.einsum("kiJ,ljJ->klij", oo, oo) + torch.einsum("kcld,icjd->klij", g, t)
    om = om + 0.5 * torch.einsum("kalb,klij->iajb", t, W)
    g_kjac = torch.einsum("acJ,kjJ->kcja", vv, oo)
    C = g_kjac - 0.5 * torch.einsum("kcld,jdka->lcja", g, t)                # [k, c, j, a]
    D = 2.0 * torch.einsum("aiJ,kcJ->kcia", vo, ov) - g_kjac
    D = D + torch.einsum("lckd,kdja->lcja", g - 0.5 * g.permute(2, 1, 0, 3), u)
    x = -1.5 * torch.einsum("kaic,kcjb->iajb", t, C)
    om = om + 0.5 * torch.einsum("iakc,kcjb->iajb", u, D) + x / 3.0 + (2.0 / 3.0) * x.permute(2, 1, 0, 3)
    om2 = _pack_half(om + om.permute(2, 3, 0, 1), o, v)
    # ladder sum_cd g_acbd t_cidj in blocks of a
    tcd = t.permute(1, 3, 0, 2).reshape(v * v, o * o)                       # [c, d, i, j]
    step = max(1, int(1.0e9 // (8.0 * v * v * v)))
    rows = []
    for a0 in range(0, v, step):
        G = torch.einsum("acJ,bdJ->abcd", vv[a0:a0 + step], vv)
        rows.append((G.reshape(-1, v * v) @ tcd).reshape(-1, v, o, o))
    lad = torch.cat(rows, 0).permute(2, 0, 3, 1)                            # [i, a, j, b]
    return torch.cat([om1.T.reshape(-1), om2 + _pack_half(lad, o, v)])


def _solve(x):
    """Amplitudes at |Omega| < 1e-11 by quasi-Newton steps with DIIS."""
    o, v, nov = x.o, x.v, x.nov
    d1 = (x.eps[None, o:] - x.eps[:o, None]).reshape(nov)
    M, m = _packed_index(nov, x.device)
    d2 = d1[M] + d1[m]
    t = torch.zeros(x.n_amp, dtype=torch.float64, device=x.device)
    Lai = x.L[:o, o:].reshape(nov, x.J)
    t[nov:] = -(Lai @ Lai.T)[M, m] / d2
    den = torch.cat([d1, torch.where(M == m, 0.5 * d2, d2)])               # the residual's diagonal is halved
    errs, pars = [], []
    for _ in range(80):
        om = _omega(t[:nov].reshape(o, v), t[nov:], x.L, x.h, o)
        if torch.linalg.vector_norm(om) < 1e-11:
            break
        r = -om / den
        errs, pars = (errs + [r])[-8:], (pars + [t + r])[-8:]
        E, k = torch.stack(errs), len(errs)
        A = -torch.ones(k + 1, k + 1, dtype=torch.float64, device=x.device)
        A[:k, :k] = E @ E.T / (r @ r)
        A[k, k] = 0.0
        rhs = torch.zeros(k + 1, dtype=torch.float64, device=x.device)
        rhs[k] = -1.0
        t = torch.linalg.solve(A, rhs)[:k] @ torch.stack(pars)
    return t


def exact(case, seed):
    o, v, call = case["n_o"], case["n_v"], case["call"]
    if call in ("vjp", "transpose") and v > 160:
        return None                                                         # reverse mode keeps v^4 doubles
    device = "cuda" if torch.cuda.is_available() else "cpu"
    x = _Inputs(case, seed, device=device, amplitudes=call != "solve")
    nov = x.nov
    t = _solve(x) if call == "solve" else x.t
    t1, t2 = t[:nov].reshape(o, v), t[nov:]
    if call == "solve":
        return {"energy": float(_energy(t1, t2, x.L, o)), "t": t}
    if call == "omega":
        return _omega(t1, t2, x.L, x.h, o)
    if call == "iteration":
        return {"energy": float(_energy(t1, t2, x.L, o)), "omega": _omega(t1, t2, x.L, x.h, o)}
    if call == "vjp":
        b = x.vectors(1)[0]
        ins = [y.detach().clone().requires_grad_(True) for y in (t1, t2, x.L, x.h)]
        d1, d2, dL, dh = torch.autograd.grad(_omega(*ins, o), ins, b)
        return {"dt": torch.cat([d1.reshape(-1), d2]), "dL": dL.permute(2, 1, 0).contiguous(), "dh": dh}
    vec = x.vectors(case["n_vec"])
    M = torch.arange(nov, device=device)
    diag = nov + M * (M + 1) // 2 + M                                       # ai == bj
    out = torch.empty_like(vec)
    for k in range(case["n_vec"]):
        c = vec[k].clone()
        if call == "jacobian":
            c[diag] *= 2.0
            out[k] = torch.func.jvp(lambda p, q: _omega(p, q, x.L, x.h, o), (t1, t2),
                                    (c[:nov].reshape(o, v), c[nov:]))[1]
        else:
            ins = [y.detach().clone().requires_grad_(True) for y in (t1, t2)]
            d1, d2 = torch.autograd.grad(_omega(*ins, x.L, x.h, o), ins, c)
            out[k] = torch.cat([d1.reshape(-1), d2])
            out[k, diag] *= 2.0
    return out
