"""Workloads of the variational hot path, each through the calls a program makes.

A program that optimises a basis of explicitly correlated Gaussians keeps one
Context per basis and calls, in this order of frequency: the energy of a trial
function beside a fixed basis, the energy and gradient of the whole basis or of
its newest function, batches of either, and, at the end, expectation values.
Every case below is one such call on a seeded random basis (the distributions
of ecg_b200.synth) of the systems in synth.SYSTEMS:

  trial         EnergyIA(K, K): one trial function beside K - 1 fixed ones
                (the BasisEnlI trial loop); bordered factorisation step
  energy        EnergyIA(1, K): the energy of the whole basis
  gradient      EnergyIB(0, K), fused adjoint gradient: one optimiser step
  plain         EnergyIB(0, K), the drop-in form that fills Glob_D
  function      EnergyIB(K - 1, K): energy and gradient of the newest function
  candidates    a batch of trial functions beside one fixed basis
  candgrad      the same with each trial function's gradient
  general       EnergyGB(0, K) of a 'G' context: no shift known, the which-th
                eigenvalue by inertia bisection, and its gradient
  expectation   the expectation-value pass over a converged eigenvector

An iterative call starts from the eigenvector and the energy of a nearby
basis, as inside an optimisation: prepare() solves the seeded basis, and run()
evaluates it with every parameter moved by 1e-6 (relative), from the solved
basis's eigenvector with the shift lambda~ = 1.000001 E.  run() restores that
start vector each time, as a line search that returns to its accepted point.
How many iterations a call took is not among the outputs: it is how the answer
was found, not the answer.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "atom-mol-nonbo_b200"))

from ecg_b200 import Context, synth  # noqa: E402

INVIT_PARAMETER = 1.000001  # lambda~ / E of the example inputs
STEP = 1e-6                 # relative size of the parameter step
# EIGVAL_TOLERANCE, a factor of ten above the residual that rounding leaves at
# the largest basis here, so that the error code does not hang on it; looser
# for the batched trials, whose energies are only ranked
TOL, TOL_BATCH, MAX_ITER = 1e-11, 1e-10, 20


def listed():
    return [
        # the first functions of a three-particle basis: launches and latency
        dict(name="trial_n2_k201", kind="trial", system="h_minus_like", K=201),
        # a trial beside a grown four-particle basis
        dict(name="trial_n3_k2001", kind="trial", system="h2_like", K=2001),
        # a whole three-particle basis
        dict(name="energy_n2_k500", kind="energy", system="h_minus_like", K=500),
        # optimiser steps on four particles: ordinary and large
        dict(name="gradient_n3_k1500", kind="gradient", system="h2_like", K=1500),
        dict(name="gradient_n3_k4000", kind="gradient", system="h2_like", K=4000),
        # five particles, fourteen projector terms, a ragged size
        dict(name="gradient_n4_k1013", kind="gradient", system="li_minus_like", K=1013),
        # the largest basis: three electrons, six projector terms
        dict(name="gradient_li_k10000", kind="gradient", system="li_like", K=10000),
        # the drop-in form with the derivative array
        dict(name="plain_n3_k1000", kind="plain", system="h2_like", K=1000),
        # basis enlargement in batches: ranking, then optimisation of the best
        dict(name="candidates_n3_k2000", kind="candidates", system="h2_like", K=2000, count=256),
        dict(name="candgrad_n3_k1500", kind="candgrad", system="h2_like", K=1500, count=100),
        # the generalised-eigenproblem context, where bases are small
        dict(name="general_n2_k240", kind="general", system="h_minus_like", K=240),
        # after the optimisation
        dict(name="expectation_n3_k1000", kind="expectation", system="h2_like", K=1000),
    ]


def draw(rng):
    kind = rng.choice(["trial", "energy", "gradient", "gradient", "plain", "function", "candidates", "candgrad",
                       "general", "expectation"])
    most = dict(trial=4000, energy=4000, gradient=4000, plain=1200, function=4000, candidates=2500, candgrad=2500,
                general=1200, expectation=1500)[kind]
    name = rng.choice(["h_minus_like", "h2_like", "li_like", "li_minus_like"])
    if name == "h_minus_like":
        # functions of two coordinates soon become linearly dependent; an
        # energy stands that for longer than an eigenvector
        most = 600 if kind in ("trial", "energy") else 250
    elif name == "li_minus_like":
        most = min(most, 600) if kind == "plain" else most
        most = min(most, 1500)
    case = dict(kind=kind, system=name, K=round(math.exp(rng.uniform(math.log(100), math.log(most)))))
    if kind in ("candidates", "candgrad"):
        case["count"] = round(math.exp(rng.uniform(math.log(8), math.log(256))))
    return case


def _random_basis(case, seed):
    sysm = synth.make_system(case["system"])
    # the lithium-like systems scale each coordinate by its reduced mass
    scale = synth.reduced_mass_scale(sysm.masses) if case["system"].startswith("li") else None
    return sysm, synth.random_basis(sysm.n, case["K"], seed, row_scale=scale)


def _inputs(case, seed):
    """(system, basis before the step, basis or trial functions after it)."""
    sysm, p0 = _random_basis(case, seed)
    rng = np.random.default_rng([seed, 1])
    kind = case["kind"]
    if kind in ("candidates", "candgrad"):
        p1 = synth.candidates(p0, case["count"], seed)
    elif kind == "trial":
        p1 = p0[-1:].copy()
        p0 = p0[:-1]
    elif kind == "function":
        p1 = p0[-1:] * (1.0 + STEP * rng.uniform(-1.0, 1.0, p0[-1:].shape))
    elif kind == "expectation":
        p1 = p0
    else:
        p1 = p0 * (1.0 + STEP * rng.uniform(-1.0, 1.0, p0.shape))
    return sysm, p0, np.ascontiguousarray(p1)


def prepare(case, seed):
    sysm, p0, p1 = _inputs(case, seed)
    kind, K = case["kind"], case["K"]
    nbase = len(p0)
    room = K + 1 if kind in ("candidates", "candgrad") else K
    method = "G" if kind in ("general", "expectation") else "I"
    ctx = Context(sysm, room, max_nfo=K if kind == "plain" else 0, method=method)
    ctx.set_params(p0)
    s = dict(kind=kind, K=K, ctx=ctx, p=p1)
    if method == "G":
        s["E"], err, _ = ctx.energy_ga(1, nbase, want_vector=True)
        assert err == 0, f"eigenproblem of the seeded basis: {err}"
        return s
    # the lowest state, from below, then the solved basis at its working shift
    floor = synth.SYSTEMS[case["system"]]["e_floor"]
    ctx.set_vectors(nbase, last_eigvec=np.ones(nbase, dtype=np.complex128))
    E, _, _ = ctx.energy_ia(1, nbase, floor, -1e-12, max_iter=300, specif_norm=0)
    E, _, _ = ctx.energy_ia(1, nbase, E * INVIT_PARAMETER, -1e-12, max_iter=50, specif_norm=0)
    s["lam"] = E * INVIT_PARAMETER
    ctx.energy_ia(1, nbase, s["lam"], TOL, max_iter=50, specif_norm=0)
    s["x0"] = np.zeros(room, dtype=np.complex128)
    s["x0"][:nbase] = ctx.vectors(nbase)[1]
    return s


def run(s):
    ctx, K, kind, p = s["ctx"], s["K"], s["kind"], s["p"]
    if kind == "expectation":
        return ctx.expectation_values(K, s["E"])
    if kind == "general":
        ctx.set_params(p)
        E, g, err = ctx.energy_gb_adjoint(0, K)
        return dict(E=E, gradient=g, err=int(err))
    ctx.set_vectors(len(s["x0"]), last_eigvec=s["x0"])
    if kind == "candidates":
        E, err, _, _ = ctx.eval_candidates(K, p, s["lam"], TOL_BATCH, MAX_ITER)
        return dict(E=E, err=err)
    if kind == "candgrad":
        E, err, _, _, g = ctx.eval_candidates_grad(K, p, s["lam"], TOL_BATCH, MAX_ITER)
        return dict(E=E, err=err, gradient=g)
    ctx.set_params(p, first=K - len(p) + 1)
    if kind == "trial":
        E, err, _ = ctx.energy_ia(K, K, s["lam"], TOL, MAX_ITER)
        return dict(E=E, err=int(err))
    if kind == "energy":
        E, err, _ = ctx.energy_ia(1, K, s["lam"], TOL, MAX_ITER)
        return dict(E=E, err=int(err))
    fn = ctx.energy_ib if kind == "plain" else ctx.energy_ib_adjoint
    E, g, err, _ = fn(K - len(p), K, s["lam"], TOL, MAX_ITER)
    return dict(E=E, gradient=g, err=int(err))


def _pair_flops(n, gradient):
    """Operations of one projector term of one pair: real multiplications and
    additions of the n x n complex algebra, roots and divisions as one each."""
    tri = n * (n + 1) // 2
    factor = 8 * (n ** 3 - n) // 6 + 6 * n * n // 2 + 8 * tri  # L D L^T of C, its inverse
    inverse = 8 * n * (n + 1) * (n + 2) // 6
    energy = factor + inverse + 8 * n ** 3 + 8 * n * n + tri * 24 + 40
    if not gradient:
        return energy
    return energy + tri * 20 + 2 * (8 * tri + 8 * n ** 3 + 16 * tri)


def work(case):
    sysm = synth.make_system(case["system"])
    n, T, K, kind = sysm.n, sysm.T, case["K"], case["kind"]
    pairs = K * (K + 1) / 2
    ld = 4.0 * K ** 3 / 3.0
    step = 16.0 * K * K  # S v and the two triangular solves, 8 flops an entry
    npt = sysm.npt
    data = 8.0 * npt * K + 16.0 * K
    if kind == "trial":
        # the row, and S and the factor read once
        return dict(bytes=data + 16.0 * K * K, flops=T * K * _pair_flops(n, False) + 3 * step)
    if kind == "function":
        return dict(bytes=data + 16.0 * K * K, flops=T * K * _pair_flops(n, True) + 3 * step)
    if kind in ("candidates", "candgrad"):
        B = case["count"]
        fl = B * (T * K * _pair_flops(n, kind == "candgrad") + 8.0 * K * K + 3 * step + 16.0 * K * K)
        return dict(bytes=data + 8.0 * npt * B + 24.0 * K * K, flops=fl)
    if kind == "expectation":
        return dict(bytes=data, flops=pairs * T * 9000.0 * (n / 3.0) ** 3)
    fl = pairs * T * _pair_flops(n, kind != "energy")
    if kind == "general":
        # isolating the eigenvalue takes a factorisation at each end and one to iterate with
        return dict(bytes=data + 8.0 * npt * K, flops=fl + 3 * ld)
    return dict(bytes=data + 8.0 * npt * K, flops=fl + ld + 3 * step)


# --- the same quantities in plain torch, 64 bits ---------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _sym(p, n, off):
    out, x = [[None] * n for _ in range(n)], off
    for i in range(n):
        for j in range(i, n):
            out[i][j] = out[j][i] = p[..., x]
            x += 1
    return out


def _gram(p, n):
    L, x = [[None] * n for _ in range(n)], 0
    for i in range(n):
        for j in range(i, n):
            L[j][i] = p[..., x]
            x += 1
    A = [[None] * n for _ in range(n)]
    for i in range(n):
        for j in range(i, n):
            A[i][j] = A[j][i] = sum(L[i][k] * L[j][k] for k in range(i + 1))
    det = 1.0
    for i in range(n):
        det = det * L[i][i]
    return A, det


def _term(sysm, pb, pk, t):
    """(T, V, S) of one projector term, bra functions pb and ket functions pk, broadcast."""
    n, np_ = sysm.n, sysm.np
    P, M, q = sysm.yhy_mats[t], sysm.mass_matrix, sysm.charges
    Ab, db = _gram(pb, n)
    Bb = _sym(pb, n, np_)
    Ak, dk = _gram(pk, n)
    Bk = _sym(pk, n, np_)

    def permuted(X):
        Y = [[None] * n for _ in range(n)]
        for i in range(n):
            for j in range(i, n):
                Y[i][j] = Y[j][i] = sum(float(P[a, i] * P[b, j]) * X[a][b] for a in range(n) for b in range(n)
                                        if P[a, i] * P[b, j] != 0)
        return Y

    Ap, Bp = permuted(Ak), permuted(Bk)
    Cb = [[torch.complex(Ab[i][j], -Bb[i][j]) for j in range(n)] for i in range(n)]
    Ck = [[torch.complex(Ap[i][j], Bp[i][j]) for j in range(n)] for i in range(n)]
    W = [[Cb[i][j] + Ck[i][j] for j in range(n)] for i in range(n)]
    L = [[None] * n for _ in range(n)]
    d = [None] * n
    for i in range(n):
        d[i] = W[i][i]
        for j in range(i + 1, n):
            L[j][i] = W[j][i] / d[i]
        for j in range(i + 1, n):
            for k in range(i + 1, j + 1):
                W[j][k] = W[k][j] = W[j][k] - L[j][i] * W[k][i]
    X = [[None] * n for _ in range(n)]  # the inverse of the unit lower factor
    for i in range(n):
        for j in range(i + 1, n):
            X[j][i] = -L[j][i] - sum(L[j][k] * X[k][i] for k in range(i + 1, j))
    inv = [[None] * n for _ in range(n)]
    for i in range(n):
        for j in range(i, n):
            s = (X[j][i] if j > i else 1.0) / d[j]
            for k in range(j + 1, n):
                s = s + X[k][i] * X[k][j] / d[k]
            inv[i][j] = inv[j][i] = s
    det = d[0]
    for i in range(1, n):
        det = det * d[i]
    c = (db * dk).abs() / det
    S = 2.0 ** (1.5 * n) * (c * torch.sqrt(c))
    tr = 0.0
    for i in range(n):
        for j in range(n):
            kin = sum(Ck[j][a] * inv[a][b] * Cb[b][i] for a in range(n) for b in range(n))
            tr = tr + float(M[i, j]) * kin
    V = 0.0
    for i in range(n):
        V = V + float(q[0] * q[i + 1]) / torch.sqrt(inv[i][i])
        for j in range(i + 1, n):
            V = V + float(q[i + 1] * q[j + 1]) / torch.sqrt(inv[i][i] + inv[j][j] - 2.0 * inv[i][j])
    return 6.0 * S * tr, 2.0 / math.sqrt(math.pi) * S * V, S


def _sums(sysm, pb, pk):
    T = V = S = 0.0
    for t in range(sysm.T):
        a, b, s = _term(sysm, pb, pk, t)
        c = float(sysm.yhy_coeffs[t])
        T, V, S = T + c * a, V + c * b, S + c * s
    return T, V, S


def _rows(K):
    return max(1, min(K, 400_000 // K))


def _matrices(sysm, p, split=False):
    """Normalised H and S (or T and V apart) of a basis, and 1 / sqrt(diag S)."""
    K = len(p)
    f = 1.0 / torch.sqrt(_sums(sysm, p, p)[2].real)
    out = [torch.empty(K, K, dtype=torch.complex128, device=p.device) for _ in range(3 if split else 2)]
    with torch.no_grad():
        for k in range(0, K, _rows(K)):
            rows = slice(k, min(K, k + _rows(K)))
            T, V, S = _sums(sysm, p[rows, None], p[None])
            g = f[rows, None] * f[None]
            for m, v in zip(out, (S, T, V) if split else (S, T + V)):
                m[rows] = g * v
    for m in out:  # rows are bras; the lower triangle holds, as the stored matrices have it
        m.copy_(torch.tril(m) + torch.tril(m, -1).mH)
        m.diagonal().imag.zero_()
    return out, f


def _lowest(H, S, lam, x):
    lu = torch.linalg.lu_factor(H - lam * S)
    for _ in range(12):
        x = torch.linalg.lu_solve(*lu, (S @ x)[:, None])[:, 0]
        x = x / torch.view_as_real(x).abs().max()
    t = (x.conj() @ (S @ x)).real
    return ((x.conj() @ (H @ x)).real / t).item(), x / torch.sqrt(t)


def _full_gradient(sysm, p, f, c, E):
    K = len(p)
    p = p.clone().requires_grad_()
    for k in range(0, K, max(1, _rows(K) // 4)):
        rows = slice(k, min(K, k + max(1, _rows(K) // 4)))
        w = (c.conj() * f)[rows, None] * (c * f)[None]
        for t in range(sysm.T):
            T, V, S = _term(sysm, p[rows, None], p[None], t)
            (float(sysm.yhy_coeffs[t]) * (w * (T + V - E * S)).real.sum()).backward()
    return p.grad


def _row_gradient(sysm, pc, fc, p, f, cK, c, E):
    """Gradients of functions pc (B, npt), each beside the basis p: coefficients cK (B), c (B, K), energies E (B)."""
    pc = pc.clone().requires_grad_()
    w = (2.0 * cK.conj() * fc)[:, None] * (c * f[None])
    T, V, S = _sums(sysm, pc[:, None], p[None])
    e = (w * (T + V - E[:, None] * S)).real.sum()
    T, V, S = _sums(sysm, pc, pc)
    e = e + ((cK.abs() * fc) ** 2 * (T + V - E * S).real).sum()
    e.backward()
    return pc.grad


def _start(sysm, p0, floor):
    (S, H), _ = _matrices(sysm, p0)
    x = torch.ones(len(p0), dtype=torch.complex128, device=p0.device)
    lam = floor
    for _ in range(3):
        E, x = _lowest(H, S, lam, x)
        lam = E * INVIT_PARAMETER
    return S, H, lam, x


def exact(case, seed):
    kind, K = case["kind"], case["K"]
    if K * K * synth.make_system(case["system"]).T > 1e8:
        return None  # minutes of elementwise work
    sysm, p0, p1 = _inputs(case, seed)
    dev = _device()
    p0, p1 = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (p0, p1))
    if kind == "expectation":
        (S, T, V), _ = _matrices(sysm, p0, split=True)
        # the lowest pair of the pencil: C^-1 H C^-H with S = C C^H
        E, c = _general(T + V, S)
        v = {m: (c.conj() @ (A @ c)).real.item() for m, A in (("T", T), ("V", V), ("S", S), ("H", T + V))}
        return v
    if kind == "general":
        (S, H), f = _matrices(sysm, p1)
        E, c = _general(H, S)
        return dict(E=E, gradient=_full_gradient(sysm, p1, f, c, E).reshape(-1), err=None)
    S0, H0, lam, x = _start(sysm, p0, synth.SYSTEMS[case["system"]]["e_floor"])
    if kind in ("candidates", "candgrad"):
        return _exact_batch(case, sysm, p0, p1, S0, H0, lam, x)
    p = torch.cat([p0[:K - len(p1)], p1])
    (S, H), f = _matrices(sysm, p)
    v = torch.zeros(K, dtype=torch.complex128, device=dev)
    v[:len(x)] = x
    E, c = _lowest(H, S, lam, v)
    if kind in ("trial", "energy"):
        return dict(E=E, err=None)
    if kind == "function":
        one = torch.tensor([E], dtype=torch.float64, device=dev)
        g = _row_gradient(sysm, p[-1:], f[-1:], p[:-1], f[:-1], c[-1:], c[None, :-1], one)
    else:
        g = _full_gradient(sysm, p, f, c, E)
    return dict(E=E, gradient=g.reshape(-1), err=None)


def _general(H, S):
    """Lowest eigenpair without a shift known beforehand: dense solution, then refined by inverse iteration."""
    C = torch.linalg.cholesky(S)
    A = torch.linalg.solve_triangular(C, H, upper=False)
    A = torch.linalg.solve_triangular(C, A.mH.contiguous(), upper=False).mH
    w, v = torch.linalg.eigh(0.5 * (A + A.mH))
    x = torch.linalg.solve_triangular(C.mH.contiguous(), v[:, :1].contiguous(), upper=True)[:, 0]
    E = w[0].item()
    return _lowest(H, S, E - 1e-7 * abs(E), x)


def _exact_batch(case, sysm, p0, pc, S0, H0, lam, x):
    """Every trial's iterations at once: its own row and column beside the base."""
    f0 = 1.0 / torch.sqrt(_sums(sysm, p0, p0)[2].real)
    T, V, S = _sums(sysm, pc, pc)
    fc = 1.0 / torch.sqrt(S.real)
    mu = (T + V).real * fc * fc - lam
    B, K = len(pc), len(p0)
    s = torch.empty(B, K, dtype=torch.complex128, device=p0.device)
    m = torch.empty_like(s)
    with torch.no_grad():
        for j in range(0, B, _rows(K)):
            rows = slice(j, min(B, j + _rows(K)))
            T, V, S = _sums(sysm, pc[rows, None], p0[None])
            g = fc[rows, None] * f0[None]
            s[rows], m[rows] = g * S, g * (T + V - lam * S)
    s, m = s.mH.contiguous(), m.mH.contiguous()  # columns S(:, K), M(:, K) of each trial
    M0 = H0 - lam * S0
    lu = torch.linalg.lu_factor(M0)
    G = torch.linalg.lu_solve(*lu, m)
    delta = mu - (m.conj() * G).sum(0)
    v, vk = x[:, None].repeat(1, B), torch.zeros(B, dtype=torch.complex128, device=p0.device)
    active = torch.ones(B, dtype=torch.bool, device=p0.device)
    for _ in range(MAX_ITER):
        w, wk = S0 @ v + s * vk, (s.conj() * v).sum(0) + vk
        y = torch.linalg.lu_solve(*lu, w)
        xk = (wk - (m.conj() * y).sum(0)) / delta
        y = y - G * xk
        top = torch.maximum(torch.view_as_real(y).abs().amax((0, 2)), torch.view_as_real(xk).abs().amax(-1))
        y, xk = y / top, xk / top
        tc = ((y.conj() * v).sum(0) + xk.conj() * vk) / ((v.abs() ** 2).sum(0) + vk.abs() ** 2)
        off = math.sqrt(2.0 * (K + 1)) * torch.sqrt(((y - tc * v).abs() ** 2).sum(0) + (xk - tc * vk).abs() ** 2)
        v, vk = torch.where(active, y, v), torch.where(active, xk, vk)
        active = active & (off > TOL_BATCH)
        if not bool(active.any()):
            break
    t1 = (v.conj() * (S0 @ v)).sum(0).real + 2.0 * (vk.conj() * (s.conj() * v).sum(0)).real + vk.abs() ** 2
    t2 = (v.conj() * (M0 @ v)).sum(0).real + 2.0 * (vk.conj() * (m.conj() * v).sum(0)).real + mu * vk.abs() ** 2
    E = t2 / t1 + lam
    if case["kind"] == "candidates":
        return dict(E=E, err=None)
    r = 1.0 / torch.sqrt(t1)
    g = torch.empty(B, sysm.npt, dtype=torch.float64, device=p0.device)
    few = max(1, _rows(K) // (4 * sysm.T))
    for j in range(0, B, few):
        rows = slice(j, min(B, j + few))
        g[rows] = _row_gradient(sysm, pc[rows], fc[rows], p0, f0, (vk * r)[rows], (v * r).T[rows], E[rows])
    return dict(E=E, err=None, gradient=g)
