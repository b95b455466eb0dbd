"""The calls whose speed is looked after, each through the package's public
Python entry points.

  kind       entry points                                     stands for
  solve      Engine: set_U_device, solve,                     f(A)b with vectors on the GPU
             get_solution_device
  solve-host Engine.solve_host                                f(A)b from and to host arrays
  staged     LanczosEngine: set_U, build_subspace,            the reference's MATLAB loop, one
             lin_sys_solves, apply_V, get_xsol, update_U,     time step of it (two columns)
             get_U
  loop       Engine: set_state, time_loop, get_state          the time loop in one call
  batch      BatchEngine: set_U_device, solve,                many uneven problems in one launch
             get_solution_device
  adjoint    frac_fe_solve forward and backward               one gradient of an inverse problem
  pairs      eigs.deflation_pairs                             the set-up's eigenpairs

Operators: ``fd2d`` is the N x N five-point Dirichlet Laplacian, ``fd3d`` the
N^3 seven-point one with a variable coefficient, ``disk`` a P1 finite-element
operator with a log-normal coefficient on a Delaunay disk of about N nodes
(the nonuniform one), ``neumann`` the monodomain's N x N Neumann Laplacian.
Operators depend on the size alone and are kept between calls of ``prepare``,
as a program keeps its mesh; right-hand sides, initial states and the
adjoint's coefficients come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gpumatfun_gb300 import adjoint, eigs, engine, params, problems, workloads

DEV = "cuda"


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest grid that is used in earnest: latency and launches
        dict(name="fd2d-64", kind="solve", op="fd2d", N=64, R=1, prec="fp64", m=60, C=32, d=0, k=10, reorth=0),
        # the plain workload (256 x 256, ten deflated modes), host arrays in and out
        dict(name="fd2d-256-host", kind="solve-host", op="fd2d", N=256, R=1, prec="fp64", m=60, C=32, d=0, k=10,
             reorth=0),
        # a serving batch: uneven grids, four right-hand sides each, one launch
        dict(name="batch-24-mixed", kind="batch", op="fd2d", N=512, nprob=24, R=4, prec="mixed", m=32, C=32, d=0, k=0,
             reorth=0),
        # the fractional monodomain at the reference's own rules for m and C
        dict(name="monodomain-128-loop", kind="loop", op="neumann", N=128, steps=4, R=2, prec="fp64", k=10),
        # the same, larger and in mixed precision
        dict(name="monodomain-256-mixed", kind="loop", op="neumann", N=256, steps=2, R=2, prec="mixed", k=10),
        # one Fisher-KPP step on a finite-element disk through the reference's handle methods
        dict(name="disk-20k-staged", kind="staged", op="disk", N=20_000, R=2, prec="fp64", m=80, C=48, d=8, k=0,
             reorth=0),
        # the headline operator and parameters: a disk of a million nodes, degree 8
        dict(name="disk-1M", kind="solve", op="disk", N=1_000_000, R=1, prec="fp64", m=80, C=48, d=8, k=0, reorth=0),
        # four right-hand sides in mixed precision
        dict(name="disk-300k-mixed-r4", kind="solve", op="disk", N=300_000, R=4, prec="mixed", m=80, C=48, d=8, k=0,
             reorth=0),
        # three dimensions, streamed from HBM, mixed precision
        dict(name="fd3d-160-mixed", kind="solve", op="fd3d", N=160, R=1, prec="mixed", m=100, C=32, d=0, k=0, reorth=0),
        # three dimensions in FP64, an odd side, reorthogonalised once
        dict(name="fd3d-117-cgs", kind="solve", op="fd3d", N=117, R=1, prec="fp64", m=60, C=32, d=0, k=0, reorth=1),
        # forward and backward of the adjoint on a disk
        dict(name="adjoint-40k", kind="adjoint", op="disk", N=40_000, R=1, prec="fp64", m=200, C=32, d=8),
        # the set-up's deflation pairs
        dict(name="pairs-15k", kind="pairs", op="disk", N=15_000, k=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve-host", "staged", "loop", "batch", "adjoint", "pairs"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "pairs":
        return dict(kind=kind, op="disk", N=_log(rng, 3000, 15_000), k=rng.randint(4, 20))
    if kind == "adjoint":
        return dict(kind=kind, op="disk", N=_log(rng, 3000, 40_000), R=1, prec=prec, m=rng.randint(60, 200),
                    C=rng.choice([24, 32]), d=8)
    if kind == "loop":
        return dict(kind=kind, op="neumann", N=_log(rng, 48, 256), steps=rng.randint(1, 4), R=2, prec=prec,
                    k=rng.randint(4, 12))
    if kind == "batch":
        return dict(kind=kind, op="fd2d", N=_log(rng, 96, 512), nprob=rng.randint(4, 24), R=rng.choice([1, 2, 4]),
                    prec=prec, m=rng.randint(24, 40), C=rng.choice([24, 32]), d=0, k=0, reorth=0)
    if kind == "staged":
        return dict(kind=kind, op="disk", N=_log(rng, 3000, 200_000), R=2, prec=prec, m=rng.randint(40, 80),
                    C=rng.choice([32, 48]), d=rng.choice([0, 4, 8]), k=0, reorth=0)
    op = rng.choice(["fd2d", "fd3d", "disk"])
    R = rng.choice([1, 1, 2, 4])
    if op == "disk":
        return dict(kind=kind, op=op, N=_log(rng, 5000, 500_000), R=R, prec=prec, m=rng.randint(40, 80),
                    C=rng.choice([32, 48]), d=rng.choice([0, 4, 8]), k=0, reorth=0)
    if op == "fd3d":
        return dict(kind=kind, op=op, N=_log(rng, 24, 120), R=R, prec=prec, m=rng.randint(40, 80), C=32, d=0, k=0,
                    reorth=rng.choice([0, 0, 0, 1]) if R == 1 else 0)
    return dict(kind=kind, op=op, N=_log(rng, 48, 700), R=R, prec=prec, m=rng.randint(40, 80), C=rng.choice([24, 32]),
                d=rng.choice([0, 0, 3]), k=rng.choice([0, 6, 10]), reorth=0)


# ------------------------------------------------------------------ operators
@functools.lru_cache(maxsize=None)
def _disk(N):
    mesh = problems.disk_mesh(N, seed=0)
    g = problems.gaussian_random_field(mesh.nodes[mesh.tris].mean(axis=1), sigma=1.0, ell=0.1, seed=1)
    kappa = np.exp(g)
    A, ms, _ = problems.fe_operator(mesh, kappa)
    # Gershgorin bound, and the unit disk's smallest eigenvalue at the smallest coefficient
    return mesh, kappa, A, ms, 5.78 * float(kappa.min()), float(abs(A).sum(axis=1).max())


@functools.lru_cache(maxsize=None)
def _fd3d(N):
    A = problems.laplacian_3d_var(N)
    h = 1.0 / (N + 1)
    return A, 0.5 * 12 * math.sin(math.pi * h / 2) ** 2 / (h * h), float(2 * A.diagonal().max())


@functools.lru_cache(maxsize=None)
def _sides(N, nprob):
    return [int(v) for v in workloads.batch_sizes(nprob, 64, N, seed=3)]


@functools.lru_cache(maxsize=64)
def _fd2d_problem(N, k, m, C, d, R, batch):
    if batch:   # one diffusion step u <- exp(-dt K A^(3/4)) u on [0, 2.5]^2
        f = [params.frac_exp(1e-4 * 0.05, 1.5)] * R
        return workloads.fd2d_problem(N, 0, m, C, f, R=R, scale=((N + 1) / 2.5) ** 2, degree=d)
    return workloads.fd2d_problem(N, k, m, C, [params.frac_exp(1e-3, 1.5)] * R, R=R, scale=float((N + 1) ** 2), degree=d)


@functools.lru_cache(maxsize=8)
def _monodomain(N, k):
    return workloads.monodomain_problem(N, k=k)


def _problem(case):
    """The operator and method parameters (a workloads.FabProblem) of one case."""
    R, m, C, d = case["R"], case["m"], case["C"], case["d"]
    if case["op"] == "fd2d":
        return _fd2d_problem(case["N"], case["k"], m, C, d, R, False)
    none = np.zeros(0)
    if case["op"] == "fd3d":
        A, l1, lN = _fd3d(case["N"])
        funcs = [params.frac_exp(5e-4, 1.2)] * R
        row_weight = None
    else:
        _, _, A, row_weight, l1, lN = _disk(case["N"])
        if case["kind"] == "staged":
            funcs = [params.frac_exp(1e-4, 1.5), params.frac_phi(1e-4, 1.5)]
        else:
            funcs = [params.frac_power(-0.8)] * R
    n = A.shape[0]
    return workloads.make_problem(case["op"], A, np.zeros((n, R)), np.zeros((n, 0)), none, funcs, m, C, l1, lN,
                                  degree=d, prob_dim=lN / 4, row_weight=row_weight)


def _random(seed, *shape):
    """Uniform [0, 1) on the GPU, from the seed."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _rhs(seed, R, n):
    """R normalised right-hand sides, one per row (column-major n x R)."""
    U = _random(seed, R, n)
    return U / U.norm(dim=1, keepdim=True)


def _state0(case, seed):
    """Initial state of the time loops: columns [solution, reaction], and ode."""
    if case["kind"] == "staged":
        n = _disk(case["N"])[2].shape[0]
        u = _random(seed, n).cpu().numpy()
        return np.asfortranarray(np.stack([u, 0.05 * u * (1 - u)], axis=1)), np.zeros(n)
    P, dt, ode, f = _monodomain(case["N"], case["k"])
    x = P.U[:, 0] + 0.05 * _random(seed, P.n).cpu().numpy()
    y = f["c1ion"] / f["vamp"] ** 2 * x * (x - f["vrest"]) * (x - f["vpeak"]) - ode
    return np.asfortranarray(np.stack([x, dt * y], axis=1)), ode.copy()


DT = 0.05


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "pairs":
        A = _disk(case["N"])[2]
        # the operator of another time step: A plus a multiple of the identity
        shift = float(torch.rand(1, generator=torch.Generator().manual_seed(seed), dtype=torch.float64)) * 5.0
        B = A.copy()
        B.setdiag(B.diagonal() + shift)
        st["A"] = B
        return st
    if kind == "adjoint":
        mesh, kappa0, A, _, l1, lN = _disk(case["N"])
        n = A.shape[0]
        op = adjoint.FracFEOperator(mesh, kappa0, m=case["m"], C=case["C"], degree=case["d"], l1=l1 / 2, lN=lN * 2,
                                    precision=case["prec"])
        kappa = torch.from_numpy(kappa0).to(DEV) * (0.8 + 0.4 * _random(seed, kappa0.size))
        st.update(op=op, kappa=kappa.requires_grad_(True), b=_rhs(seed + 1000, 1, n)[0].clone().requires_grad_(True),
                  data=0.01 * _rhs(seed + 2000, 1, n)[0])
        return st
    if kind == "loop":
        P, dt, _, f = _monodomain(case["N"], case["k"])
        U, ode = _state0(case, seed)
        st["engine"] = engine.Engine(P.A, P.U, P.Q, P.lam, P.flam, P.m, P.gamma, P.gs_re, P.gs_im, P.wts, P.shifts,
                                     dt=dt, ode=ode, fhn=f, precision=case["prec"])
        st.update(U=U, ode=ode)
        return st
    if kind == "staged":
        P = _problem(case)
        U, ode = _state0(case, seed)
        z = 0.0
        st["engine"] = engine.LanczosEngine(
            U, P.A, None, None, P.m, P.gamma, P.gs_re, P.gs_im, np.zeros(0), np.zeros(0), DT, ode, z, z, z, z, 1.0, z,
            z, z, z, np.ones(P.n), P.wts[0], P.wts[1], P.shifts, row_weight=P.row_weight, precision=case["prec"])
        st["U"] = U
        return st
    if kind == "batch":
        Ps = [_fd2d_problem(N, 0, case["m"], case["C"], case["d"], case["R"], True)
              for N in _sides(case["N"], case["nprob"])]
        st["engine"] = engine.BatchEngine(Ps, precision=case["prec"])
        n = sum(P.n for P in Ps)
    else:
        P = _problem(case)
        st["engine"] = engine.Engine.from_problem(P, precision=case["prec"], reorth=case["reorth"])
        n = P.n
    U = _rhs(seed, case["R"], n)
    if kind == "solve-host":
        st["b"] = np.asfortranarray(U.cpu().numpy().T)
    else:
        st["U"] = U
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pairs":
        lam, Q, _ = eigs.deflation_pairs(state["A"], case["k"])
        return lam, Q
    if kind == "adjoint":
        kappa, b = state["kappa"], state["b"]
        x = adjoint.frac_fe_solve(kappa, b, state["op"])
        gk, gb = torch.autograd.grad(0.5 * (x - state["data"]).square().sum(), (kappa, b))
        return x.detach(), gk, gb
    e = state["engine"]
    if kind == "loop":
        e.set_state(state["U"], state["ode"])
        e.time_loop(case["steps"], monodomain=True)
        return e.get_state()
    if kind == "staged":
        e.set_U(state["U"])
        e.build_subspace()
        e.lin_sys_solves()
        e.apply_V()
        x = e.get_xsol()
        e.update_U()
        return x, e.get_U()
    if kind == "solve-host":
        return e.solve_host(state["b"])
    U = state["U"]
    e.set_U_device(U.data_ptr())
    e.solve()
    x = torch.empty_like(U)
    e.get_solution_device(x.data_ptr())
    return x


# ------------------------------------------------------------------ work
def _solve_flops(n, nnz, R, m, d, k, reorth=0):
    step = 2 * nnz * (d + 1) + n * (2 * d + 12) + (2 * n * (m + 1) * reorth if reorth else 0)
    return R * (m * step + 2 * m * n * (d + 1) + d * 2 * nnz + 8 * k * n)


def _solve_bytes(n, nnz, R, k, prec):
    return nnz * ((8 if prec == "fp64" else 4) + 4) + 4 * n + 8 * n * (2 * R + k)


def work(case):
    """Inputs read once, outputs written once, and the method's own operations."""
    kind, prec = case["kind"], case.get("prec", "fp64")
    if kind == "pairs":
        A = _disk(case["N"])[2]
        n, nnz = A.shape[0], A.nnz
        # four filter applications of degree about 400 on 32 vectors
        return dict(bytes=12 * nnz + 8 * n * (case["k"] + 1), flops=1600 * 64 * nnz)
    if kind == "adjoint":
        mesh, _, A, _, _, _ = _disk(case["N"])
        n, nnz, m, C, d, nt = A.shape[0], A.nnz, case["m"], case["C"], case["d"], mesh.tris.shape[0]
        grad = 2 * (8 * n * m * C + d * C * (4 * nnz + 8 * n)) + nt * C * 42
        return dict(bytes=3 * 8 * n + 2 * 8 * nt + 12 * nnz, flops=2 * _solve_flops(n, nnz, 1, m, d, 0) + grad)
    if kind == "loop":
        P = _monodomain(case["N"], case["k"])[0]
        n, nnz = P.n, P.A.nnz
        return dict(bytes=_solve_bytes(n, nnz, 2, P.k, prec) + 16 * n,
                    flops=case["steps"] * (_solve_flops(n, nnz, 2, P.m, P.d, P.k) + 20 * n))
    if kind == "batch":
        ns = [N * N for N in _sides(case["N"], case["nprob"])]
        return dict(bytes=sum(_solve_bytes(n, 5 * n, case["R"], 0, prec) for n in ns),
                    flops=sum(_solve_flops(n, 5 * n, case["R"], case["m"], case["d"], 0) for n in ns))
    N = case["N"]
    if case["op"] == "disk":
        n, nnz = N, 7 * N
    else:
        n, nnz = (N * N, 5 * N * N) if case["op"] == "fd2d" else (N ** 3, 7 * N ** 3)
    return dict(bytes=_solve_bytes(n, nnz, case["R"], case["k"], prec),
                flops=_solve_flops(n, nnz, case["R"], case["m"], case["d"], case["k"], case["reorth"]))


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _csr(A):
    return torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)),
                                   torch.from_numpy(A.indices.astype(np.int64)),
                                   torch.from_numpy(np.asarray(A.data, dtype=np.float64)), size=A.shape).to(DEV)


class _Krylov:
    """Lanczos on A p(A) from u, then the shifted solves (sigma_j - T) y_j = w_j beta_0 e_1."""

    def __init__(self, A, gamma, sigma, m, u, w, reorth=0):
        n = u.numel()
        V = torch.empty(m, n, dtype=torch.float64, device=DEV)
        alpha, beta = torch.zeros(m, dtype=torch.float64), torch.zeros(m + 1, dtype=torch.float64)
        beta[0] = u.norm().item()
        v, vp = u / beta[0].item(), None
        for j in range(m):
            V[j] = v
            p = gamma[0] * v
            for g in gamma[1:]:
                p = A @ p + g * v
            t = A @ p
            if vp is not None:
                t -= beta[j].item() * vp
            alpha[j] = torch.dot(t, v).item()
            t -= alpha[j].item() * v
            for _ in range(reorth):
                t -= V[:j + 1].T @ (V[:j + 1] @ t)
            beta[j + 1] = t.norm().item()
            vp, v = v, t / beta[j + 1].item()
        T = torch.diag(alpha) + torch.diag(beta[1:m], 1) + torch.diag(beta[1:m], -1)
        e1 = torch.zeros(m, 1, dtype=torch.complex128)
        e1[0, 0] = 1.0
        M = torch.from_numpy(sigma)[:, None, None] * torch.eye(m, dtype=torch.complex128) - T
        y = torch.linalg.solve(M.to(DEV), e1.to(DEV)[None])[:, :, 0] * beta[0].item()
        self.V, self.y, self.w = V, y, torch.from_numpy(w).to(DEV)     # y (C, m), unweighted

    def apply(self, A, gs):
        coef = torch.einsum("ic,cm->im", gs, self.w[:, None] * self.y).imag.contiguous()
        P = coef @ self.V
        x = P[0].clone()
        for i in range(1, gs.shape[0]):
            x = A @ x + P[i]
        return x


def _exact_solve(A, P, U, reorth=0):
    """(X, update) for right-hand sides U (R, n): deflated Krylov part, and the deflated modes' part."""
    gs = torch.from_numpy(P.gs_re + 1j * P.gs_im).to(DEV)
    Q = torch.from_numpy(np.ascontiguousarray(P.Q)).to(DEV)
    X, upd = [], []
    for r in range(U.shape[0]):
        z = Q.T @ U[r]
        u = U[r] - Q @ z
        upd.append(Q @ (torch.from_numpy(np.ascontiguousarray(P.flam[:, r])).to(DEV) * z))
        w = P.wts[r][:, 0] + 1j * P.wts[r][:, 1]
        X.append(_Krylov(A, P.gamma, P.sigma, P.m, u, w, reorth).apply(A, gs))
    return torch.stack(X), torch.stack(upd)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pairs":
        return None   # eigenvectors have no sign of their own, and a dense solve takes too long
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "loop":
        P, dt, _, f = _monodomain(case["N"], case["k"])
        A = _csr(P.A)
        U0, ode = _state0(case, seed)
        U, o = torch.from_numpy(np.ascontiguousarray(U0.T)).to(DEV), torch.from_numpy(ode).to(DEV)
        for _ in range(case["steps"]):
            X, upd = _exact_solve(A, P, U)
            u = X.sum(dim=0) + upd.sum(dim=0)
            o = o + dt * (f["aode"] * u + f["bode"] * o) + f["code"]
            src = f["c1ion"] / f["vamp"] ** 2 * (u - f["vrest"]) * u * (u - f["vpeak"])
            U = torch.stack([u, dt * (src - o)])
        return U.T.cpu().numpy(), o.cpu().numpy()
    if kind == "staged":
        P = _problem(case)
        U0, _ = _state0(case, seed)
        U = torch.from_numpy(np.ascontiguousarray(U0.T)).to(DEV)
        U[1] *= DT
        X, upd = _exact_solve(_csr(P.A), P, U)
        u = (X.sum(dim=0) + upd.sum(dim=0)).clamp(min=0.0)
        return X.T.cpu().numpy(), torch.stack([u, DT * u * (1.0 - u)], dim=1).cpu().numpy()
    if kind == "batch":
        Ps = [_fd2d_problem(N, 0, case["m"], case["C"], case["d"], case["R"], True)
              for N in _sides(case["N"], case["nprob"])]
        U = _rhs(seed, case["R"], sum(P.n for P in Ps))
        out, at = [], 0
        for P in Ps:
            out.append(_exact_solve(_csr(P.A), P, U[:, at:at + P.n])[0])
            at += P.n
        return torch.cat(out, dim=1)
    P = _problem(case)
    U = _rhs(seed, case["R"], P.n)
    X, upd = _exact_solve(_csr(P.A), P, U, case["reorth"])
    S = X + upd
    return S.T.cpu().numpy() if kind == "solve-host" else S


def _exact_adjoint(case, seed):
    """x = f(A(kappa)) b and its gradients from the two Krylov states, as plain matrix products."""
    mesh, kappa0, A0, ms, l1, lN = _disk(case["N"])
    m, C, d = case["m"], case["C"], case["d"]
    l1, lN = l1 / 2, lN * 2
    con = params.hht_contour(l1, lN, C)
    gamma = params.polynomial_coeffs(d, lN / 4.0)
    gs, sigma = params.shifted_poly_coeffs(gamma, con.xi)
    w = con.weights(params.frac_power(-0.8))
    n = A0.shape[0]
    kappa = torch.from_numpy(kappa0).to(DEV) * (0.8 + 0.4 * _random(seed, kappa0.size))
    b, data = _rhs(seed + 1000, 1, n)[0], 0.01 * _rhs(seed + 2000, 1, n)[0]
    A = _csr(problems.fe_operator(mesh, kappa.cpu().numpy())[0])
    gst = torch.from_numpy(gs).to(DEV)
    kb = _Krylov(A, gamma, sigma, m, b, w)
    x = kb.apply(A, gst)
    g = x - data
    kg = _Krylov(A, gamma, sigma, m, g, w)
    db = kg.apply(A, gst)

    def lifted(kr, weight):
        # rows of q_j(A) V y_j, all nodes of the contour at once
        y = kr.y * weight[:, None]
        Z = torch.cat([y.real @ kr.V, y.imag @ kr.V]).T.contiguous()          # n x 2C
        gr, gi = gst.real, gst.imag

        def times(i):
            zr, zi = Z[:, :C], Z[:, C:]
            return torch.cat([gr[i] * zr - gi[i] * zi, gr[i] * zi + gi[i] * zr], dim=1)
        S = times(0)
        for i in range(1, d + 1):
            S = A @ S + times(i)
        return S
    Rj, Sj = lifted(kb, torch.ones(C, dtype=torch.complex128, device=DEV)), lifted(kg, kg.w)
    area, G = problems.p1_element_grads(mesh.nodes, mesh.tris)
    Ke = torch.from_numpy(np.einsum("tid,tjd->tij", G, G) * area[:, None, None]).to(DEV)
    idx = np.full(mesh.nodes.shape[0], n, dtype=np.int64)
    inner = np.flatnonzero(~mesh.boundary)
    idx[inner] = np.arange(n)
    tri = torch.from_numpy(idx[mesh.tris]).to(DEV)
    msi = torch.cat([1.0 / torch.from_numpy(ms), torch.zeros(1, dtype=torch.float64)]).to(DEV)
    Kc = Ke * msi[tri][:, :, None] * msi[tri][:, None, :]
    zero = torch.zeros(1, 2 * C, dtype=torch.float64, device=DEV)
    Rt, St = torch.cat([Rj, zero])[tri], torch.cat([Sj, zero])[tri]            # (nt, 3, 2C)
    KR = Kc @ Rt
    dk = (St[:, :, :C] * KR[:, :, C:] + St[:, :, C:] * KR[:, :, :C]).sum(dim=(1, 2))
    return x, dk, db
