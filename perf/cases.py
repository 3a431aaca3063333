"""The workloads on which this library is timed.

Each case is one call (or the few calls that always go together) of the public
interface, the way a simulation makes it: the drop-in functions on host arrays,
the device entry points of the C ABI inside a Newton loop, the linear solves
with each preconditioner, whole Newton solves, and one training step of the
learned preconditioner. Meshes are Kuhn-subdivided boxes (grid numbering) and
balls carved out of them with a shuffled vertex numbering, as mesh generators
leave it; rest vertices are jittered, stiffness varies from tet to tet, and the
state is a smooth deformation plus vertex noise.

The linear systems of the solver cases are assembled here in 64 bits and
rounded once to the FP32 values that the solver takes, so they do not depend on
the library's own assembly.
"""
import ctypes
import functools
import itertools
import math
import random

import numpy as np
import torch

import bartels_gb300 as bg
from bartels_gb300 import _lib, lpcg

DT, RHO, NU = 0.01, 1000.0, 0.45


# ------------------------------------------------------------------- cases ---
def listed():
    return [
        # the drop-in functions on host arrays, on a mesh of the size that the examples and tests use: a
        # line search or an optimiser that evaluates energy and gradient once per step
        dict(name="dropin_q_dq_n8", kind="dropin", model="neohookean", shape="box", nx=8, ny=8, nz=8, strain=0.05),
        # energy and gradient on device arrays: every Newton iteration and every line-search trial of the
        # 5.3M-tet benchmark cube
        dict(name="q_dq_nh_n96", kind="elements", model="neohookean", shape="box", nx=96, ny=96, nz=96, strain=0.02),
        # the same with the SVD-based law on a ragged box of ordinary size
        dict(name="q_dq_corot_n41", kind="elements", model="corotational", shape="box", nx=45, ny=41, nz=37,
             strain=0.2),
        # Newton Hessian M + dt^2 K without projection at benchmark size
        dict(name="hess_nh_n96", kind="hessian", model="neohookean", psd=False, shape="box", nx=96, ny=96, nz=96,
             strain=0.02),
        # projected Newton Hessian of a body that sags and is slightly compressed (most elements need the projection)
        dict(name="hess_psd_nh_n56", kind="hessian", model="neohookean", psd=True, shape="box", nx=56, ny=56, nz=56,
             strain=-0.005),
        # projected Hessian under strong compression on a carved, shuffled mesh
        dict(name="hess_psd_stvk_ball", kind="hessian", model="stvk", psd=True, shape="ball", nx=33, ny=37, nz=35,
             strain=-0.3),
        # the drop-in search direction (a sparse direct solve in the reference) on host CSR arrays
        dict(name="direction_csr_n14", kind="direction", shape="box", nx=14, ny=13, nz=15, young=2e6),
        # the linear solve of a Newton iteration on the benchmark cube, multigrid-preconditioned
        dict(name="solve_mg_n96", kind="solve", precond="multigrid", shape="box", nx=96, ny=96, nz=96, young=2e6),
        # the same with the learned smoother (network forward and factor included) on an ordinary mesh
        dict(name="solve_lmg_n48", kind="solve", precond="learned_multigrid", shape="box", nx=52, ny=48, nz=44,
             young=2e6),
        # a batch of small meshes of uneven size packed into one plan, each with its own convergence test
        dict(name="packed_mg_24", kind="packed", precond="multigrid", count=24, nmin=8, nmax=22),
        # a whole implicit-Euler step from rest under gravity through the host-array call
        dict(name="newton_n24", kind="newton", model="neohookean", precond="multigrid", shape="box", nx=24, ny=24,
             nz=24, young=2e6),
        # one training step of the learned preconditioner on a training-size cube
        dict(name="train_n24", kind="train", shape="box", nx=24, ny=24, nz=24, young=2e6, probes=8),
    ]


def _dims(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {k: max(3, min(96, round(n * rng.uniform(0.8, 1.25)))) for k in ("nx", "ny", "nz")}


def draw(rng: random.Random):
    kind = rng.choice(["dropin", "elements", "elements", "hessian", "hessian", "direction", "solve", "solve", "packed",
                       "newton", "train"])
    shape = rng.choice(["box", "box", "ball"])
    model = rng.choice(["neohookean", "neohookean", "stvk", "corotational"])
    young = math.exp(rng.uniform(math.log(2e5), math.log(1e7)))
    strain = rng.choice([0.02, 0.1, -0.005, -0.05, -0.2])
    if kind == "dropin":
        return dict(kind=kind, model=model, shape=shape, strain=strain, **_dims(rng, 4, 20))
    if kind == "elements":
        hi = 36 if model == "corotational" else 80
        return dict(kind=kind, model=model, shape=shape, strain=strain, **_dims(rng, 6, hi))
    if kind == "hessian":
        psd = rng.random() < 0.6
        return dict(kind=kind, model=model, psd=psd, shape=shape, strain=strain, **_dims(rng, 6, 40 if psd else 72))
    if kind == "direction":
        return dict(kind=kind, shape=shape, young=young, **_dims(rng, 5, 14))
    if kind == "solve":
        precond = rng.choice(["multigrid", "multigrid", "learned_multigrid", "jacobi"])
        return dict(kind=kind, precond=precond, shape=shape, young=young,
                    **_dims(rng, 8, 24 if precond == "jacobi" else 56))
    if kind == "packed":
        lo = rng.randint(5, 10)
        return dict(kind=kind, precond=rng.choice(["multigrid", "jacobi"]), count=rng.randint(4, 32), nmin=lo,
                    nmax=rng.randint(lo + 2, 20))
    if kind == "newton":
        precond = rng.choice(["multigrid", "jacobi"])
        return dict(kind=kind, model=rng.choice(["neohookean", "stvk"]), precond=precond, shape="box", young=young,
                    **_dims(rng, 6, 12 if precond == "jacobi" else 22))
    return dict(kind="train", shape=shape, young=young, probes=rng.choice([4, 8]), **_dims(rng, 10, 28))


# ------------------------------------------------------------------ meshes ---
@functools.lru_cache(maxsize=4)
def _mesh(shape, nx, ny, nz):
    """Rest vertices (nV, 3), tets (nT, 4) and the edge length of a Kuhn-subdivided nx x ny x nz box of unit mean
    side, or of the ellipsoid carved out of it with shuffled vertex and tet numbers."""
    h = 1.0 / round((nx * ny * nz) ** (1.0 / 3.0))
    mx, my = nx + 1, ny + 1
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(my), np.arange(mx), indexing="ij")
    V = h * np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1).astype(np.float64)
    ck, cj, ci = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    if shape == "ball":
        c = np.stack([(ci.ravel() + 0.5) / nx, (cj.ravel() + 0.5) / ny, (ck.ravel() + 0.5) / nz], axis=1) - 0.5
        keep = (c * c).sum(axis=1) <= 0.25
    else:
        keep = slice(None)
    base = (ci + mx * (cj + my * ck)).ravel()[keep].astype(np.int32)
    step = (1, mx, mx * my)
    E = np.empty((len(base), 6, 4), np.int32)
    for t, p in enumerate(itertools.permutations(range(3))):
        a, b = base + step[p[0]], base + step[p[0]] + step[p[1]]
        odd = p in ((0, 2, 1), (1, 0, 2), (2, 1, 0))
        E[:, t, 0], E[:, t, 3] = base, base + sum(step)
        E[:, t, 1], E[:, t, 2] = (b, a) if odd else (a, b)
    E = E.reshape(-1, 4)
    if shape == "ball":
        r = np.random.RandomState(nx * 10007 + ny * 101 + nz)
        used = np.unique(E)
        new = r.permutation(len(used)).astype(np.int32)
        at = np.zeros(len(V), np.int32)
        at[used] = new
        W = np.empty((len(used), 3))
        W[new] = V[used]
        V, E = W, at[E][r.permutation(len(E))]
    return V, np.ascontiguousarray(E), h


def _pack(count, nmin, nmax, seed):
    r = np.random.RandomState(seed % (1 << 31))
    Vs, Es, voff, toff = [], [], [0], [0]
    for n in np.random.RandomState(count * 1009 + nmin * 31 + nmax).randint(nmin, nmax + 1, count):
        V, E, h = _mesh("box", int(n), int(n), int(n))
        Vs.append(V + 0.05 * h * r.uniform(-1, 1, V.shape) * (V[:, 2:] > 0))
        Es.append(E + voff[-1])
        voff.append(voff[-1] + len(V))
        toff.append(toff[-1] + len(E))
    return np.concatenate(Vs), np.concatenate(Es).astype(np.int32), voff, toff


def _case_mesh(case):
    return _mesh(case["shape"], case["nx"], case["ny"], case["nz"])


def _params(model, nT, young, r):
    """Per-tet parameters in the reference's convention, stiffness log-normal around young."""
    y = young * np.exp(0.3 * r.standard_normal(nT))
    lam, mu = y * NU / ((1 + NU) * (1 - 2 * NU)), y / (2 * (1 + NU))
    return np.stack([0.5 * mu, 0.5 * lam] if model == "neohookean" else [lam, mu], axis=1)


def _deformed(V, h, strain, r):
    """Positions: a stretch of 1 + strain along z (Poisson contraction across), a smooth bend and vertex noise."""
    s = np.array([1 - 0.3 * strain, 1 - 0.25 * strain, 1 + strain])
    a = 0.3 * abs(strain)
    w = a * np.stack([np.sin(2 * V[:, 2] + r.uniform(0, 3)), np.cos(2 * V[:, 0] + r.uniform(0, 3)),
                      np.sin(2 * V[:, 1] + r.uniform(0, 3))], axis=1)
    return V * s + w + min(0.02, abs(strain)) * 0.5 * h * r.uniform(-1, 1, V.shape)


def _geometry(case, seed):
    """Rest vertices, tets, edge length and the generator of the case's inputs."""
    V, E, h = _case_mesh(case)
    r = np.random.default_rng(seed)
    V = V + 0.08 * h * r.uniform(-1, 1, V.shape) * (V[:, 2:] > V[:, 2].min() + 1e-9)
    return V, E, h, r


# ------------------------------------------------- 64-bit element mathematics ---
def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _grads(V, E):
    """Shape-function gradients (nT, 4, 3) and volumes (nT,)."""
    x = V[E]
    D = (x[:, 1:] - x[:, :1]).transpose(1, 2)
    G = torch.linalg.inv(D)
    return torch.cat([-G.sum(1, keepdim=True), G], 1), torch.linalg.det(D) / 6


def _def_grad(q, E, phi):
    return q[E].transpose(1, 2) @ phi


def _cof(F):
    return torch.stack([torch.linalg.cross(F[..., 1], F[..., 2]), torch.linalg.cross(F[..., 2], F[..., 0]),
                        torch.linalg.cross(F[..., 0], F[..., 1])], -1)


def _psi_pk1(model, F, p):
    """Energy density and first Piola-Kirchhoff stress."""
    p0, p1 = p[:, 0], p[:, 1]
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    if model == "neohookean":
        G = _cof(F)
        J = (F * G).sum((1, 2)) / 3
        psi = p0 * ((F * F).sum((1, 2)) - 3 - 2 * torch.log(J)) + p1 * (J - 1) ** 2
        P = 2 * p0[:, None, None] * F + (2 * p1 * (J - 1) - 2 * p0 / J)[:, None, None] * G
    elif model == "stvk":
        Em = 0.5 * (F.transpose(1, 2) @ F - eye)
        tr = Em.diagonal(dim1=1, dim2=2).sum(1)
        psi = p1 * (Em * Em).sum((1, 2)) + 0.5 * p0 * tr * tr
        P = F @ (2 * p1[:, None, None] * Em + (p0 * tr)[:, None, None] * eye)
    else:
        U, S, Vh = torch.linalg.svd(F)
        tr = S.sum(1) - 3
        psi = p1 * ((S - 1) ** 2).sum(1) + 0.5 * p0 * tr * tr
        P = (U * (2 * p1[:, None] * (S - 1) + (p0 * tr)[:, None])[:, None, :]) @ Vh
    return psi, P


def _hess9(model, F, p):
    """d2psi/dF2 as (n, 3, 3, 3, 3): entry [k, i, l, j] for dF(k, i) dF(l, j); the corotational law in the
    reference's layout, which is its Hessian at F transposed."""
    p0, p1 = p[:, 0], p[:, 1]
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    big = torch.einsum("kl,ij->kilj", eye, eye)[None]

    def s(x):
        return x[:, None, None, None, None]

    if model == "neohookean":
        G = _cof(F)
        J = (F * G).sum((1, 2)) / 3
        eps = torch.zeros(3, 3, 3, dtype=F.dtype, device=F.device)
        for a, b, c in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
            eps[a, b, c], eps[a, c, b] = 1, -1
        d2J = torch.einsum("klm,ijn,tmn->tkilj", eps, eps, F)
        return (s(2 * p0) * big + s(2 * p0 / J ** 2 + 2 * p1) * torch.einsum("tki,tlj->tkilj", G, G)
                + s(2 * p1 * (J - 1) - 2 * p0 / J) * d2J)
    if model == "stvk":
        Em = 0.5 * (F.transpose(1, 2) @ F - eye)
        S = 2 * p1[:, None, None] * Em + (p0 * Em.diagonal(dim1=1, dim2=2).sum(1))[:, None, None] * eye
        return (torch.einsum("kl,tji->tkilj", eye, S) + s(p1) * (torch.einsum("tkj,tli->tkilj", F, F)
                + torch.einsum("tkm,tlm,ij->tkilj", F, F, eye)) + s(p0) * torch.einsum("tki,tlj->tkilj", F, F))
    U, S, Vh = torch.linalg.svd(F.transpose(1, 2))
    W = Vh.transpose(1, 2)
    R = U @ Vh
    H = s(2 * p1) * big + s(p0) * torch.einsum("tki,tlj->tkilj", R, R)
    c = p0 * (S.sum(1) - 3) - 2 * p1
    for i, j in ((0, 1), (0, 2), (1, 2)):
        T = (U[:, :, i, None] * W[:, None, :, j] - U[:, :, j, None] * W[:, None, :, i]) / math.sqrt(2.0)
        H = H + s(2 * c / (S[:, i] + S[:, j])) * torch.einsum("tki,tlj->tkilj", T, T)
    return H


def _element_matrices(model, F, phi, vol, p, psd_tol, cK, cM):
    """(n, 4, 3, 4, 3) element matrices cK K + cM M, K projected by clamping its eigenvalues to psd_tol."""
    K = torch.einsum("tai,tkilj,tbj->takbl", phi, _hess9(model, F, p), phi) * vol[:, None, None, None, None]
    if psd_tol is not None:
        shape, parts = K.shape, []
        for part in K.reshape(-1, 12, 12).split(20000):  # the batched eigen-solver takes no more at once
            L, Q = torch.linalg.eigh(part)
            parts.append((Q * L.clamp(min=psd_tol)[:, None, :]) @ Q.transpose(1, 2))
        K = torch.cat(parts).reshape(shape)
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    M = (torch.ones(4, 4, dtype=F.dtype, device=F.device) + torch.eye(4, dtype=F.dtype, device=F.device)) / 20
    return cK * K + (cM * RHO * vol)[:, None, None, None, None] * torch.einsum("ab,kl->akbl", M, eye)[None]


class _Pattern:
    """Block pattern of a mesh and the place of every element block in the values of its CSR matrix."""

    def __init__(self, nV, E):
        Eg = _dev(E).long()
        keys = torch.unique((Eg[:, :, None] * nV + Eg[:, None, :]).reshape(-1))
        self.n, self.nnz, self.E = 3 * nV, 9 * keys.numel(), Eg
        self.rb = torch.searchsorted(keys, torch.arange(nV + 1, device=keys.device) * nV)
        self.row, self.col = keys // nV, keys % nV
        self.keys = keys

    def add(self, values, t0, t1, K):
        """values += the element matrices K of tets t0..t1."""
        e = self.E[t0:t1]
        nV = self.n // 3
        nb = (self.rb[1:] - self.rb[:-1])[e] * 3
        three = torch.arange(3, device=e.device)
        for a in range(4):
            for b in range(4):
                j = torch.searchsorted(self.keys, e[:, a] * nV + e[:, b]) - self.rb[e[:, a]]
                at = (9 * self.rb[e[:, a]] + 3 * j)[:, None, None] + nb[:, a, None, None] * three[:, None] + three
                values.index_add_(0, at.reshape(-1), K[:, a, :, b, :].reshape(-1))

    def csr(self, values):
        """The matrix in 64 bits (torch CSR, 3x3 blocks expanded into scalar rows)."""
        nb = self.rb[1:] - self.rb[:-1]
        crow = torch.zeros(self.n + 1, dtype=torch.int64, device=nb.device)
        crow[1:] = torch.cumsum((3 * nb).repeat_interleave(3), 0)
        at = torch.arange(self.nnz, device=nb.device)
        v = torch.repeat_interleave(torch.arange(self.n, device=nb.device), (3 * nb).repeat_interleave(3))
        k = at - crow[v]
        col = 3 * self.col[self.rb[v // 3] + k // 3] + k % 3
        return torch.sparse_csr_tensor(crow, col, values, (self.n, self.n), check_invariants=False)


@functools.lru_cache(maxsize=2)
def _pattern(shape, nx, ny, nz):
    V, E, _ = _mesh(shape, nx, ny, nz)
    return _Pattern(len(V), E)


def _assemble(pat, V, q, params, model, psd_tol, cK, cM, chunk=300000):
    V, q, p = _dev(V), _dev(q), _dev(params)
    values = torch.zeros(pat.nnz, dtype=torch.float64, device="cuda")
    for t0 in range(0, len(pat.E), chunk):
        t1 = min(len(pat.E), t0 + chunk)
        e = pat.E[t0:t1]
        phi, vol = _grads(V, e)
        pat.add(values, t0, t1, _element_matrices(model, _def_grad(q, e, phi), phi, vol, p[t0:t1], psd_tol, cK, cM))
    return values


def _system(pat, V, h, young, r):
    """A Newton system M + dt^2 K of a slightly stretched body as FP32 values, and a right-hand side."""
    E = pat.E.cpu().numpy()
    params = _params("neohookean", len(E), young, r)
    q = V * np.array([1.01, 1.015, 1.02]) + 0.002 * np.sin(2 * V[:, [1, 2, 0]]) + 1e-3 * h * r.uniform(-1, 1, V.shape)
    values = _assemble(pat, V, q, params, "neohookean", None, DT * DT, 1.0).float()
    pinned = V[:, 2] <= V[:, 2].min() + 1e-9
    f = np.zeros(V.shape)
    f[:, 2] = -9.81 * RHO * h ** 3 * DT
    b = np.where(pinned[:, None], 0.0, f + 0.3 * np.abs(f).max() * r.standard_normal(V.shape)).ravel()
    return values, b, pinned, params


def _cg64(A, minv, b, free, tol=1e-14, iters=20000):
    """Conjugate gradients in 64 bits on the free unknowns, diagonally scaled."""
    x, r = torch.zeros_like(b), b * free
    z = minv * r
    p, rz, stop = z.clone(), r @ z, tol * float(b.norm())
    for it in range(iters):
        Ap = (A @ p) * free
        alpha = rz / (p @ Ap)
        x += alpha * p
        r -= alpha * Ap
        if it % 20 == 19 and float(r.norm()) <= stop:
            break
        z = minv * r
        rz2 = r @ z
        p, rz = z + (rz2 / rz) * p, rz2
    return x


# ----------------------------------------------------------------- prepare ---
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


_C = {}


def _net(kind):
    """The shipped network: one for inference, shared as a program shares it; one per training state."""
    if kind == "train":
        return lpcg.LearnedPreconditioner.load()
    if "net" not in _C:
        _C["net"] = lpcg.LearnedPreconditioner.load()
    return _C["net"]


def _use(plan, precond):
    if precond == "learned_multigrid":
        _net("use").attach(plan, multigrid=True)
    elif precond == "multigrid":
        lpcg.use_multigrid(plan)
    else:
        lpcg.use_block_jacobi(plan)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "packed":
        V, E, voff, toff = _pack(case["count"], case["nmin"], case["nmax"], seed)
        r = np.random.default_rng(seed)
        pat = _Pattern(len(V), E)
        values, b, pinned, _ = _system(pat, V, 1.0 / case["nmax"], 2e6, r)
        plan = bg.MeshPlan(V, E)
        plan.set_problem(pinned=pinned.astype(np.uint8))
        vo, to = np.array(voff, np.int32), np.array(toff, np.int64)
        _lib.check(bg.lib().bartels_plan_set_segments(
            plan.handle, case["count"], vo.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
            to.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))), "set_segments")
        _use(plan, case["precond"])
        b = _dev(b)
        return dict(kind="solve", plan=plan, values=values, b=b, x=torch.zeros_like(b), precond=case["precond"])
    V, E, h, r = _geometry(case, seed)
    if kind in ("solve", "direction", "train"):
        pat = _pattern(case["shape"], case["nx"], case["ny"], case["nz"])
        values, b, pinned, params = _system(pat, V, h, case["young"], r)
        if kind == "direction":
            P = bg.fixed_point_constraint_matrix(V, np.flatnonzero(pinned))
            A = bg.MeshPlan(V, E).csr(values.double().cpu().numpy())
            return dict(kind=kind, g=b[np.repeat(~pinned, 3)], H=P @ A @ P.T)
        plan = bg.MeshPlan(V, E)
        plan.set_problem(pinned=pinned.astype(np.uint8))
        if kind == "train":
            return dict(kind=kind, plan=plan, values=values, net=_net("train"), probes=case["probes"],
                        seed=seed & 0xFFFF)
        _use(plan, case["precond"])
        b = _dev(b)
        return dict(kind=kind, plan=plan, values=values, b=b, x=torch.zeros_like(b), precond=case["precond"])
    if kind == "newton":
        params = _params(case["model"], len(E), case["young"], r)
        plan = bg.MeshPlan(V, E)
        plan.set_element_data(params=params, density=np.full(len(E), RHO))
        force = plan.const_ext_force(None, np.array([0.0, 0.0, -9.81 * RHO]))
        pinned = V[:, 2] <= V[:, 2].min() + 1e-9
        plan.set_problem(q_base=V.ravel(), x_hat=np.zeros(3 * len(V)), f_ext=force, pinned=pinned.astype(np.uint8))
        _use(plan, case["precond"])
        prm = bg.newton_params(model=case["model"], psd_mode=_lib.PSD_SIMPLE_FIX, psd_tol=1e-6, mass_coeff=1.0, scale=DT,
                               force_scale=DT, gradient_tol=1e-8, relative=1, max_iterations=20,
                               inner_rel_tol=1e-1 if case["precond"] == "jacobi" else 1e-2)
        return dict(kind=kind, plan=plan, prm=prm, x0=np.zeros(3 * len(V)))
    model = case["model"]
    params = _params(model, len(E), 1e6, r)
    q = _deformed(V, h, case["strain"], r).ravel()
    if kind == "dropin":
        return dict(kind=kind, f=getattr(bg, "linear_tetmesh_%s_q" % model),
                    df=getattr(bg, "linear_tetmesh_%s_dq" % model),
                    args=(V, E, q, bg.linear_tetmesh_dphi_dX(V, E), bg.volume(V, E), params))
    plan = bg.MeshPlan(V, E)
    plan.set_element_data(params=params, density=np.full(len(E), RHO))
    q = _dev(q)
    state = dict(kind=kind, plan=plan, model=bg.api.MODELS[model], q=q)
    if kind == "elements":
        return dict(state, e=torch.zeros(1, dtype=torch.float64, device="cuda"), g=torch.zeros_like(q))
    return dict(state, psd=_lib.PSD_SIMPLE_FIX if case["psd"] else _lib.PSD_NONE,
                values=torch.zeros(plan.nnz, dtype=torch.float32, device="cuda"))


# --------------------------------------------------------------------- run ---
def run(state):
    kind, L = state["kind"], bg.lib()
    if kind == "dropin":
        return dict(energy=np.float64(state["f"](*state["args"])), gradient=state["df"](*state["args"]))
    if kind == "direction":
        # to the accuracy of the sparse direct solve that the reference makes here
        d, ok, _ = bg.search_direction_newton_sparse(state["g"], state["H"], rel_tol=1e-12)
        return dict(d=d, ok=ok)
    plan = state["plan"]
    if kind == "elements":
        _lib.check(L.bartels_tetmesh_q_d(plan.ctx.handle, plan.handle, state["model"], _ptr(state["q"]),
                                         _ptr(state["e"])), "q_d")
        _lib.check(L.bartels_tetmesh_dq_d(plan.ctx.handle, plan.handle, state["model"], _ptr(state["q"]),
                                          _ptr(state["g"])), "dq_d")
        return dict(energy=state["e"], gradient=state["g"])
    if kind == "hessian":
        _lib.check(L.bartels_plan_hessian_d(plan.ctx.handle, plan.handle, state["model"], state["psd"], 1e-6, 0,
                                            DT * DT, 1.0, _ptr(state["q"]), _ptr(state["values"])), "hessian_d")
        return dict(values=state["values"])
    if kind == "solve":
        rep = lpcg.plan_pcg(plan, state["values"], state["b"], state["x"], rel_tol=1e-9,
                            inner_rel_tol=1e-1 if state["precond"] == "jacobi" else 1e-2)
        return dict(x=state["x"], ok=bool(rep.converged))
    if kind == "newton":
        x, rep = plan.newton_solve(state["x0"], state["prm"])
        return dict(x=x, ok=rep.status == bg.CONVERGED)
    loss = state["net"].train_step(plan, state["values"], None, nprobes=state["probes"], seed=state["seed"], lr=1e-3)
    return dict(loss=np.float64(loss), gradient=state["net"].grad())


# -------------------------------------------------------------------- work ---
def _counts(case):
    """Vertices, tets and Hessian entries."""
    if case["kind"] == "packed":
        sizes = np.random.RandomState(case["count"] * 1009 + case["nmin"] * 31 + case["nmax"]).randint(
            case["nmin"], case["nmax"] + 1, case["count"])
        return np.sum([_counts(dict(kind="", shape="box", nx=int(n), ny=int(n), nz=int(n))) for n in sizes], axis=0)
    x, y, z = case["nx"], case["ny"], case["nz"]
    if case["shape"] == "ball":
        V, E, _ = _case_mesh(case)
        pairs = np.concatenate([np.sort(E[:, [a, b]], axis=1) for a, b in itertools.combinations(range(4), 2)])
        edges = len(np.unique(pairs[:, 0].astype(np.int64) * len(V) + pairs[:, 1]))
        return np.array([len(V), len(E), 9 * (len(V) + 2 * edges)])
    X, Y, Z = x + 1, y + 1, z + 1
    edges = x * Y * Z + X * y * Z + X * Y * z + x * y * Z + x * Y * z + X * y * z + x * y * z
    return np.array([X * Y * Z, 6 * x * y * z, 9 * (X * Y * Z + 2 * edges)])


def work(case):
    nV, nT, nnz = (int(v) for v in _counts(case))
    kind = case["kind"]
    if kind in ("dropin", "elements"):
        return dict(bytes=112 * nT + 48 * nV, flops=300 * nT)
    if kind == "hessian":
        return dict(bytes=64 * nT + 24 * nV + 4 * nnz, flops=(6000 if case["psd"] else 900) * nT)
    if kind == "direction":
        return dict(bytes=12 * nnz + 48 * nV, flops=2 * nnz)
    if kind in ("solve", "packed"):
        return dict(bytes=4 * nnz + 48 * nV, flops=2 * nnz)
    if kind == "newton":
        return dict(bytes=112 * nT + 48 * nV, flops=1200 * nT + 2 * nnz)
    # the network's node layers forward and backward, and every Hessian entry once
    return dict(bytes=4 * nnz, flops=3 * 2 * 64 * (3 * (128 + 128) + 128) * nV)


# ------------------------------------------------------------------- exact ---
def exact(case, seed):
    kind = case["kind"]
    if kind in ("newton", "train"):
        return None
    if kind == "packed":
        V, E, _, _ = _pack(case["count"], case["nmin"], case["nmax"], seed)
        pat, r, h, young = _Pattern(len(V), E), np.random.default_rng(seed), 1.0 / case["nmax"], 2e6
    else:
        V, E, h, r = _geometry(case, seed)
        if kind in ("solve", "direction"):
            pat, young = _pattern(case["shape"], case["nx"], case["ny"], case["nz"]), case["young"]
    if kind in ("packed", "solve", "direction"):
        values, b, pinned, _ = _system(pat, V, h, young, r)
        A = pat.csr(values.double())
        free = _dev(np.repeat(~pinned, 3).astype(np.float64))
        nb = 3 * (pat.rb[1:] - pat.rb[:-1])
        diag_block = torch.searchsorted(pat.keys, torch.arange(len(V), device="cuda") * (len(V) + 1)) - pat.rb[:-1]
        at = (9 * pat.rb[:-1] + 3 * diag_block)[:, None] + torch.arange(3, device="cuda") * (nb[:, None] + 1)
        x = _cg64(A, 1.0 / values.double()[at.reshape(-1)], _dev(b), free)
        if kind == "direction":
            return dict(d=-x[free > 0], ok=None)
        return dict(x=x, ok=None)
    params = _params(case["model"], len(E), 1e6, r)
    q = _deformed(V, h, case["strain"], r)
    if kind == "hessian":
        pat = _pattern(case["shape"], case["nx"], case["ny"], case["nz"])
        return dict(values=_assemble(pat, V, q, params, case["model"], 1e-6 if case["psd"] else None, DT * DT, 1.0))
    Vg, Eg, qg, p = _dev(V), _dev(E).long(), _dev(q), _dev(params)
    energy, g = torch.zeros((), dtype=torch.float64, device="cuda"), torch.zeros_like(qg)
    for t0 in range(0, len(E), 500000):
        e = Eg[t0:t0 + 500000]
        phi, vol = _grads(Vg, e)
        psi, P = _psi_pk1(case["model"], _def_grad(qg, e, phi), p[t0:t0 + 500000])
        energy += (psi * vol).sum()
        ge = torch.einsum("tki,tai->tak", P, phi) * vol[:, None, None]
        g.index_add_(0, e.reshape(-1), ge.reshape(-1, 3))
    if kind == "dropin":
        return dict(energy=energy, gradient=g.reshape(-1))
    return dict(energy=energy.reshape(1), gradient=g.reshape(-1))
