"""What a user of this framework has it do, as cases that can be timed: implicit-Euler steps of soft bodies through
``MixedFEMSolver.step`` and ``BatchedSolver.step``, and the assembly of one Newton system through the solver's stage
calls.  Sizes run from the 240-tet cantilever to the 786,432-tet beam of ``beams.CONFIGS``; ``draw`` gives more of the
same ranges.

A state is a model with its solver (the plan a program keeps) and one moment of a motion: positions perturbed as the
configs perturb them, and a smooth swing of about 1 m/s with some noise, as a body in the middle of a simulation has.
One pass takes the step from that moment (``state_in`` is only read); s and lambda persist in the solver, as in a
program that steps it.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "warp-mfem_gb300"))

from mfem_gb300 import MixedFEMSolver, Model, beams  # noqa: E402
from mfem_gb300.batched import BatchedSolver  # noqa: E402

DEVICE = "cuda:0"
DT = 1.0 / 60.0
GRAVITY = (0.0, -9.81, 0.0)

# A step of one body; the defaults are the benchmark's (plain update, fp32 block-Jacobi PCG, 8 Newton iterations).
STEP = dict(kind="step", nx=64, ny=16, nz=16, cell=0.03125, energy="neohookean", e_hi=1.0e6, order="grid",
            preconditioner="block_jacobi", precision="fp32", iterations=8, line_search=False, contact=False)
ASSEMBLE = dict(kind="assemble", nx=96, ny=25, nz=23, cell=0.03125, energy="neohookean", e_hi=1.0e6, order="grid")
BATCH = dict(kind="batch", bodies=96, shape_seed=4, preconditioner="block_jacobi", iterations=8)


def listed():
    return [
        # the small ARAP cantilever: an interactive toy, where latency counts
        dict(STEP, name="cantilever_arap", nx=10, ny=2, nz=2, cell=0.1, energy="arap", e_hi=1.0e4),
        # a coarse character on the ground: unordered vertices, barrier contact with friction, the default line search
        dict(STEP, name="coarse_contact", nx=12, ny=6, nz=6, order="shuffled", line_search=True, contact=True,
             iterations=3),
        # a mid-size body
        dict(STEP, name="beam_12k", nx=32, ny=8, nz=8),
        # the benchmark's beam, the reference's solve
        dict(STEP, name="nh_beam"),
        # the same with the factorised approximate inverse, refreshed once a step
        dict(STEP, name="nh_beam_fsai", preconditioner="fsai"),
        # a mesh as a generator numbers it, in no banded order
        dict(STEP, name="unordered_38k", nx=44, ny=13, nz=11, order="shuffled"),
        # 16-bit blocks and the learned factor inside the fp64 refinement
        dict(STEP, name="learned_fp16", nx=40, ny=11, nz=10, preconditioner="learned", precision="fp16"),
        # fp32 blocks inside the fp64 refinement, an odd size
        dict(STEP, name="refined_fp32", nx=49, ny=12, nz=13, precision="fp32_refined"),
        # the largest mesh, its stiffness spread over three decades
        dict(STEP, name="stiff_beam", nx=128, ny=32, nz=32, e_hi=1.0e7),
        # one Newton system of a large mesh: element terms, H, rhs and block-Jacobi
        dict(ASSEMBLE, name="assemble_331k"),
        # many uneven bodies in one plan
        dict(BATCH, name="batch_96"),
        # a few bodies, with the factorised approximate inverse
        dict(BATCH, name="batch_20_fsai", bodies=20, shape_seed=9, preconditioner="fsai"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, most_tets):
    """A beam of 240 tets or more, 2 to 5 times as long as high, ragged cross sections."""
    tets = math.exp(rng.uniform(math.log(240.0), math.log(most_tets)))
    aspect = rng.uniform(2.0, 5.0)
    side = (tets / 6.0 / aspect) ** (1.0 / 3.0)
    ny = max(2, int(round(side * rng.uniform(0.85, 1.18))))
    nz = max(2, int(round(side * rng.uniform(0.85, 1.18))))
    nx = max(3, min(int(tets / 6.0 / (ny * nz)), 5 * min(ny, nz)))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    pick = rng.random()
    if pick < 0.12:
        return dict(ASSEMBLE, energy=rng.choice(["neohookean", "arap"]), order=rng.choice(["grid", "shuffled"]),
                    **_cells(rng, 3.3e5))
    if pick < 0.30:
        return dict(BATCH, bodies=_log_int(rng, 4, 96), shape_seed=rng.randrange(1000),
                    preconditioner=rng.choice(["block_jacobi", "block_jacobi", "fsai"]))
    case = dict(STEP, energy=rng.choice(["neohookean", "neohookean", "arap"]), e_hi=rng.choice([1.0e5, 1.0e6, 1.0e7]))
    solve = rng.random()
    if solve < 0.55:
        case.update(_cells(rng, 6.0e5), order=rng.choice(["grid", "grid", "shuffled"]))
    elif solve < 0.75:
        case.update(_cells(rng, 2.0e5), preconditioner=rng.choice(["fsai", "fsai", "learned"]))
    else:
        case.update(_cells(rng, 1.0e5), precision=rng.choice(["fp16", "fp32_refined", "fp32_refined"]),
                    preconditioner=rng.choice(["block_jacobi", "fsai", "learned"]), e_hi=1.0e6)
    if case["precision"] == "fp32" and rng.random() < 0.35:
        case.update(line_search=True, iterations=3, contact=rng.random() < 0.5)
    return case


# -- inputs -----------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _grid(nx, ny, nz, cell):
    """The mesh of a beam without its materials: what a program loads once."""
    spec = beams.BeamSpec(name="beam", cells=(nx, ny, nz), extent=(nx * cell, ny * cell, nz * cell), energy="arap",
                          E=(1.0e4, 1.0e4), nu=0.45)
    return beams.build_beam(spec)


@functools.lru_cache(maxsize=2)
def _bodies(count, shape_seed):
    return beams.batched_bodies(n_bodies=count, seed=shape_seed)


def _swing(rest, free, rng, noise):
    """A smooth velocity field of about 1 m/s, growing from the clamped end, with noise on it."""
    x = (rest - rest.min(0)) / max(float(np.ptp(rest, axis=0).max()), 1e-9)
    v = np.empty_like(x)
    for a in range(3):
        v[:, a] = 1.4 * np.sin(x @ rng.normal(0.0, 2.0, 3) + rng.uniform(0.0, 6.0))
    v *= np.minimum(1.0, 3.0 * x[:, :1])
    return (v + rng.normal(0.0, noise, x.shape)) * free[:, None]


def _inputs(case, seed):
    """Host arrays of one case: rest, tets, poses, materials, masses, (q, qd), energies per tet, gravity."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 17])
    f32 = np.float32
    if case["kind"] == "batch":
        batch = _bodies(case["bodies"], case["shape_seed"])
        m = batch.union
        rest = m.rest_q.astype(np.float64)
        free = m.particle_inv_mass > 0
        v = np.concatenate([_swing(rest[a:b], free[a:b], rng, 0.05)
                            for a, b in zip(batch.vertex_offsets[:-1], batch.vertex_offsets[1:])])
        mat = m.tet_materials.copy()
        mat[:, :2] *= np.exp(rng.uniform(-0.5, 0.5, (m.T, 1))).astype(f32)
        per_tet = np.diff(batch.tet_offsets)
        q = rest + rng.normal(0.0, 1.0e-3, rest.shape) * free[:, None]
        return dict(rest=m.rest_q, tets=m.tet_indices, poses=m.tet_poses, mat=mat, mass=m.particle_mass,
                    inv_mass=m.particle_inv_mass, q=q.astype(f32), qd=v.astype(f32),
                    arap=np.repeat([e == "arap" for e in batch.energies], per_tet),
                    gravity=np.repeat(batch.gravity, np.diff(batch.vertex_offsets), axis=0), batch=batch)
    m = _grid(case["nx"], case["ny"], case["nz"], case["cell"])
    lo, hi = 1.0e4, case["e_hi"]  # log-uniform per tet; the cantilever's material is constant
    E = np.exp(rng.uniform(math.log(lo), math.log(hi), m.T)) if hi > lo else np.full(m.T, 1.0e5)
    mu, lam = beams.lame(E, 0.45)
    free = m.particle_inv_mass > 0
    rest = m.rest_q.astype(np.float64)
    v = _swing(rest, free, rng, 0.05)
    q = rest + rng.normal(0.0, 0.03 * case["cell"], rest.shape) * free[:, None]
    tets = m.tet_indices
    arrays = dict(rest=m.rest_q, mass=m.particle_mass, inv_mass=m.particle_inv_mass, q=q.astype(f32),
                  qd=v.astype(f32))
    if case["order"] == "shuffled":
        p = np.random.default_rng(m.n).permutation(m.n)  # the mesh's own numbering: the same for every seed
        new = np.empty(m.n, dtype=np.int32)
        new[p] = np.arange(m.n, dtype=np.int32)
        tets = new[tets]
        arrays = {k: np.ascontiguousarray(a[p]) for k, a in arrays.items()}
    return dict(arrays, tets=tets, poses=m.tet_poses, mat=np.stack([mu, lam, 0 * mu], axis=1).astype(f32),
                arap=np.full(m.T, case["energy"] == "arap"), gravity=np.asarray(GRAVITY, f32))


# a ground plane that the body's lower side reaches into, as in a drop
CONTACT = dict(contact_d0=1.0e-3, contact_d1=2.0e-2, contact_stiffness=1.0e3, friction_mu=0.3, friction_eps_v=1.0e-2)
PLANE_Y = -0.012


def prepare(case, seed):
    d = _inputs(case, seed)
    dev = torch.device(DEVICE)
    t = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    if case["kind"] == "batch":
        import dataclasses
        batch = d["batch"]
        batch = dataclasses.replace(batch, union=dataclasses.replace(batch.union, tet_materials=d["mat"]))
        solver = BatchedSolver(batch, device=DEVICE, preconditioner=_preconditioner(case), factor_refresh=8,
                               iterations=case["iterations"])
        s_in, s_out = solver.state(), solver.state()
    else:
        model = Model(d["rest"], np.zeros_like(d["rest"]), d["mass"], d["inv_mass"], d["tets"], d["poses"], d["mat"],
                      d["gravity"], device=DEVICE)
        kw = dict(energy=case["energy"], line_search=case.get("line_search", False))
        if case.get("contact"):
            h = math.sqrt(0.5)
            model.add_shape_plane((0.0, PLANE_Y, 0.0, -h, 0.0, 0.0, h))  # normal along +y
            kw.update(CONTACT)
        if case["kind"] == "step":
            kw.update(preconditioner=_preconditioner(case), factor_refresh=8, solver_precision=case["precision"],
                      inner_tolerance=1.0e-2, outer_tolerance=1.0e-6)
        solver = MixedFEMSolver(model, iterations=case.get("iterations", 8), **kw)
        s_in, s_out = model.state(), model.state()
    s_in.particle_q.copy_(t(d["q"]))
    s_in.particle_qd.copy_(t(d["qd"]))
    if case["kind"] == "assemble":
        solver.predict(s_in.particle_q, s_in.particle_qd, DT)
        s_out.particle_q.copy_(s_in.particle_q + 0.5 * DT * s_in.particle_qd)  # where a Newton iteration stands
    return dict(kind=case["kind"], solver=solver, s_in=s_in, s_out=s_out)


def _preconditioner(case):
    return True if case["preconditioner"] == "block_jacobi" else case["preconditioner"]


def run(state):
    solver, s_in, s_out = state["solver"], state["s_in"], state["s_out"]
    if state["kind"] == "assemble":
        solver.update_system(s_out.particle_q)
        solver.assemble(s_out.particle_q, DT)
        return {"h": solver.read_buffer("h_values"), "rhs": solver.read_buffer("rhs"),
                "precond": solver.read_buffer("precond")}
    if state["kind"] == "batch":
        solver.step(s_in, s_out, DT)
        return {"q": s_out.particle_q, "qd": s_out.particle_qd, "s": solver.solver.tet_stretch}
    solver.step(s_in, s_out, None, None, DT)
    return {"q": s_out.particle_q, "qd": s_out.particle_qd, "s": solver.tet_stretch}


# -- work -------------------------------------------------------------------
def _sizes(nx, ny, nz):
    """(vertices, tets, blocks of H) of a beam of nx x ny x nz cells of six tets."""
    n = (nx + 1) * (ny + 1) * (nz + 1)
    edges = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    edges += nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz
    return n, 6 * nx * ny * nz, n + 2 * edges


def work(case):
    if case["kind"] == "batch":
        sizes = [_sizes(*m.spec.cells) for m in _bodies(case["bodies"], case["shape_seed"]).bodies]
        n, T, nnzb = (sum(s[k] for s in sizes) for k in range(3))
    else:
        n, T, nnzb = _sizes(case["nx"], case["ny"], case["nz"])
    tet = 16 + 36 + 12 + 24  # vertex indices, inverse pose, material, s
    if case["kind"] == "assemble":
        return {"bytes": tet * T + 24 * n + (36 * nnzb + 12 * n + 36 * n), "flops": 5500.0 * T}
    # a Newton iteration: the tet data once, s and lambda out, H written and read once, the vectors; the PCG's operations
    # at a typical iteration count of each preconditioner
    its = {"block_jacobi": 350, "fsai": 150, "learned": 180}[case["preconditioner"]]
    K = case["iterations"]
    return {"bytes": K * ((tet + 48) * T + 76 * nnzb + 60 * n) + 48.0 * n,
            "flops": K * (5500.0 * T + its * (18.0 * nnzb + 40.0 * n))}


# -- the same in 64 bits ------------------------------------------------------
def _mat(s):
    return torch.stack([s[:, 0], s[:, 3], s[:, 4], s[:, 3], s[:, 1], s[:, 5], s[:, 4], s[:, 5], s[:, 2]], 1).view(-1, 3, 3)


def _sym(M):
    return torch.stack([M[..., 0, 0], M[..., 1, 1], M[..., 2, 2], M[..., 0, 1], M[..., 0, 2], M[..., 1, 2]], -1)


def _polar(F):
    """U, sigma, V of F = U diag(sigma) V^T with U V^T a rotation (the sign on the smallest sigma)."""
    U, sig, Vh = torch.linalg.svd(F)
    V = Vh.transpose(1, 2).clone()
    flip_u, flip_v = torch.linalg.det(U), torch.linalg.det(V)
    U[:, :, 2] *= torch.sign(flip_u)[:, None]
    V[:, :, 2] *= torch.sign(flip_v)[:, None]
    sig = sig.clone()
    sig[:, 2] *= torch.sign(flip_u * flip_v)
    return U, sig, V


def _constraint(x, tets, poses, s):
    """c = SYM (sym6 S(F) - s) and G = -dc/dx [T, 6, 12]."""
    xe = x[tets]
    F = torch.stack([xe[:, 1] - xe[:, 0], xe[:, 2] - xe[:, 0], xe[:, 3] - xe[:, 0]], 2) @ poses
    U, sig, V = _polar(F)
    S = V @ torch.diag_embed(sig) @ V.transpose(1, 2)
    two = torch.tensor([1.0, 1, 1, 2, 2, 2], dtype=x.dtype, device=x.device)
    grads = torch.cat([-poses.sum(1, keepdim=True), poses], 1)  # dF[i, :] = grads[k] for dx_k along i
    G = torch.empty(len(tets), 6, 12, dtype=x.dtype, device=x.device)
    pair = (sig[:, :, None] + sig[:, None, :]).clamp_min(1e-8)
    for k in range(4):
        b = torch.einsum("tj,tjm->tm", grads[:, k], V)
        for a in range(3):
            A = U[:, a, :, None] * b[:, None, :]  # U^T dF V
            W = (A - A.transpose(1, 2)) / pair
            G[:, :, 3 * k + a] = -two * _sym(V @ (A - W * sig[:, None, :]) @ V.transpose(1, 2))
    return two * (_sym(S) - s), G


def _gmw81(H):
    """The positive definite modification of H (modified Cholesky of Gill, Murray and Wright, 1981, as the reference
    writes it) and its inverse."""
    A = [[H[:, i, j] for j in range(6)] for i in range(6)]
    eps = 1.19e-7
    gamma = torch.stack([A[i][i].abs() for i in range(6)]).amax(0)
    xi = torch.stack([A[i][j].abs() for i in range(6) for j in range(i + 1, 6)]).amax(0)
    beta2 = torch.maximum(gamma, torch.maximum(xi / math.sqrt(35.0), torch.full_like(xi, eps)))
    for j in range(6):
        theta = torch.zeros_like(xi)
        for i in range(j + 1, 6):
            c = A[j][i]
            for k in range(j):
                c = c - A[k][k] * A[k][k] * A[i][k] * A[j][k]
            A[i][j] = c
            theta = torch.maximum(theta, c.abs())
        d = torch.maximum(torch.maximum(A[j][j].abs(), theta * theta / beta2), torch.full_like(xi, math.sqrt(eps)))
        A[j][j] = torch.sqrt(d)
        for i in range(j + 1, 6):
            c = A[i][j]
            A[i][j] = c / d
            A[i][i] = A[i][i] - c * c / d
    zero = torch.zeros_like(xi)
    L = torch.stack([torch.stack([A[i][j] * A[j][j] if j < i else A[i][i] if i == j else zero for j in range(6)], 1)
                     for i in range(6)], 1)
    fixed = L @ L.transpose(1, 2)
    return fixed, torch.linalg.inv(fixed)


def _elastic(s, mat, vol, arap):
    """Energy, gradient, Hessian and its inverse in s (ARAP where `arap`, else Neo-Hookean)."""
    mu, lam = mat[:, 0], mat[:, 1]
    two = torch.tensor([1.0, 1, 1, 2, 2, 2], dtype=s.dtype, device=s.device)
    one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=s.dtype, device=s.device)
    s0, s1, s2, s3, s4, s5 = s.unbind(1)
    off2 = 2.0 * (s3 * s3 + s4 * s4 + s5 * s5)
    eye = torch.diag(two)[None]
    e_a = vol * mu * (s0 * s1 + s1 * s2 + s2 * s0 + off2 + 3.0 - 2.0 * (s0 + s1 + s2)) / 2.0
    g_a = (vol * mu)[:, None] * (two * s - one)
    H_a = (vol * mu)[:, None, None] * eye
    if bool(arap.all()):
        return e_a, g_a, H_a, torch.linalg.inv(H_a)
    J = s0 * s1 * s2 + 2.0 * s3 * s4 * s5 - (s1 * s4 * s4 + s0 * s5 * s5 + s2 * s3 * s3)
    gJ = torch.stack([s1 * s2 - s5 * s5, s0 * s2 - s4 * s4, s0 * s1 - s3 * s3, 2 * (s4 * s5 - s2 * s3),
                      2 * (s3 * s5 - s1 * s4), 2 * (s3 * s4 - s0 * s5)], 1)
    z = torch.zeros_like(s0)
    hJ = torch.stack([torch.stack(r, 1) for r in (
        (z, s2, s1, z, z, -2 * s5), (s2, z, s0, z, -2 * s4, z), (s1, s0, z, -2 * s3, z, z),
        (z, z, -2 * s3, -2 * s2, 2 * s5, 2 * s4), (z, -2 * s4, z, 2 * s5, -2 * s1, 2 * s3),
        (-2 * s5, z, z, 2 * s4, 2 * s3, -2 * s0))], 1)
    e_n = vol * (mu * (s0 * s0 + s1 * s1 + s2 * s2 + off2 - 3.0) / 2.0 - mu * (J - 1.0) + lam / 2.0 * (J - 1.0) ** 2)
    k = lam * (J - 1.0) - mu
    g_n = vol[:, None] * (mu[:, None] * two * s + k[:, None] * gJ)
    H_n, inv_n = _gmw81(vol[:, None, None] * (mu[:, None, None] * eye + lam[:, None, None] * gJ[:, :, None] * gJ[:, None]
                                              + k[:, None, None] * hJ))
    w = arap[:, None, None]
    return (torch.where(arap, e_a, e_n), torch.where(arap[:, None], g_a, g_n), torch.where(w, H_a, H_n),
            torch.where(w, torch.linalg.inv(H_a), inv_n))


class _Exact:
    """One body (or a union of bodies) in float64."""

    def __init__(self, case, seed):
        d = _inputs(case, seed)
        dev = torch.device(DEVICE if torch.cuda.is_available() else "cpu")
        f = lambda a: torch.as_tensor(np.asarray(a), device=dev).to(torch.float64)  # noqa: E731
        self.case, self.tets = case, torch.as_tensor(d["tets"], device=dev).long()
        self.rest, self.poses, self.mat, self.mass = f(d["rest"]), f(d["poses"]), f(d["mat"]), f(d["mass"])
        self.q, self.qd, self.gravity = f(d["q"]), f(d["qd"]), f(d["gravity"])
        self.arap = torch.as_tensor(d["arap"], device=dev)
        inv_mass = f(d["inv_mass"])
        self.pinned = inv_mass == 0
        self.h_mass = torch.where(self.pinned, torch.ones_like(inv_mass), 1.0 / inv_mass)
        self.attach = torch.where(self.pinned, torch.full_like(inv_mass, 10.0), torch.zeros_like(inv_mass))
        self.vol = 1.0 / (6.0 * torch.linalg.det(self.poses))
        self.two = torch.tensor([1.0, 1, 1, 2, 2, 2], dtype=torch.float64, device=dev)
        n = self.n = len(self.rest)
        self.s = torch.zeros(len(self.tets), 6, dtype=torch.float64, device=dev)
        self.s = _constraint(self.rest, self.tets, self.poses, self.s)[0] / self.two
        self.lam = torch.zeros_like(self.s)
        r = self.tets[:, :, None].expand(-1, 4, 4).reshape(-1)
        c = self.tets[:, None, :].expand(-1, 4, 4).reshape(-1)
        diag = torch.arange(n, device=dev) * (n + 1)
        keys = torch.unique(torch.cat([r * n + c, diag]))
        self.slots = torch.searchsorted(keys, r * n + c)
        self.diag = torch.searchsorted(keys, diag)
        self.rows, self.cols = keys // n, keys % n
        deg = torch.bincount(self.rows, minlength=n)
        rp = torch.cat([torch.zeros(1, dtype=torch.long, device=dev), deg.cumsum(0)])
        k = torch.arange(len(keys), device=dev) - rp[self.rows]
        a3 = torch.arange(3, device=dev)
        self.place = ((9 * rp[self.rows] + 3 * k)[:, None, None] + (3 * deg[self.rows])[:, None, None] * a3[:, None]
                      + a3[None, :]).reshape(-1)
        self.crow = torch.cat([torch.zeros(1, dtype=torch.long, device=dev),
                               (3 * deg).repeat_interleave(3).cumsum(0)])
        self.ccol = torch.empty(9 * len(keys), dtype=torch.long, device=dev)
        self.ccol[self.place] = (3 * self.cols[:, None, None] + a3[None, None, :]).expand(-1, 3, 3).reshape(-1)
        self.start = None

    def kinetic(self, x):
        return (self.mass[:, None] * (x - self.x_tilde) + self.attach[:, None] * (x - self.rest)) / (DT * DT)

    def contact(self, x):
        """Energy, gradient and diagonal blocks of the plane's barrier and the lagged friction."""
        d0, d1, kc = CONTACT["contact_d0"], CONTACT["contact_d1"], CONTACT["contact_stiffness"]

        def log_barrier(d):
            l = torch.log(d / d1)
            return (-(d - d1) ** 2 * l, -(2 * (d - d1) * l + (d - d1) ** 2 / d),
                    -(2 * l + 4 * (d - d1) / d - (d - d1) ** 2 / d ** 2))

        def barrier(d):
            out = log_barrier(d.clamp(d0, d1))
            b, db, ddb = (float(v) for v in log_barrier(torch.tensor(d0, dtype=torch.float64)))
            low = d <= d0
            ext = (b + db * (d - d0) + 0.5 * ddb * (d - d0) ** 2, db + ddb * (d - d0), torch.full_like(d, ddb))
            return [torch.where(d >= d1, torch.zeros_like(d), torch.where(low, e, o)) for e, o in zip(ext, out)]

        normal = torch.tensor([0.0, 1.0, 0.0], dtype=x.dtype, device=x.device)
        e, de, dde = barrier(x[:, 1] - PLANE_Y)
        force = kc * (-barrier(self.start[:, 1] - PLANE_Y)[1]).clamp_min(0.0)
        ev, scale = CONTACT["friction_eps_v"] * DT, CONTACT["friction_mu"] * force
        u = x - self.start
        ut = u - u[:, 1:2] * normal
        y = ut.norm(dim=1)
        slide = y >= ev
        f0 = torch.where(slide, y, -y ** 3 / (3 * ev * ev) + y * y / ev + ev / 3)
        f1 = torch.where(slide, 1.0 / y.clamp_min(1e-12), -y / (ev * ev) + 2 / ev)
        nn = normal[:, None] * normal[None, :]
        block = (kc * dde.clamp_min(0.0))[:, None, None] * nn + (scale * f1)[:, None, None] * (
            torch.eye(3, dtype=x.dtype, device=x.device) - nn)
        on = scale > 0
        return ((kc * e).sum() + (scale * f0)[on].sum(), (kc * de)[:, None] * normal + (scale * f1)[:, None] * ut, block)

    def terms(self, x):
        c, G = _constraint(x, self.tets, self.poses, self.s)
        _, g_s, H_s, inv = _elastic(self.s, self.mat, self.vol, self.arap)
        H_l = H_s / (self.two[:, None] * self.two[None, :])
        g_l = c + self.two * torch.einsum("tij,tj->ti", inv, g_s)
        return c, G, g_s, inv, H_l, g_l

    def assemble(self, x, el):
        _, G, _, _, H_l, g_l = el
        P = H_l @ G
        K = (G.transpose(1, 2) @ P).view(-1, 4, 3, 4, 3).permute(0, 1, 3, 2, 4).reshape(-1, 3, 3)
        H = torch.zeros(len(self.rows), 3, 3, dtype=x.dtype, device=x.device).index_add_(0, self.slots, K)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        H[self.diag] += ((self.h_mass + self.attach) / (DT * DT))[:, None, None] * eye
        g = torch.zeros_like(x).index_add_(0, self.tets.reshape(-1), torch.einsum("tji,tj->ti", P, g_l).reshape(-1, 3))
        g = g - self.kinetic(x)
        if self.case.get("contact"):
            _, gc, Hc = self.contact(x)
            H[self.diag] += Hc
            g = g - gc
        return H, g

    def solve(self, H, g, minv):
        vals = torch.empty(9 * len(H), dtype=H.dtype, device=H.device)
        vals[self.place] = H.reshape(-1)
        A = torch.sparse_csr_tensor(self.crow, self.ccol, vals, (3 * self.n, 3 * self.n))
        M = lambda r: (minv @ r.view(-1, 3, 1)).reshape(-1)  # noqa: E731
        r = g.reshape(-1).clone()
        x, z = torch.zeros_like(r), M(r)
        p, rz, stop = z, r @ z, 1e-20 * float(r @ r)
        for it in range(6000):
            Ap = A @ p
            alpha = rz / (p @ Ap)
            x, r = x + alpha * p, r - alpha * Ap
            if it % 16 == 15 and float(r @ r) <= stop:
                break
            z = M(r)
            rz, old = r @ z, rz
            p = z + (rz / old) * p
        return x.view(-1, 3)

    def merit(self, x, s):
        dx, at = x - self.x_tilde, x - self.rest
        f = (0.5 * (self.mass * (dx * dx).sum(1)).sum() + 0.5 * (self.attach * (at * at).sum(1)).sum()) / (DT * DT)
        xe = x[self.tets]
        F = torch.stack([xe[:, 1] - xe[:, 0], xe[:, 2] - xe[:, 0], xe[:, 3] - xe[:, 0]], 2) @ self.poses
        _, sig, V = _polar(F)
        c = self.two * (_sym(V @ torch.diag_embed(sig) @ V.transpose(1, 2)) - s)
        f = f + (_elastic(s, self.mat, self.vol, self.arap)[0] - (c * self.lam).sum(1)).sum()
        return float(f + self.contact(x)[0] if self.case.get("contact") else f)

    def search(self, x, el, dx, ds):
        """The backtracking search: Armijo on the merit, steps halved, at most 20 trials."""
        g = self.kinetic(x)
        GtL = torch.zeros_like(x).index_add_(0, self.tets.reshape(-1),
                                             torch.einsum("tik,ti->tk", el[1], self.lam).reshape(-1, 3))
        g = g - GtL
        if self.case.get("contact"):
            g = g + self.contact(x)[1]
        t = -0.01 * float((g * dx).sum() + ((el[2] + self.two * self.lam) * ds).sum())
        f0, alpha, j = self.merit(x, self.s), 1.0, 0
        while True:
            f1 = self.merit(x + alpha * dx, self.s + alpha * ds)
            more = (f0 - f1) + 1e-8 < alpha * t and j < 20
            j += 1
            if not more:
                break
            alpha *= 0.5
        return (x + alpha * dx, self.s + alpha * ds) if j < 20 else (x, self.s)

    def predict(self):
        self.x_tilde = self.q + DT * self.qd + 0.5 * DT * DT * self.gravity
        self.start = self.q

    def step(self):
        self.predict()
        x = self.q
        for _ in range(self.case["iterations"]):
            el = self.terms(x)
            H, g = self.assemble(x, el)
            dx = self.solve(H, g, torch.linalg.inv(H[self.diag]))
            _, G, g_s, inv, H_l, g_l = el
            Gdx = torch.einsum("tij,tj->ti", G, dx[self.tets].reshape(-1, 12))
            self.lam = -torch.einsum("tij,tj->ti", H_l, g_l - Gdx)
            ds = -torch.einsum("tij,tj->ti", inv, self.two * self.lam + g_s)
            if self.case.get("line_search"):
                x, self.s = self.search(x, el, dx, ds)
            else:
                x, self.s = x + dx, self.s + ds
        return {"q": x, "qd": (x - self.q) / DT, "s": self.s}


def exact(case, seed):
    e = _Exact(case, seed)
    if case["kind"] != "assemble":
        return e.step()
    e.predict()
    # the point is what prepare() hands over, in float32
    x = (e.q.float() + 0.5 * DT * e.qd.float()).double()
    H, g = e.assemble(x, e.terms(x))
    return {"h": H.reshape(-1), "rhs": g.reshape(-1), "precond": torch.linalg.inv(H[e.diag]).reshape(-1)}
