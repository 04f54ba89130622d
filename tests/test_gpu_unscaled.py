"""Solves without a preconditioner (or with every block below the singular
threshold, so that it is the identity) on stiffly attached bodies: they keep the
standard recurrence where they had it, batches and meshes without a windowed
single-reduction layout, and converge as the forms that explicit settings
select do."""
import dataclasses

import numpy as np
import pytest
import torch

from mfem_gb300 import _lib, beams
from mfem_gb300.batched import BatchedSolver
from test_gpu_resident import shuffled
from test_gpu_resident_forms import DEV, solver_of

pytestmark = pytest.mark.gpu
IDENTITY = [dict(preconditioner=False), dict(preconditioner_singular_threshold=1e30)]


def moving(solver, q0, dt):
    q = torch.as_tensor(q0, device=DEV)
    x = q.clone()
    v = np.random.default_rng(7).normal(0.0, 0.3, q0.shape).astype(np.float32)
    solver.predict(q, torch.as_tensor(v, device=DEV), dt)
    solver.update_system(x)
    solver.assemble(x, dt)
    solver.global_solve(0)
    torch.cuda.synchronize()
    return solver.read_buffer("dx")


@pytest.mark.parametrize("kw", IDENTITY, ids=["none", "identity"])
@pytest.mark.parametrize("sizes", [dict(nx=(2, 5), nyz=(1, 2)), dict(nx=(6, 14), nyz=(2, 5))], ids=["one", "cluster"])
@pytest.mark.parametrize("seed", [1, 3])
def test_unscaled_bodies_converge(kw, sizes, seed):
    batch = beams.batched_bodies(8, seed=seed, **sizes)
    out = []
    for variant in ("auto", "global_memory"):
        bs = BatchedSolver(batch, device=DEV, iterations=1, cg_max_iterations=5000, attachment_stiffness=1e4,
                           pcg_variant=variant, **kw)
        out.append((moving(bs.solver, batch.union.q0, batch.dt), bs.body_stats()[0]))
    (xa, sa), (xb, sb) = out
    assert (sa["status"] == _lib.MFEM_OK).all(), sa
    assert (sa["iterations"] == sb["iterations"]).all() and torch.equal(xa, xb)


@pytest.mark.parametrize("kw", IDENTITY, ids=["none", "identity"])
def test_unscaled_shuffled_mesh_converges(kw):
    spec = dataclasses.replace(beams.CONFIGS["nh_beam"], cells=(40, 24, 20), E=(1e4, 1e5))
    mesh = shuffled(beams.build_beam(spec), seed=3)
    out = []
    for variant in ("auto", "gather"):
        solver = solver_of(mesh, cg_max_iterations=5000, attachment_stiffness=1e4, pcg_variant=variant, **kw)
        out.append((moving(solver, mesh.q0, mesh.spec.dt), solver.solve_stats()[0]))
    (xa, sa), (xb, sb) = out
    assert sa["status"] == _lib.MFEM_OK and sa["iterations"] == sb["iterations"], (sa, sb)
    assert torch.equal(xa, xb)
