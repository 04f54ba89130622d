"""A batch's plan holds no layout of its union as one mesh, whether it is made
in one call (mfem_plan_create_bodies) or by mfem_plan_set_bodies on a plan.

What the resident PCG adds to a batch's plan is its lists, per block of H 4
bytes of slot and 2 of column, padded to whole slices (by less than a half),
and per vertex some 80 bytes of rows, halos and destinations.  The union's
lists would be as many again, and a buffer for the blocks that do not fit on
the chip beside them (28 MB in all for 48,683 vertices, against 6)."""
import ctypes

import numpy as np
import pytest
import torch

from mfem_gb300 import Model, MixedFEMSolver, _lib, beams
from mfem_gb300.batched import BatchedSolver

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def two_calls(batch, model, **kw):
    u = batch.union
    solver = MixedFEMSolver(model, iterations=1, line_search=False, cg_tolerance=u.spec.cg_tolerance, **kw)
    h = dict(voff=np.ascontiguousarray(batch.vertex_offsets, dtype=np.int32),
             toff=np.ascontiguousarray(batch.tet_offsets, dtype=np.int32),
             energy=np.array([_lib.ENERGY[e] for e in batch.energies], dtype=np.int32),
             gravity=np.ascontiguousarray(batch.gravity, dtype=np.float32))
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    _lib.check(solver._lib.mfem_plan_set_bodies(solver._plan, batch.n_bodies, P(h["voff"]), P(h["toff"]), P(h["energy"]),
                                                P(h["gravity"])), solver._plan)
    return solver


@pytest.mark.parametrize("calls", ["one", "two"])
def test_a_batch_holds_no_layout_of_its_union(calls):
    batch = beams.batched_bodies(40, seed=4, nx=(12, 24), nyz=(5, 9))
    u = batch.union
    assert 40000 <= u.n <= 60000
    model = Model(u.rest_q, np.zeros_like(u.rest_q), u.particle_mass, u.particle_inv_mass, u.tet_indices, u.tet_poses,
                  u.tet_materials, u.gravity, device=DEV)

    def make(**kw):
        if calls == "two":
            return two_calls(batch, model, **kw)
        return BatchedSolver(batch, device=DEV, **kw).solver

    make()  # what the first plan of a process loads
    sizes = {}
    for variant in ("standard", "auto"):
        keep = make(pcg_variant=variant)
        before = used()
        keep.close()
        del keep
        sizes[variant] = before - used()
    solver = make()
    nnzb = solver.nnzb
    lists = 9 * nnzb + 80 * u.n
    assert sizes["auto"] - sizes["standard"] <= lists + (4 << 20), (sizes, lists)


def test_refused_bodies_stay_refused():
    batch = beams.batched_bodies(3, seed=1, nx=(2, 4), nyz=(1, 2))
    bad = beams.batched_bodies(3, seed=1, nx=(2, 4), nyz=(1, 2))
    bad.vertex_offsets = np.array([0, 1, 2, bad.union.n])
    with pytest.raises(_lib.MfemError) as err:
        BatchedSolver(bad, device=DEV)
    assert err.value.code == _lib.MFEM_BAD_ARG and "another body" in str(err.value)
    with pytest.raises(_lib.MfemError):
        BatchedSolver(batch, device=DEV, solver_precision="fp16")
    with pytest.raises(_lib.MfemError):
        BatchedSolver(beams.batched_bodies(1, seed=1, nx=(2, 4), nyz=(1, 2)), device=DEV, solver_precision="fp16")
