"""Which form of the PCG a plan runs, and what the forms promise one another:
the resident form that a size selects, the ordered sums' equality with the
windowed kernel bit for bit, the retry after a factor's breakdown in every
scope, and the windowed and global-memory forms where explicit settings
select them."""
import numpy as np
import pytest
import torch

from mfem_gb300 import Model, MixedFEMSolver, _lib, beams, factor_net as F
from mfem_gb300.batched import BatchedSolver
from test_gpu_failure import run_steps
from test_gpu_resident import shuffled

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def windowed_ctas(mesh):
    """The CTAs of the default windowed plan: given explicitly they select it."""
    return min(sms(), -(-mesh.n // 64))


def first_system(solver, q0, dt):
    q = torch.as_tensor(q0, device=DEV)
    x = q.clone()
    solver.predict(q, torch.zeros_like(q), dt)
    solver.update_system(x)
    solver.assemble(x, dt)
    solver.global_solve(0)
    torch.cuda.synchronize()
    return solver.read_buffer("dx")


def solver_of(mesh, line_search=False, **kw):
    model = Model.from_beam(mesh, device=DEV)
    return MixedFEMSolver(model, iterations=kw.pop("iterations", 1), energy=mesh.spec.energy, line_search=line_search,
                          **kw)


def solve(mesh, **kw):
    solver = solver_of(mesh, **kw)
    return solver, first_system(solver, mesh.q0, mesh.spec.dt)


# -- the form a size selects ---------------------------------------------------
@pytest.mark.parametrize("cells,parts,cached", [
    ((8, 8, 5), 4, True), ((10, 8, 8), 8, True), ((16, 16, 6), 16, True), ((17, 12, 8), 16, True),
    ((16, 32, 10), -1, True), ((34, 33, 16), -1, True), ((64, 34, 34), -1, False)],
    ids=lambda c: "x".join(map(str, c)) if isinstance(c, tuple) else None)
@pytest.mark.parametrize("order", ["grid", "shuffled"])
def test_a_size_selects_its_resident_form(cells, parts, cached, order):
    mesh = beams.build_beam("nh_beam", cells=cells)
    assert mesh.n > 384
    if order == "shuffled":
        mesh = shuffled(mesh)
    lay = solver_of(mesh).pcg_layout()
    assert lay["ctas"] == (parts if parts > 0 else min(sms(), -(-mesh.n // 128))), lay
    assert lay["cache_matrix"] == cached, lay
    assert lay["smem_bytes"] != solver_of(mesh, pcg_ctas=windowed_ctas(mesh)).pcg_layout()["smem_bytes"]


@pytest.mark.parametrize("pc", ["block_jacobi", "fsai"])
def test_a_batch_runs_on_clusters(pc):
    batch = beams.batched_bodies(12, seed=3, nx=(2, 24), nyz=(1, 9))
    rows = np.diff(batch.vertex_offsets)
    lay = BatchedSolver(batch, device=DEV, preconditioner=pc).layout()
    assert lay["threads"] == 512 and lay["ctas"] >= int((-(-rows // 384)).sum()), lay
    assert BatchedSolver(batch, device=DEV, preconditioner=pc, pcg_variant="global_memory").layout()["threads"] < 512


# -- ordered sums: the windowed kernel's iterates ------------------------------
# one CTA of one and of two blocks, clusters of 3 to 16 CTAs with up to six
# blocks a CTA (one and two rows a thread), a grid
@pytest.mark.parametrize("cells", [(3, 2, 2), (6, 5, 2), (10, 4, 4), (16, 8, 8), (24, 11, 11), (50, 9, 9), (36, 12, 12),
                                   (64, 16, 16)], ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("precision", ["fp32", "fp32_refined"])
def test_ordered_sums_have_the_windowed_iterates(cells, precision):
    mesh = beams.build_beam("nh_beam", cells=cells)
    a, xa = solve(mesh, line_search=True, solver_precision=precision)
    b, xb = solve(mesh, line_search=True, solver_precision=precision, pcg_ctas=windowed_ctas(mesh))
    assert a.pcg_layout()["smem_bytes"] != b.pcg_layout()["smem_bytes"]  # two forms
    assert b.pcg_layout()["variant"] == "single_reduction" and b.pcg_layout()["cache_matrix"]
    assert a.solve_stats() == b.solve_stats()
    assert torch.equal(xa, xb)


@pytest.mark.parametrize("cells", [(3, 2, 2), (10, 4, 4)], ids=lambda c: "x".join(map(str, c)))
def test_ordered_sums_on_a_small_shuffled_mesh(cells):
    mesh = shuffled(beams.build_beam("nh_beam", cells=cells))
    a, xa = solve(mesh)
    b, xb = solve(mesh, pcg_ctas=windowed_ctas(mesh))
    assert a.solve_stats() == b.solve_stats() and torch.equal(xa, xb)


# -- a factor that breaks the PCG down -----------------------------------------
def overflowing_net():
    net = F.FactorNet()
    with torch.no_grad():
        net.diag.bias[:3] = 1.0e30  # softplus(1e30) = 1e30: M r overflows
    return net.pack()


@pytest.mark.parametrize("cells,order", [((10, 6, 5), "grid"), ((24, 13, 12), "shuffled"), ((34, 20, 17), "grid")],
                         ids=["462", "4550_shuffled", "13230"])
def test_breakdown_falls_back_to_block_jacobi_on_a_grid(cells, order):
    mesh = beams.build_beam("nh_beam", cells=cells)
    if order == "shuffled":
        mesh = shuffled(mesh)
    a, xa = solve(mesh, preconditioner="learned", factor_net_params=overflowing_net())
    b, xb = solve(mesh)
    sa, sb = a.solve_stats()[0], b.solve_stats()[0]
    assert a.pcg_layout()["smem_bytes"] > 0
    assert sa["status"] == _lib.MFEM_OK and abs(sa["iterations"] - sb["iterations"]) <= max(2, sb["iterations"] // 50)
    assert float((xa - xb).abs().max()) <= 1e-4 * float(xb.abs().max())


@pytest.mark.parametrize("sizes", [dict(nx=(2, 7), nyz=(1, 3)), dict(nx=(12, 24), nyz=(5, 9))], ids=["one", "cluster"])
def test_breakdown_falls_back_to_block_jacobi_in_a_batch(sizes):
    batch = beams.batched_bodies(6, seed=5, **sizes)
    out = []
    for kw in (dict(preconditioner="learned", factor_net_params=overflowing_net()), dict()):
        bs = BatchedSolver(batch, device=DEV, **kw)
        assert bs.layout()["threads"] == 512
        out.append((first_system(bs.solver, batch.union.q0, batch.dt), bs.body_stats()[0]))
    (xa, sa), (xb, sb) = out
    assert (sa["status"] == _lib.MFEM_OK).all() and (sb["status"] == _lib.MFEM_OK).all()
    assert (np.abs(sa["iterations"] - sb["iterations"]) <= np.maximum(2, sb["iterations"] // 50)).all(), (sa, sb)
    for k in range(6):
        o = slice(3 * batch.vertex_offsets[k], 3 * batch.vertex_offsets[k + 1])
        assert float((xa[o] - xb[o]).abs().max()) <= 1e-4 * float(xb[o].abs().max()), k


@pytest.mark.parametrize("precision", ["fp16", "fp32_refined"])
@pytest.mark.parametrize("cells,order", [((10, 6, 5), "grid"), ((24, 13, 12), "shuffled")], ids=["462", "4550_shuffled"])
def test_breakdown_of_an_inner_solve_falls_back_to_block_jacobi(precision, cells, order):
    mesh = beams.build_beam("nh_beam", cells=cells)
    if order == "shuffled":
        mesh = shuffled(mesh)
    kw = dict(solver_precision=precision, outer_tolerance=1e-6, inner_tolerance=1e-2)
    a, xa = solve(mesh, preconditioner="learned", factor_net_params=overflowing_net(), **kw)
    b, xb = solve(mesh, **kw)
    sa, sb = a.mixed_stats()[0], b.mixed_stats()[0]
    assert sa["status"] == _lib.MFEM_OK and sa["rel_residual"] <= 1e-6, sa
    if precision == "fp16":
        assert not sa["fp32_inner"], sa  # the retry comes before the switch to the fp32 blocks
    assert float((xa - xb).abs().max()) <= 1e-4 * float(xb.abs().max())


# -- what a refined factor solve solves -----------------------------------------
@pytest.mark.parametrize("precision", ["fp16", "bf16", "fp32_refined"])
@pytest.mark.parametrize("pc", ["fsai", "learned"])
def test_factor_refinement_has_the_block_jacobi_refinements_solution(precision, pc):
    mesh = beams.build_beam("nh_beam", cells=(24, 13, 12))
    kw = dict(outer_tolerance=1e-6, inner_tolerance=1e-2)
    a, xa = solve(mesh, preconditioner=pc, solver_precision=precision, **kw)
    b, xb = solve(mesh, solver_precision="fp32_refined", **kw)
    assert a.mixed_stats()[0]["rel_residual"] <= 1e-6 and b.mixed_stats()[0]["rel_residual"] <= 1e-6
    assert float((xa - xb).abs().max()) <= 1e-4 * float(xb.abs().max())


# -- the forms that explicit settings select -----------------------------------
@pytest.mark.parametrize("kw", [dict(), dict(solver_precision="fp32_refined"), dict(solver_precision="fp16"),
                                dict(preconditioner="fsai"), dict(preconditioner="fsai", solver_precision="fp16")],
                         ids=["single_reduction", "mixed_fp32", "mixed_fp16", "factor", "factor_fp16"])
def test_windowed_forms_agree_with_the_default_and_recover_from_a_timeout(kw):
    mesh = beams.build_beam("nh_beam", cells=(16, 4, 4))
    q = {}
    for ctas in (0, windowed_ctas(mesh)):
        solver = solver_of(mesh, iterations=mesh.spec.iterations, pcg_ctas=ctas, **kw)
        s0, s1 = solver.model.state(), solver.model.state()
        s0.particle_q.copy_(torch.as_tensor(mesh.q0, device=DEV))
        start = s0.particle_q.clone()
        s0, s1 = run_steps(solver, mesh, s0, s1, 1)
        assert all(st["status"] == _lib.MFEM_OK for st in solver.solve_stats())
        q[ctas] = s0.particle_q.cpu().numpy()
        solver.inject_timeout()
        solver.step(s0, s1, None, None, mesh.spec.dt)
        with pytest.raises(_lib.MfemError) as err:
            solver.solve_stats()
        assert err.value.code == _lib.MFEM_TIMEOUT
        s1.particle_q.copy_(start)
        run_steps(solver, mesh, s1, s0, 2)
        assert all(st["status"] == _lib.MFEM_OK for st in solver.solve_stats())
    a, b = q.values()
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


def test_windowed_variants_agree():
    """The cached single-reduction kernel and the standard one over a few
    steps, as tests of the default plan compare the resident form."""
    mesh = beams.build_beam("nh_beam", cells=(16, 4, 4))
    out = []
    for variant in ("standard", "single_reduction"):
        solver = solver_of(mesh, iterations=8, pcg_variant=variant, pcg_ctas=windowed_ctas(mesh))
        assert solver.pcg_layout()["variant"] == variant and solver.pcg_layout()["cache_matrix"]
        s0, s1 = solver.model.state(), solver.model.state()
        s0.particle_q.copy_(torch.as_tensor(mesh.q0, device=DEV))
        s0, s1 = run_steps(solver, mesh, s0, s1, 3)
        assert all(st["status"] == _lib.MFEM_OK for st in solver.solve_stats())
        out.append(s0.particle_q.cpu().numpy())
    assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[1]).max()
