"""A kernel's shared-memory limit belongs to the process: a plan created later,
with less shared memory, leaves an earlier plan's launches valid.  For the
windowed forms of the PCG, which explicit CTAs select."""
import pytest

from mfem_gb300 import Model, MixedFEMSolver, beams

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("kw", [dict(), dict(pcg_variant="standard"), dict(pcg_variant="gather"),
                                dict(preconditioner="fsai"), dict(solver_precision="fp16")],
                         ids=["single_reduction", "standard", "gather", "factor", "refinement"])
def test_a_smaller_plan_leaves_an_earlier_one_valid(kw):
    solvers = []
    for cells, ctas in (((14, 7, 7), 8), ((4, 2, 2), 2)):
        mesh = beams.build_beam("nh_beam", cells=cells)
        model = Model.from_beam(mesh, device=DEV)
        solvers.append((mesh, model, MixedFEMSolver(model, iterations=1, energy=mesh.spec.energy, line_search=False,
                                                    pcg_ctas=ctas, use_cuda_graph=False, **kw)))
    big, small = (s.pcg_layout() for _, _, s in solvers)
    assert big["variant"] == small["variant"] and big["smem_bytes"] > max(small["smem_bytes"], 48 * 1024), (big, small)
    for mesh, model, solver in solvers:
        a, b = model.state(), model.state()
        solver.step(a, b, None, None, mesh.spec.dt)
        assert solver.solve_stats()[0]["status"] == 0
