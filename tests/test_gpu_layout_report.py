"""mfem_plan_pcg_layout names the form a plan's solves run in: the CTAs and
shared memory are the resident PCG's where that form takes the solves, and
those of the form with explicit CTAs where it does not."""
import pytest
import torch

from mfem_gb300 import Model, MixedFEMSolver, beams
from test_gpu_resident import shuffled

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CELLS = (34, 20, 17)  # 13,230 vertices: a grid


def layout(order, **kw):
    mesh = beams.build_beam("nh_beam", cells=CELLS)
    if order == "shuffled":
        mesh = shuffled(mesh)
    model = Model.from_beam(mesh, device=DEV)
    return MixedFEMSolver(model, iterations=1, energy=mesh.spec.energy, line_search=False, **kw).pcg_layout()


@pytest.mark.parametrize("order", ["grid", "shuffled"])
def test_block_jacobi_sizes_are_those_of_the_form_that_runs(order):
    fp32 = layout(order)
    assert fp32["ctas"] == -(-13230 // 128)  # 128 rows a CTA
    for precision in ("fp16", "fp32_refined"):
        assert layout(order, solver_precision=precision) == fp32, precision
    explicit = layout(order, pcg_ctas=torch.cuda.get_device_properties(0).multi_processor_count)
    assert explicit["ctas"] != fp32["ctas"] and explicit["variant"] == fp32["variant"]
    # BF16 blocks, and a refinement without a preconditioner, keep the other form
    assert layout(order, solver_precision="bf16") == explicit
    assert layout(order, solver_precision="fp32_refined", preconditioner=False) == explicit


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16", "fp32_refined"])
def test_factor_plan_of_a_shuffled_mesh_reports_its_resident_sizes(precision):
    lay = layout("shuffled", preconditioner="fsai", solver_precision=precision)
    assert lay["variant"] == "global_memory"
    assert lay["smem_bytes"] > 0 and lay["cache_matrix"], lay
    explicit = layout("shuffled", preconditioner="fsai", solver_precision=precision, pcg_ctas=100)
    assert explicit["smem_bytes"] == 0 and explicit["ctas"] == 100, explicit
