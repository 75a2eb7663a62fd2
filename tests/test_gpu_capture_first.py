"""
Calls captured into a CUDA graph before the mesh has a frame or an incidence (a material on the host, which the frame
forms do not read through the device): the graph computes what the eager call does, and leaves the mesh as it was.
"""
import pytest
import torch

from difffea_b200.adjoint import compute_implicit_vjp
from difffea_b200.cuda_mesh import cuda_mesh
from difffea_b200.operators import (compute_block_jacobi, compute_jacobi_diagonal, global_residual, make_A_operator_cuda)
from difffea_b200.postprocess import compute_fields, element_fields, internal_force, support_reactions
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _all_fields(u, th, p):
    out = compute_fields(u, th, p)
    return torch.cat([out[k].reshape(-1) for k in sorted(out)])


CALLS = {
    "residual": global_residual, "product": lambda u, th, p: make_A_operator_cuda(u, th, p)(u),
    "product32": lambda u, th, p: make_A_operator_cuda(u, th, p, "fp32")(u.float()),
    "diagonal": compute_jacobi_diagonal, "blocks": compute_block_jacobi, "force": internal_force, "elements": element_fields,
    "fields": _all_fields, "reactions": support_reactions, "vjp": lambda u, th, p: compute_implicit_vjp(u, th, p, u),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_a_capture_as_the_first_call(name):
    p = build_rectangle_problem("quad4", 20, 10, 2.0, 1.0, load=(0.0, -1e-3), device=DEV)
    p = dict(p, mat_p=p["mat_p"].cpu(), mat_scalable=p["mat_scalable"].cpu())
    g = torch.Generator().manual_seed(3)
    u = ((torch.rand(p["f"].numel(), dtype=torch.float64, generator=g) - 0.5) * 4e-3).to(DEV) * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).to(DEV)
    mesh = cuda_mesh(p)
    if name == "product32":
        mesh.ensure_grad32()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = CALLS[name](u, th, p)
    assert mesh.frame is None and mesh.node_elem is None
    graph.replay()
    captured = out.clone()
    # the eager call takes the frame form: rounding of the pulled-back moduli and of the order of sums
    assert rel(captured.double(), CALLS[name](u, th, p).double()) < (1e-6 if name == "product32" else 1e-12)
    assert mesh.node_elem is not None
    graph.replay()
    assert torch.equal(out, captured)
