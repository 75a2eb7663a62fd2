"""A mesh without elements: no internal force, the load alone in the residual."""
import pytest
import torch

from difffea_b200.operators import global_residual, residual_and_norm, strain_energy
from difffea_b200.postprocess import internal_force, support_reactions
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et", ["quad4", "tri3", "quad9"])
def test_quantities_without_elements(et):
    p = build_rectangle_problem(et, 3, 2, 2.0, 1.0, load=(0.0, -1e-3), device="cuda")
    p = dict(p, conn=p["conn"][:0].clone(), dN_dX=p["dN_dX"][:0].clone(), w_detJ=p["w_detJ"][:0].clone())
    u = torch.linspace(-1.0, 1.0, p["f"].numel(), dtype=torch.float64, device="cuda")
    th = torch.ones(0, dtype=torch.float64, device="cuda")
    want = -0.5 * p["m"] * p["f"]
    assert torch.equal(global_residual(u, th, p, 0.5), want)
    R, norm = residual_and_norm(u, th, p, 0.5)
    assert torch.equal(R, want) and norm == pytest.approx(float(torch.linalg.vector_norm(want)), rel=1e-14)
    assert float(strain_energy(u, th, p)) == 0.0
    assert torch.equal(internal_force(u, th, p), torch.zeros_like(u))
    assert torch.equal(support_reactions(u, th, p), torch.zeros(2, dtype=torch.float64, device="cuda"))
