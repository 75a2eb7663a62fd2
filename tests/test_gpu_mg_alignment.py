"""Multigrid on vectors that start between two nodal pairs (8 bytes past a 16-byte boundary)."""
import pytest
import torch

from difffea_b200.multigrid import Multigrid
from difffea_b200.operators import make_preconditioner, make_tangent_operator
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _between(t):
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    out.copy_(t)
    assert out.data_ptr() % 16 == 8
    return out


@pytest.mark.parametrize("et,nx,ny", [("quad4", 20, 10), ("quad9", 9, 7), ("tri6", 8, 5)])
@pytest.mark.parametrize("graphs", [False, True])
def test_cycle_and_solve(et, nx, ny, graphs):
    p = build_rectangle_problem(et, nx, ny, 2.0, 1.0, load=(0.0, -1e-3), device=DEV)
    g = torch.Generator(device=DEV).manual_seed(nx)
    n = p["f"].numel()
    u = (torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 0.5) * 2e-3 * p["m"]
    r = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    th = torch.ones(p["conn"].shape[0], dtype=torch.float64, device=DEV)
    M = make_preconditioner("multigrid", u, th, p)
    assert torch.equal(M(_between(r)), M(r))
    A = make_tangent_operator("cuda", u, th, p)
    mg = Multigrid(A.mesh, p, graphs=graphs)
    mg.setup(A.moduli, A.code, A.diag)
    x, y, b = torch.empty_like(r), _between(r), _between(p["m"] * r)
    for _ in range(3):                                   # launches, the captured loop, its replay
        ends = mg.pcg(p["m"] * r, x, 1e-10, 50)
        assert mg.pcg(b, y, 1e-10, 50) == ends and ends[1] == "converged"
        assert torch.equal(x, y)
