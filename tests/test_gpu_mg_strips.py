"""
Multigrid on thin strips, whose levels stop shrinking in one direction: the levels after the first small one then add as
much shared memory again to the cluster tail, which has to start below it.
"""
import pytest
import torch

from difffea_b200.multigrid import Multigrid
from difffea_b200.newton_krylov import newton_krylov_solve
from difffea_b200.operators import make_tangent_operator
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("et,nx,ny", [("quad4", 4800, 2), ("quad4", 5000, 1), ("quad4", 3900, 4), ("quad4", 3000, 6),
                                      ("quad4", 5900, 10), ("quad9", 2950, 3), ("tri3", 4800, 2)])
def test_the_cycle_of_a_strip(et, nx, ny):
    p = build_rectangle_problem(et, nx, ny, float(nx), float(ny), load=(0.0, -1e-3), device=DEV, build_on_device=True)
    g = torch.Generator(device=DEV).manual_seed(nx)
    n = p["f"].numel()
    u = (torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 0.5) * 0.02 * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, device=DEV, generator=g))
    r = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    A = make_tangent_operator("cuda", u, th, p)
    clustered, plain = Multigrid(A.mesh, p, graphs=False), Multigrid(A.mesh, p, graphs=False)
    plain.h.stencil = None                                       # a launch per step
    for mg in (clustered, plain):
        mg.setup(A.moduli, A.code, A.diag)
    # sums in another order: rounding through a few smoothing steps and one dense solve of at most 48 nodes, whose strip
    # of up to 24 cells has a condition number below 1e6
    for a, b in zip(clustered.levels[:-1], plain.levels[:-1]):
        assert abs(a.lam - b.lam) <= 1e-10 * b.lam
    assert rel(clustered(r), plain(r)) < 1e-9


def test_a_solve_on_a_strip():
    p = build_rectangle_problem("quad4", 3000, 6, 3000.0, 6.0, load=(1e-3, 0.0), device=DEV, build_on_device=True)
    th = torch.ones(p["conn"].shape[0], dtype=torch.float64, device=DEV)
    u, info = newton_krylov_solve(p, th, 1, 1e-8 * float(torch.linalg.vector_norm(p["f"])), verbose=False,
                                  preconditioner="multigrid")[:2]
    assert bool(torch.isfinite(u).all()) and float(u.abs().max()) > 0.0
