"""
The multigrid's conjugate-gradient steps in two launches (reference-frame moduli) and its smoothing with the updates in
the node passes, against the general form (physical moduli in the colour form: a launch per operation), for every number
of smoothing steps; the host-driven loop against the graph-driven one; and the ends that are not convergence.
"""
import pytest
import torch

from difffea_b200 import _lib
from difffea_b200.multigrid import Multigrid
from difffea_b200.operators import make_tangent_operator
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _setup(et, nx, ny, degree, amplitude=0.02, graphs=False, fixed=None):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device=DEV, build_on_device=True)
    g = torch.Generator(device=DEV).manual_seed(nx + 7 * degree)
    n = p["f"].numel()
    u = (torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 0.5) * amplitude / ny * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, device=DEV, generator=g))
    b = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    A = make_tangent_operator("cuda", u, th, p)
    assert A.code == _lib.DFEA_F64REF
    fused, general = Multigrid(A.mesh, p, degree=degree, graphs=graphs), Multigrid(A.mesh, p, degree=degree, graphs=graphs)
    general.h.fe_work = None
    fused.setup(A.moduli, A.code, A.diag)
    general.setup(A.C, _lib.DFEA_F64, A.diag)
    return A, b, fused, general


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("et,nx,ny", [("quad4", 3, 2), ("quad4", 33, 20), ("quad4", 120, 61), ("quad9", 7, 5),
                                      ("quad9", 47, 22), ("tri3", 30, 21), ("tri6", 23, 12), ("quad8", 30, 11)])
def test_two_launch_steps_give_the_general_forms_cycle_and_solve(et, nx, ny, degree):
    A, b, fused, general = _setup(et, nx, ny, degree)
    # the bounds come from CG coefficients, equal to rounding; a cycle adds a few smoothing steps and a dense solve
    for lf, lg in zip(fused.levels[:-1], general.levels[:-1]):
        assert abs(lf.lam - lg.lam) <= 1e-9 * lg.lam
    z, z_ref = fused(b), general(b)
    assert rel(z, z_ref) < 1e-9
    assert torch.equal(z, fused(b))
    x, x_ref = torch.empty_like(b), torch.empty_like(b)
    it, word = fused.pcg(b, x, 1e-11, 400)
    it_ref, word_ref = general.pcg(b, x_ref, 1e-11, 400)
    assert word == word_ref == "converged" and abs(it - it_ref) <= 1
    assert float((b - A(x)).norm()) <= 2e-11 * float(b.norm())
    assert float((b - A(x_ref)).norm()) <= 2e-11 * float(b.norm())


@pytest.mark.parametrize("form", ["fused", "general"])
def test_graph_driven_solves_are_the_host_driven_ones(form):
    A, b, f0, g0 = _setup("quad9", 33, 14, 2)
    host = f0 if form == "fused" else g0
    _, _, f1, g1 = _setup("quad9", 33, 14, 2, graphs=True)
    graph = f1 if form == "fused" else g1
    x, y = torch.empty_like(b), torch.empty_like(b)
    end = host.pcg(b, x, 1e-9, 200)
    for _ in range(3):                                     # the first runs directly, the second captures, the third replays
        graph.setup(*((A.moduli, A.code) if form == "fused" else (A.C, _lib.DFEA_F64)), A.diag)
        assert graph.pcg(b, y, 1e-9, 200) == end
        assert torch.equal(x, y)


@pytest.mark.parametrize("graphs", [False, True])
def test_ends_without_convergence(graphs):
    A, b, fused, general = _setup("quad4", 24, 9, 2, graphs=graphs)
    x, x_ref = torch.empty_like(b), torch.empty_like(b)
    for mg in (fused, general):
        for _ in range(2):
            assert mg.pcg(b, x, 1e-14, 3) == (3, "max_iter")
            assert mg.pcg(b, x, 1e-14, 0) == (0, "max_iter") and not x.any()
            assert mg.pcg(torch.zeros_like(b), x, 1e-8, 50)[1] == "zero_rhs" and not x.any()
    A, b, fused, general = _setup("quad4", 24, 9, 2, amplitude=6.0, graphs=graphs)   # far from equilibrium: indefinite
    for _ in range(2):
        end, end_ref = fused.pcg(b, x, 1e-8, 50), general.pcg(b, x_ref, 1e-8, 50)
        assert end == end_ref and end[1] == "negative_curvature"
        if end[0] == 0:                                    # x = z, a cycle (inverted elements: NaN at the same entries)
            live = ~x_ref.isnan()
            assert torch.equal(live, ~x.isnan())
            assert rel(x[live], x_ref[live]) < 1e-9
