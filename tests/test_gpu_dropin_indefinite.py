"""The PCG that the drop-in puts in place of a package's own gives pcg()'s answer, on indefinite operators too."""
import sys
from types import ModuleType

import pytest
import torch

from difffea_b200.dropin import register
from difffea_b200.newton_krylov import pcg
from difffea_b200.operators import make_jacobi_preconditioner, make_tangent_operator
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu


def test_negative_curvature_through_the_drop_in(monkeypatch):
    package = ModuleType("a_solver_package")             # with the names that the drop-in replaces
    package.operators, package.newton_krylov = (ModuleType("a_solver_package." + n) for n in ("operators", "newton_krylov"))
    for module in (package.operators, package.newton_krylov):
        module.make_tangent_operator = module.make_preconditioner = module.pcg = None
        monkeypatch.setitem(sys.modules, module.__name__, module)
    monkeypatch.setitem(sys.modules, package.__name__, package)
    package.operators.TANGENT_OPERATORS = package.operators.PRECONDITIONERS = ()
    p = build_rectangle_problem("quad9", 19, 4, 19 / 4, 1.0, load=(0.0, -1e-3), device="cuda")
    g = torch.Generator().manual_seed(7 * 19 + 4)
    n = p["f"].numel()
    u = ((2.0 * torch.rand(n, dtype=torch.float64, generator=g) - 1.0) * 0.025 / 4).cuda() * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).cuda()
    b = p["m"] * torch.randn(n, dtype=torch.float64, generator=g).cuda()
    # the preconditioner of another point than the operator's: its diagonal has to be found again too
    M = make_jacobi_preconditioner(0.5 * u, th, p)
    A = make_tangent_operator("cuda", u, th, p)
    want = pcg(A, b, M, rtol=1e-12, max_iter=3000)
    assert A.last_status == "negative_curvature"
    undo = register(package)
    try:
        A = package.operators.make_tangent_operator("cuda", u, th, p)
        x, k = package.newton_krylov.pcg(A, b, M, rtol=1e-12, max_iter=3000)
    finally:
        undo()
    assert A.last_status == "negative_curvature" and k == want[1] and torch.equal(x, want[0])
