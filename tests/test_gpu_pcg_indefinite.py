"""
PCG on operators that are not positive definite.  The iterate at the first non-positive curvature is amplified rounding
there (two orders of summation differ by 1e-5 to 1 of it on these systems), so every device form of the solve has to end
with the same one: that of the physical moduli, one launch per colour, bit for bit.
"""
import pytest
import torch

from difffea_b200 import ops
from difffea_b200.krylov import DevicePCG
from difffea_b200.materials import device_material
from difffea_b200.newton_krylov import pcg
from difffea_b200.operators import make_preconditioner, make_tangent_operator
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _system(et, nx, ny, amplitude):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device=DEV)
    g = torch.Generator().manual_seed(7 * nx + ny)
    n, h = p["f"].numel(), 1.0 if et in ("quad4", "tri3") else 0.5
    u = ((2.0 * torch.rand(n, dtype=torch.float64, generator=g) - 1.0) * amplitude * h / ny).to(DEV) * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).to(DEV)
    return p, u, th, p["m"] * torch.randn(n, dtype=torch.float64, generator=g).to(DEV)


def _by_colours(A, p, u, th, b, pre, max_iter=3000):
    """The solve from the physical moduli, diagonal and blocks of (u, theta), a launch per colour."""
    mat = ops.material_args(device_material(p))
    C, diag = ops.qp_moduli(A.mesh_id, u, th, *mat, False, True)
    blocks = torch.empty(2 * A.mesh.n_dof, dtype=torch.float64, device=DEV)
    torch.ops.difffea_b200.qp_moduli_out(A.mesh_id, u, th, *mat, torch.empty(0, dtype=torch.float64, device=DEV), 0,
                                         torch.empty_like(diag), blocks)
    x = torch.empty_like(b)
    h = DevicePCG(A.mesh, C, diag if pre == "jacobi" else blocks, b.clone(), x, preconditioner=pre)
    k, status = h.solve(1e-12, max_iter)
    h.close()
    return x, k, status


# cluster form, fused form (the last two); a few dozen iterations to a thousand
SYSTEMS = [("quad9", 19, 4, 0.05), ("quad9", 46, 11, 0.05), ("tri3", 37, 9, 0.1), ("tri6", 40, 10, 0.05),
           ("quad4", 97, 23, 0.1), ("quad9", 120, 60, 0.1), ("tri3", 500, 125, 0.1)]


@pytest.mark.parametrize("et,nx,ny,amplitude", SYSTEMS)
@pytest.mark.parametrize("pre", ["jacobi", "block_jacobi"])
def test_negative_curvature_has_one_answer(et, nx, ny, amplitude, pre):
    p, u, th, b = _system(et, nx, ny, amplitude)
    A, M = make_tangent_operator("cuda", u, th, p), make_preconditioner(pre, u, th, p)
    want, k_want, status = _by_colours(A, p, u, th, b, pre)
    assert status == "negative_curvature"
    for _ in range(2):                                   # the second solve of an operator as the first
        x, k = pcg(A, b, M, rtol=1e-12, max_iter=3000)
        assert A.last_status == status and k == k_want and torch.equal(x, want)
    # a preconditioner made at another point keeps its own diagonal
    M0 = make_preconditioner(pre, torch.zeros_like(u), th, p)
    x0, _ = pcg(A, b, M0, rtol=1e-12, max_iter=3000)
    assert not torch.equal(x0, want)


def test_a_point_that_was_written_to_is_not_read():
    p, u, th, b = _system("quad9", 19, 4, 0.05)
    A, M = make_tangent_operator("cuda", u, th, p), make_preconditioner("jacobi", u, th, p)
    want, k_want, _ = _by_colours(A, p, u, th, b, "jacobi")
    C = A.moduli.clone()
    u.zero_()                                            # A stays the operator of the old u
    x, k = pcg(A, b, M, rtol=1e-12, max_iter=3000)
    assert A.last_status == "negative_curvature" and torch.equal(A.moduli, C) and abs(k - k_want) <= 3


def test_a_diagonal_that_was_written_to_is_the_one_used():
    p, u, th, b = _system("quad4", 97, 23, 0.1)
    A, M = make_tangent_operator("cuda", u, th, p), make_preconditioner("jacobi", u, th, p)
    M.diag.copy_(torch.ones_like(M.diag))                # plain CG
    x, _ = pcg(A, b, M, rtol=1e-12, max_iter=3000)
    C, _ = ops.qp_moduli(A.mesh_id, u, th, *ops.material_args(device_material(p)), False, True)
    want = torch.empty_like(b)
    h = DevicePCG(A.mesh, C, torch.ones_like(b), b.clone(), want)
    _, status = h.solve(1e-12, 3000)
    assert A.last_status == status == "negative_curvature" and torch.equal(x, want)


def test_definite_operators_keep_the_fast_form():
    p, u, th, b = _system("quad4", 97, 23, 0.05)
    A, M = make_tangent_operator("cuda", u, th, p), make_preconditioner("jacobi", u, th, p)
    x, k = pcg(A, b, M, rtol=1e-12, max_iter=3000)
    assert A.last_status == "converged" and A._pcg.form == "cluster" and A._indefinite is None
    want, k_want, _ = _by_colours(A, p, u, th, b, "jacobi")
    # both residuals are below 1e-12 |b|, the condition number is below 1e5
    assert abs(k - k_want) <= 3 and float(torch.linalg.vector_norm(x - want) / torch.linalg.vector_norm(want)) < 2e-7
