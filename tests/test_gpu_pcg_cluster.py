"""
The cluster form of the device PCG (one launch, vectors in distributed shared memory) against the fused launch form and
the oracle: one block and sixteen, ragged node ranges and tiles, both storage precisions, both preconditioners, and
every way a solve ends.
"""
import pytest
import torch

from difffea_b200 import _lib, ops
from difffea_b200.krylov import DevicePCG
from difffea_b200.materials import device_material
from difffea_b200.newton_krylov import pcg
from difffea_b200.operators import compute_block_jacobi, make_jacobi_preconditioner, make_tangent_operator
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel
from oracle import reference_path as oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _system(et, nx, ny, sign=1.0):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device=DEV)
    g = torch.Generator().manual_seed(7 * nx + ny)
    n = p["f"].numel()
    u = ((torch.rand(n, dtype=torch.float64, generator=g) - 0.5) * 0.02 / ny).to(DEV) * p["m"]
    th = sign * torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).to(DEV)
    b = torch.randn(n, dtype=torch.float64, generator=g).to(DEV)          # not masked: the identity rows take part
    return p, u, th, b, make_tangent_operator("cuda", u, th, p)


def _solve(A, C, d, b, form, rtol, cap, pre="jacobi"):
    bb, x = b.clone(), torch.full_like(b, float("nan"))
    h = DevicePCG(A.mesh, C, d, bb, x, use_graph=2, form=form, moduli="ref", preconditioner=pre)
    k, status = h.solve(rtol, cap)
    x1 = x.clone()
    assert h.solve(rtol, cap) == (k, status) and torch.equal(x1, x)        # reproducible, and reusable
    h.close()
    return x1, k, status


def _f32(A, p, u, th):
    C = torch.empty(A.mesh.moduli_numel_ref(), dtype=torch.float32, device=DEV)
    torch.ops.difffea_b200.frame_moduli_out(A.mesh_id, u, th, *ops.material_args(device_material(p)), C,
                                            _lib.DFEA_F32REF, torch.empty_like(u), torch.empty(0, device=DEV).double(),
                                            A.mesh.frame_work())
    return C


SIZES = [("quad4", 1, 1), ("quad4", 16, 4), ("quad4", 33, 1), ("quad4", 47, 11), ("quad4", 97, 23), ("quad9", 5, 3),
         ("quad9", 29, 13), ("quad8", 21, 9), ("tri6", 17, 13), ("tri3", 9, 5), ("tri3", 61, 37)]


@pytest.mark.parametrize("et,nx,ny", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("pre", ["jacobi", "block_jacobi"])
def test_cluster_form_matches_the_fused_form(et, nx, ny, precision, pre):
    p, u, th, b, A = _system(et, nx, ny)
    C = A.moduli if precision == "fp64" else _f32(A, p, u, th)
    d = A.diag if pre == "jacobi" else compute_block_jacobi(u, th, p)
    xf, kf, sf = _solve(A, C, d, b, "fused", 1e-11, 5000, pre)
    xc, kc, sc = _solve(A, C, d, b, "cluster", 1e-11, 5000, pre)
    # both stop at ||r|| <= 1e-11 ||b|| with rounding apart; the meshes' condition numbers are below 1e5
    # (the 33 x 1 strip's tangent is indefinite at this state: both end there with the same word)
    assert sf == sc and abs(kf - kc) <= 2 and rel(xc, xf) < 1e-7
    assert sc == "converged" or (et, nx, ny) == ("quad4", 33, 1)
    if precision == "fp64" and sc == "converged":
        assert rel(A(xc), b) < 1e-10                                      # the recurrence's residual is the true one


def test_cluster_form_follows_the_reference_recurrences():
    p, u, th, b, A = _system("quad4", 24, 8)
    M = make_jacobi_preconditioner(u, th, p)
    P = oracle.as_problem(p)
    d = oracle.jacobi_diagonal(u.cpu(), th.cpu(), P)
    x_ref, k_ref = oracle.pcg(oracle.make_operator("qp_ew", u.cpu(), th.cpu(), P), b.cpu(), lambda r: r / d, rtol=1e-10,
                              max_iter=2000)
    x, k = pcg(A, b, M, rtol=1e-10, max_iter=2000)                        # the closures' solve takes the cluster form
    assert abs(k - k_ref) <= 1 and rel(x, x_ref) < 1e-9


def test_cluster_form_ends():
    p, u, th, b, A = _system("quad4", 24, 8)
    x, k, status = _solve(A, A.moduli, A.diag, torch.zeros_like(b), "cluster", 1e-9, 50)
    assert (k, status) == (0, "zero_rhs") and float(x.abs().max()) == 0.0
    x, k, status = _solve(A, A.moduli, A.diag, b, "cluster", 1e-30, 7)
    xf, kf, sf = _solve(A, A.moduli, A.diag, b, "fused", 1e-30, 7)
    assert (k, status) == (kf, sf) == (7, "max_iter") and rel(x, xf) < 1e-12
    q, v, tn, bn, An = _system("quad4", 24, 8, sign=-1.0)
    bn = q["m"] * bn
    x, k, status = _solve(An, An.moduli, An.diag, bn, "cluster", 1e-9, 50)
    assert (k, status) == (0, "negative_curvature") and rel(x, bn / An.diag) < 1e-15


def test_meshes_that_do_not_fit_are_refused_or_take_the_launch_form():
    p, u, th, b, A = _system("quad9", 120, 60)
    with pytest.raises(RuntimeError, match="shared memory of a cluster"):
        DevicePCG(A.mesh, A.moduli, A.diag, b.clone(), torch.empty_like(b), form="cluster", moduli="ref")
    xf, kf, sf = _solve(A, A.moduli, A.diag, b, "fused", 1e-3, 200)
    bb, x = b.clone(), torch.empty_like(b)
    h = DevicePCG(A.mesh, A.moduli, A.diag, bb, x, use_graph=2, form="fused", moduli="ref", cluster=True)
    assert h.solve(1e-3, 200) == (kf, sf) and torch.equal(x, xf)
