"""
The reference-frame element kernels (one warp per Gauss point, element pass + node pass) against the oracle, at
element counts around the block's 32 (Tri3: 128) elements and for every element type and material route, and the
kernels that read dN/dX for problems whose dN/dX is not Jinv^T dN/dxi.
"""
import pytest
import torch

from difffea_b200.adjoint import compute_implicit_vjp
from difffea_b200.cuda_mesh import cuda_mesh
from difffea_b200.operators import (global_residual, make_block_jacobi_preconditioner, make_jacobi_preconditioner,
                                    make_tangent_operator, strain_energy)
from difffea_b200.postprocess import compute_fields, internal_force
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel
from oracle import reference_path as oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _problem(et, nx, ny, material="neo_hookean", params=None):
    p = build_rectangle_problem(et, nx, ny, float(nx), float(ny), load=(0.01, -0.02), device=DEV, material=material,
                                material_params=params)
    g = torch.Generator().manual_seed(nx * 100 + ny)
    n = p["f"].numel()
    u = ((torch.rand(n, dtype=torch.float64, generator=g) * 2 - 1) * 0.04).to(DEV) * p["m"]
    v = torch.randn(n, dtype=torch.float64, generator=g).to(DEV)
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).to(DEV)
    return p, u, v, th


def _check(p, u, v, th):
    # FP64 with sums of at most 9 x 9 terms: 1e-12 (fields of differences 1e-11), the parity bars of the package
    P, uc, tc, vc = oracle.as_problem(p), u.cpu(), th.cpu(), v.cpu()
    C = oracle.moduli(uc, tc, P)
    A = make_tangent_operator("cuda", u, th, p)
    assert rel(A(v), oracle.apply_qp_ew(C, vc, P)) < 1e-12
    assert torch.equal(A(v), A(v))
    assert rel(global_residual(u, th, p, 0.7), oracle.residual(uc, tc, P, 0.7)) < 1e-12
    d = oracle.jacobi_diagonal(uc, tc, P)
    assert rel(A.diag, d) < 1e-12 and rel(make_jacobi_preconditioner(u, th, p).diag, d) < 1e-12
    W = float(oracle.strain_energy(uc, tc, P))
    assert abs(float(strain_energy(u, th, p)) - W) <= 1e-11 * abs(W)
    B = make_block_jacobi_preconditioner(u, th, p)(v)
    assert rel(B, oracle.block_jacobi(uc, tc, P)(vc)) < 1e-11
    return A


@pytest.mark.parametrize("et,nx,ny", [("quad4", 1, 1), ("quad4", 31, 1), ("quad4", 8, 4), ("quad4", 11, 3),
                                      ("quad9", 1, 1), ("quad9", 31, 1), ("quad9", 33, 1), ("quad8", 8, 4),
                                      ("quad8", 13, 5), ("tri6", 4, 4), ("tri6", 11, 3), ("tri3", 8, 8), ("tri3", 43, 3),
                                      ("tri3", 1, 1)])
def test_frame_kernels_at_tile_edges(et, nx, ny):
    p, u, v, th = _problem(et, nx, ny)
    assert cuda_mesh(p).ensure_frame()
    _check(p, u, v, th)


@pytest.mark.parametrize("et", ["quad4", "tri6"])
@pytest.mark.parametrize("material,params", [("mooney_rivlin", {"c10": 0.2, "c01": 0.05, "kappa": 0.7}),
                                             ("saint_venant", {"mu": 0.4, "lmbda": 0.6}),
                                             ("demiray", {"mu": 0.4, "gamma": 2.0, "lmbda": 0.6})])
def test_frame_kernels_with_differentiated_materials(et, material, params):
    p, u, v, th = _problem(et, 9, 5, material, params)
    _check(p, u, v, th)


@pytest.mark.parametrize("et", ["quad4", "quad9", "quad8", "tri6", "tri3"])
def test_frame_kernels_agree_with_the_gradient_kernels(et):
    """The same problem through both kernel families: a mesh whose frame is withheld reads dN/dX."""
    p, u, v, th = _problem(et, 23, 7)
    mesh = cuda_mesh(p)
    assert mesh.ensure_frame()

    def results():
        fields = compute_fields(u, th, p)
        A = make_tangent_operator("cuda", u, th, p)
        C = A.C.view(mesh.n_q, 8, mesh.stride, 2)[:, :, :mesh.n_el]               # without the padding slots
        return [A(v), C, global_residual(u, th, p), internal_force(u, th, p), compute_implicit_vjp(u, th, p, v)] + list(fields.values())

    framed = results()
    frame, mesh.frame = mesh.frame, None
    plain = results()
    mesh.frame = frame
    for a, b in zip(framed, plain):
        assert rel(a, b) < 1e-12


def test_gradients_that_are_no_frame_keep_the_kernels_that_read_them():
    """dN/dX perturbed entry by entry is no Jinv^T dN/dxi: the product still is the one of the given dN/dX."""
    p, u, v, th = _problem("quad4", 12, 7)
    g = torch.Generator().manual_seed(5)
    noise = 1.0 + 1e-6 * torch.randn(p["dN_dX"].shape, dtype=torch.float64, generator=g).to(DEV)
    q = {**p, "dN_dX": p["dN_dX"] * noise}
    assert not cuda_mesh(q).ensure_frame() and cuda_mesh(p).ensure_frame()
    _check(q, u, v, th)


@pytest.mark.parametrize("material,flags", [("neo_hookean", [True, False]), ("mooney_rivlin", [False, True, True]),
                                            ("demiray", [True, False, True]),
                                            ("fiber_reinforced", [True, False, True, False, False, False, False])])
def test_material_read_on_the_device_is_the_host_one(material, flags):
    """Parameters and flags as device tensors (read by the kernels) or host tensors (passed in the struct)."""
    p, u, v, th = _problem("quad4", 9, 5, material)
    u, lam = 0.2 * u, v
    outs = []
    for where in ("cuda", "cpu"):
        q = {**p, "mat_p": p["mat_p"].to(where), "mat_scalable": torch.tensor(flags, device=where)}
        outs.append([make_tangent_operator("cuda", u, th, q)(v), global_residual(u, th, q), internal_force(u, th, q),
                     compute_implicit_vjp(u, th, q, lam), strain_energy(u, th, q)] + list(compute_fields(u, th, q).values()))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
