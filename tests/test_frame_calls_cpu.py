"""What the frame calls return and refuse is what the calls they stand for return and refuse."""
import pytest
import torch

from difffea_b200 import _lib, operators, ops, postprocess
from test_frame_scratch_cpu import MAT, N, TH, U, _Mesh


def test_internal_force_is_a_vector_whatever_the_shape_of_u(monkeypatch):
    mesh = _Mesh()
    monkeypatch.setattr(ops, "_mesh", lambda mesh_id: mesh)
    monkeypatch.setattr(ops, "stream_handle", lambda: None)
    monkeypatch.setattr(_lib, "call", lambda *a: None)
    for u in (U, U.view(N, 2)):
        assert ops.frame_internal_force.implementation(0, u, TH, *MAT).shape == (2 * N,)


def test_fields_of_a_u_of_the_wrong_length(monkeypatch):
    mesh = _Mesh()
    mesh.ensure_frame = lambda: True
    monkeypatch.setattr(ops, "_mesh", lambda mesh_id: mesh)
    monkeypatch.setattr(ops, "run", lambda op, *args: op.implementation(*args))
    monkeypatch.setattr(ops, "frame_material", lambda params: MAT)
    monkeypatch.setattr(postprocess, "_prepare", lambda u, theta, params: (mesh, 0))
    with pytest.raises(ValueError, match="expected 24 entries, got 22"):
        postprocess.compute_fields(U[:-2], TH, {})


def test_the_diagonal_of_an_operator_is_that_of_its_material(monkeypatch):
    """A preconditioner reuses the diagonal of the operator made just before it -- on the same mesh, u, theta and material."""
    mesh, calls = _Mesh(), []
    mesh.ensure_frame, mesh.ensure_gather, mesh.moduli_numel_ref = lambda: True, lambda: True, lambda: 4
    params = {"conn": torch.zeros(0, dtype=torch.int64), "material": "neo_hookean",
              "mat_p": torch.tensor([0.4, 0.6], dtype=torch.float64), "mat_scalable": torch.ones(2, dtype=torch.bool)}

    def run(op, *args):
        calls.append(op)
        return torch.zeros(4, dtype=torch.float64), torch.full((2 * N,), float(len(calls)), dtype=torch.float64), None

    monkeypatch.setattr(ops, "run", run)
    monkeypatch.setattr(operators, "_prepare", lambda u, theta, p: (mesh, 0))
    u, theta = U.clone(), TH.clone()
    A = operators.make_A_operator_cuda(u, theta, params)
    assert operators.make_jacobi_preconditioner(u, theta, params).diag is A.diag and len(calls) == 1
    other = dict(params, mat_p=torch.tensor([0.8, 0.6], dtype=torch.float64))
    assert operators.compute_jacobi_diagonal(u, theta, other) is not A.diag and len(calls) == 2
    for wrong in ({"material": "nope"}, {"mat_p": torch.zeros(1, dtype=torch.float64)}):
        with pytest.raises(ValueError):
            operators.compute_jacobi_diagonal(u, theta, dict(params, **wrong))
    params["mat_p"].mul_(2.0)                            # the operator's diagonal is of the old parameters
    assert operators.compute_jacobi_diagonal(u, theta, params) is not A.diag
    A = operators.make_A_operator_cuda(u, theta, params)
    u.add_(1.0)
    assert operators.compute_jacobi_diagonal(u, theta, params) is not A.diag
