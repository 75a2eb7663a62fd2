"""What the frame calls return and refuse is what the calls they stand for return and refuse."""
import pytest
import torch

from difffea_b200 import _lib, ops, postprocess
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
