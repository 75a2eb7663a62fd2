"""What the frame calls return and refuse is what the calls they stand for return and refuse."""
import torch

from difffea_b200 import _lib, ops
from test_frame_scratch_cpu import MAT, N, TH, U, _Mesh


def test_internal_force_is_a_vector_whatever_the_shape_of_u(monkeypatch):
    mesh = _Mesh()
    monkeypatch.setattr(ops, "_mesh", lambda mesh_id: mesh)
    monkeypatch.setattr(ops, "stream_handle", lambda: None)
    monkeypatch.setattr(_lib, "call", lambda *a: None)
    for u in (U, U.view(N, 2)):
        assert ops.frame_internal_force.implementation(0, u, TH, *MAT).shape == (2 * N,)
