"""
The scratch of a frame call belongs to the call until its kernels are launched: given back to the allocator earlier, a
second thread on the same stream gets the same block between this call's element pass and its node pass.
"""
import weakref

import pytest
import torch

from difffea_b200 import ops

N, E = 12, 6
F64 = torch.float64


class _Mesh:
    device, view_ref, frame = torch.device("cpu"), None, object()
    n_nodes, n_dof, n_el = N, 2 * N, E

    def moduli_numel_ref(self):
        return 4

    def frame_work(self):
        work = torch.empty(256, dtype=torch.uint8)
        self.work = weakref.ref(work)
        return work


U, TH, MAT = torch.zeros(2 * N, dtype=F64), torch.zeros(E, dtype=F64), (0, 0, [1.0, 1.0], None, None)
CALLS = {
    "frame_moduli": (U, TH, *MAT, True, True),
    "frame_residual": (U, TH, *MAT, U, 1.0, True),
    "frame_internal_force": (U, TH, *MAT),
    "frame_all_fields": (U, TH, *MAT),
    "frame_reactions": (U, TH, *MAT, torch.zeros(2 * N, dtype=torch.bool)),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_scratch_lives_until_the_launches_are_made(monkeypatch, name):
    mesh, alive = _Mesh(), []
    monkeypatch.setattr(ops, "_mesh", lambda mesh_id: mesh)
    monkeypatch.setattr(ops, "stream_handle", lambda: None)
    monkeypatch.setattr(ops._lib, "call", lambda *a: alive.append(mesh.work() is not None))
    getattr(ops, name).implementation(0, *CALLS[name])
    assert alive == [True]
