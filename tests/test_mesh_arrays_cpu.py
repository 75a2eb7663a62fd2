"""
The arrays a mesh builds on demand, when several threads and streams share it: the attribute that says an array is there
is set only when the array is complete -- its kernels launched, the stream waited for, the view's pointers filled in.
"""
import contextlib
import ctypes
import threading
from types import SimpleNamespace

import pytest
import torch

from difffea_b200 import _lib, cuda_mesh, ops
from difffea_b200.cuda_mesh import CudaMesh


def _mesh():
    m = object.__new__(CudaMesh)
    m.device, m.n_el, m.nen, m.n_q, m.n_nodes, m.stride = torch.device("cpu"), 4, 4, 4, 9, 32
    m.grad32 = m.node_elem = m.node_elem_ptr = m.frame = m.jinv = m._frame_check = None
    m._nodes = torch.zeros(9, 2, dtype=torch.float64)
    m._lock = threading.RLock()
    m.view = _lib.MeshView()
    return m


@pytest.fixture
def log(monkeypatch):
    """What a build does, in order: the launches and the waits, with the arrays another thread can see at that moment."""
    mesh, events = _mesh(), []
    names = ("grad32", "node_elem", "node_elem_ptr", "frame", "jinv")

    def note(what):
        events.append((what, [n for n in names if getattr(mesh, n) is not None]))

    def call(name, *args):
        note(name)
        if name == "dfea_mesh_frame":
            ctypes.memset(args[3], 0, 24)          # the fit error: none

    class Stream:
        def synchronize(self):
            note("wait")

    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(cuda_mesh, "stream_handle", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    return mesh, events


@pytest.mark.parametrize("build,launch,attributes", [
    ("ensure_grad32", "dfea_mesh_grad_to_f32", ("grad32",)),
    ("ensure_node_incidence", "dfea_mesh_node_incidence", ("node_elem_ptr", "node_elem"))])
def test_nothing_is_announced_before_the_wait(log, build, launch, attributes):
    mesh, events = log
    getattr(mesh, build)()
    assert events == [(launch, []), ("wait", [])]
    for name in attributes:
        assert getattr(mesh.view, name) == getattr(mesh, name).data_ptr()
    getattr(mesh, build)()
    assert len(events) == 2                        # once


def test_inside_a_capture_nothing_is_announced(log, monkeypatch):
    """What a graph would write is there after its first replay only: such a call takes the forms that need none of it."""
    mesh, events = log
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert not mesh.ensure_frame() and not mesh.ensure_gather() and not events
    view, keep = mesh.gather_view()                # an incidence of this call's own
    assert events == [("dfea_mesh_node_incidence", [])] and view._obj.node_elem == keep[2].data_ptr()
    assert mesh.node_elem is None and not mesh.view.node_elem
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert mesh.ensure_frame() and mesh.ensure_gather() and mesh.gather_view()[1] is None


def test_the_frame_and_its_incidence_are_announced_after_their_read(log):
    mesh, events = log
    assert mesh.ensure_frame()                     # reading the fit error waits for both
    assert [e for e in events if e[1]] == [] and [e[0] for e in events] == ["dfea_mesh_node_incidence", "dfea_mesh_frame"]
    assert mesh.view.frame == mesh.frame.data_ptr() and mesh.view.node_elem == mesh.node_elem.data_ptr()


@pytest.mark.parametrize("gather", [False, True])
def test_the_product_form_does_not_depend_on_what_the_mesh_has_built(monkeypatch, gather):
    """Physical moduli: the colour form unless the caller asks for the gather form, with or without an incidence."""
    called = []
    monkeypatch.setattr(ops, "stream_handle", lambda: None)
    monkeypatch.setattr(_lib, "call", lambda name, *a: called.append(name))
    C, v = torch.zeros(16, dtype=torch.float64), torch.zeros(18, dtype=torch.float64)
    for incidence in (None, torch.zeros(16, dtype=torch.int32)):
        mesh = SimpleNamespace(device=v.device, n_dof=18, node_elem=incidence, view_ref=ctypes.byref(_mesh().view),
                               moduli_numel_ref=lambda: 10, moduli_numel=lambda *a: 16, ensure_grad32=lambda: None)
        mesh.gather_view = lambda: (mesh.view_ref, None)
        monkeypatch.setattr(ops, "_mesh", lambda mesh_id: mesh)
        ops.tangent_apply.implementation(0, C, v, gather)
    assert called == 2 * ["dfea_tangent_apply_gather" if gather else "dfea_tangent_apply"]
