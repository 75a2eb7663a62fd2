"""A hierarchy's maps are written on the stream of the mesh's device, whatever device is current when it is built."""
import contextlib
from types import SimpleNamespace

import torch

from difffea_b200 import _lib, multigrid
from difffea_b200.mesh import create_rectangle_mesh


def test_maps_are_launched_on_the_meshs_device(monkeypatch):
    nodes, conn = create_rectangle_mesh("quad4", 2.0, 1.0, 12, 6)
    entered, calls = [], []

    @contextlib.contextmanager
    def device(d):
        entered.append(d)
        yield
        entered.pop()

    class Stream:
        def synchronize(self):
            calls.append(("wait", list(entered)))

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(multigrid, "stream_handle", lambda: calls.append(("stream", list(entered))))
    monkeypatch.setattr(_lib, "call", lambda name, *a: calls.append((name, list(entered))))
    mesh = SimpleNamespace(device=torch.device("cpu"), n_nodes=nodes.shape[0], n_dof=2 * nodes.shape[0],
                           n_el=conn.shape[0], view_ref=None, ensure_frame=lambda: False)
    multigrid.Multigrid(mesh, {"conn": conn}, graphs=False)
    # the stream is asked for, the maps are launched and waited for, all with the mesh's device current
    assert [c[0] for c in calls] == ["stream", "dfea_mg_maps", "wait"]
    assert all(c[1] == [mesh.device] for c in calls)
