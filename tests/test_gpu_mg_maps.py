"""
The grid behind a structured mesh found and mapped on the device, against the host search (the same function on a host
connectivity) and the maps written out in numpy: equal entry by entry, and refused alike when one entry differs.
"""
import numpy as np
import pytest
import torch

from difffea_b200.cuda_mesh import cuda_mesh
from difffea_b200.mesh import create_rectangle_mesh
from difffea_b200.multigrid import Multigrid, structured_grid
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = [(1, 1), (1, 9), (9, 1), (8, 8), (31, 17), (64, 3), (130, 257)]


def _same(a, b):
    assert (a is None) == (b is None)
    if a is not None:
        assert a.keys() == b.keys()
        for k in a:
            assert torch.equal(a[k].cpu(), b[k]) and a[k].dtype == b[k].dtype if torch.is_tensor(a[k]) else a[k] == b[k], k


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("et", ["quad4", "quad8", "quad9", "tri3", "tri6"])
def test_device_search_is_the_host_search(et, nx, ny):
    nodes, conn = create_rectangle_mesh(et, 2.0, 1.0, nx, ny)
    n = nodes.shape[0]
    _same(structured_grid(conn.to(DEV), n), structured_grid(conn, n))
    if et in ("quad4", "quad9"):                           # numbered along the other direction, as the quarter plate is
        span = 1 if et == "quad4" else 2
        ids = torch.arange((span * nx + 1) * (span * ny + 1)).reshape(span * ny + 1, span * nx + 1).t().reshape(-1)
        other = ids[conn]
        _same(structured_grid(other.to(DEV), n), structured_grid(other, n))
    if conn.shape[0] > 1:
        for e, a in ((0, 0), (conn.shape[0] - 1, conn.shape[1] - 1), (conn.shape[0] // 2, 1)):
            bad = conn.clone()
            bad[e, a] = (bad[e, a] + 1) % n
            _same(structured_grid(bad.to(DEV), n), structured_grid(bad, n))
        _same(structured_grid(conn.flip(1).to(DEV), n), structured_grid(conn.flip(1), n))
        _same(structured_grid(conn.to(DEV).t().contiguous().t(), n), structured_grid(conn, n))     # strided
    _same(structured_grid(conn.to(DEV), n + 1), structured_grid(conn, n + 1))


@pytest.mark.parametrize("et,nx,ny", [("quad4", 33, 18), ("quad4", 7, 100), ("quad9", 16, 5), ("quad8", 9, 30),
                                      ("tri3", 21, 40), ("tri6", 12, 11)])
def test_hierarchy_maps(et, nx, ny):
    p = build_rectangle_problem(et, nx, ny, float(nx), float(ny), device=DEV, build_on_device=True)
    mesh = cuda_mesh(p)
    mg = Multigrid(mesh, p)
    ints = mg._ints.cpu().numpy()
    base = mg._ints.data_ptr()
    view = lambda at, count: ints[(at - base) // 4:(at - base) // 4 + count]
    n_cells, epc = nx * ny, 2 if et in ("tri3", "tri6") else 1
    inv = np.empty_like(mesh.perm_host)
    inv[mesh.perm_host] = np.arange(mesh.perm_host.size)
    elems = np.arange(n_cells)[:, None] + n_cells * np.arange(epc)[None, :]
    assert np.array_equal(view(mg.h.cell_slot, n_cells * epc), inv[elems.reshape(-1)])
    for l in range(1, len(mg.levels)):
        f, c = mg.levels[l - 1], mg.levels[l]
        assert np.array_equal(view(c.grid.line_x, c.gx + 1), np.minimum(2 * np.arange(c.gx + 1), f.gx))
        assert np.array_equal(view(c.grid.line_y, c.gy + 1), np.minimum(2 * np.arange(c.gy + 1), f.gy))
        assert np.array_equal(view(c.grid.cell_x, f.gx + 1), np.minimum(np.arange(f.gx + 1) // 2, c.gx - 1))
        assert np.array_equal(view(c.grid.cell_y, f.gy + 1), np.minimum(np.arange(f.gy + 1) // 2, c.gy - 1))
