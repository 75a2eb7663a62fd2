"""
The small levels of the multigrid in thread-block clusters: a cycle and its smoother bounds against the launch-per-step
driver (a hierarchy without node stencils) on grids around the blocks' node ranges, and the coarsest inverse around its
register tiles.
"""
import ctypes

import pytest
import torch

from difffea_b200 import _lib
from difffea_b200.cuda_mesh import ptr, stream_handle
from difffea_b200.multigrid import Multigrid
from difffea_b200.operators import make_tangent_operator
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("et,nx,ny", [("quad4", 13, 5), ("quad4", 31, 17), ("quad4", 64, 64), ("quad4", 150, 37),
                                      ("quad4", 260, 70), ("quad9", 16, 4), ("quad9", 61, 33), ("tri3", 40, 21),
                                      ("tri6", 23, 12), ("quad8", 30, 11)])
def test_cluster_tail_gives_the_cycle_of_the_launch_driver(et, nx, ny):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device=DEV, build_on_device=True)
    g = torch.Generator(device=DEV).manual_seed(nx)
    n = p["f"].numel()
    u = (torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 0.5) * 0.02 / ny * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, device=DEV, generator=g))
    r = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    A = make_tangent_operator("cuda", u, th, p)
    clustered, plain = Multigrid(A.mesh, p, graphs=False), Multigrid(A.mesh, p, graphs=False)
    plain.h.stencil = None
    for mg in (clustered, plain):
        mg.setup(A.moduli, A.code, A.diag)
    # sums in another order: rounding through a few smoothing steps and one dense solve
    for a, b in zip(clustered.levels[:-1], plain.levels[:-1]):
        assert abs(a.lam - b.lam) <= 1e-10 * b.lam
    z, z_ref = clustered(r), plain(r)
    assert rel(z, z_ref) < 1e-10
    assert torch.equal(z, clustered(r))


@pytest.mark.parametrize("gx,gy", [(1, 1), (3, 3), (4, 3), (7, 3), (7, 4), (7, 5), (9, 4), (10, 4), (13, 3), (13, 8)])
def test_coarsest_inverse_around_its_register_tiles(gx, gy):
    """DOFs 8, 32, 40, 64, 80, 96, 100, 110, 112 and 252: every tile size and the global-memory form."""
    n_nodes, n = (gx + 1) * (gy + 1), 2 * (gx + 1) * (gy + 1)
    gen = torch.Generator().manual_seed(gx * 16 + gy)
    B = torch.randn(gx * gy, 8, 8, dtype=torch.float64, generator=gen)
    Kc = B @ B.transpose(1, 2) + 0.5 * torch.eye(8, dtype=torch.float64)          # SPD element matrices
    fix = torch.zeros(n_nodes, dtype=torch.uint8)
    fix[0], fix[n_nodes // 2] = 3, 1
    A = torch.zeros(n, n, dtype=torch.float64)
    for c in range(gx * gy):
        X, Y = divmod(c, gy)
        nodes = [X * (gy + 1) + Y, (X + 1) * (gy + 1) + Y, (X + 1) * (gy + 1) + Y + 1, X * (gy + 1) + Y + 1]
        dofs = [2 * k + i for k in nodes for i in (0, 1)]
        free = torch.tensor([0.0 if (int(fix[d // 2]) >> (d % 2)) & 1 else 1.0 for d in dofs], dtype=torch.float64)
        Kc[c] *= free[:, None] * free[None, :]
        A[torch.tensor(dofs)[:, None], torch.tensor(dofs)[None, :]] += Kc[c]
    for k in range(n_nodes):
        for i in (0, 1):
            if (int(fix[k]) >> i) & 1:
                A[2 * k + i, 2 * k + i] += 1.0
    K = Kc.reshape(gx * gy, 64).t().contiguous().to(DEV)
    fd = fix.to(DEV)
    grid = _lib.MgGrid()
    grid.gx, grid.gy, grid.K, grid.fix = gx, gy, K.data_ptr(), fd.data_ptr()
    Ainv, work = (torch.empty(n, n, dtype=torch.float64, device=DEV) for _ in range(2))
    _lib.call("dfea_mg_dense_inverse", ctypes.byref(grid), ptr(work), ptr(Ainv), stream_handle())
    err = float((Ainv.cpu() @ A - torch.eye(n, dtype=torch.float64)).abs().max())
    cond = float(torch.linalg.cond(A))
    assert err < 64 * n * 2.3e-16 * cond                                          # Gauss-Jordan on an SPD matrix
