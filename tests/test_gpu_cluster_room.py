"""
The cluster PCG where fewer blocks than sixteen are to be had (a cap of the caller's, a device that cannot place them): a
smaller cluster where the mesh fits it, else the launch form it was asked for beside.
"""
import pytest
import torch

from difffea_b200.krylov import DevicePCG
from difffea_b200.operators import make_tangent_operator
from difffea_b200.problem import build_rectangle_problem
from golden_utils import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _system(et, nx, ny):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device=DEV)
    g = torch.Generator().manual_seed(7 * nx + ny)
    n = p["f"].numel()
    u = ((torch.rand(n, dtype=torch.float64, generator=g) - 0.5) * 0.02 / ny).to(DEV) * p["m"]
    th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).to(DEV)
    return make_tangent_operator("cuda", u, th, p), torch.randn(n, dtype=torch.float64, generator=g).to(DEV)


def _solve(A, b, form, cap, **kw):
    x = torch.full_like(b, float("nan"))
    h = DevicePCG(A.mesh, A.moduli, A.diag, b.clone(), x, use_graph=2, form=form, moduli="ref", max_blocks=cap, **kw)
    out = x, *h.solve(1e-11, 5000), h.form
    h.close()
    return out


@pytest.mark.parametrize("et,nx,ny", [("quad4", 40, 20), ("quad9", 16, 9), ("tri3", 30, 20), ("tri6", 20, 10)])
@pytest.mark.parametrize("cap", [1, 2, 3, 8, 64])
def test_a_smaller_cluster_solves_alike(et, nx, ny, cap):
    A, b = _system(et, nx, ny)
    x, k, status, form = _solve(A, b, "fused", cap, cluster=True)
    xf, kf, sf, _ = _solve(A, b, "fused", 0)
    # both stop at ||r|| <= 1e-11 ||b|| with rounding apart; the meshes' condition numbers are below 1e5
    assert form == "cluster" and status == sf == "converged" and abs(k - kf) <= 2 and rel(x, xf) < 1e-7


def test_a_mesh_too_large_for_the_blocks_there_are_takes_the_launch_form():
    A, b = _system("quad4", 97, 23)                       # sixteen blocks hold it, one does not
    x, k, status, form = _solve(A, b, "fused", 1, cluster=True)
    want = _solve(A, b, "fused", 1)
    assert form == "fused" and (k, status) == want[1:3] and torch.equal(x, want[0])
    assert _solve(A, b, "fused", 0, cluster=True)[3] == "cluster"
    with pytest.raises(RuntimeError, match="shared memory of a cluster"):
        _solve(A, b, "cluster", 1)
