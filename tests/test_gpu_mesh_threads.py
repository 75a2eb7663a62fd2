"""
A mesh that nothing has used yet, used by several threads at once, each on a stream of its own: whichever thread builds the
incidence, the FP32 gradients and the frame, all of them read finished arrays.
"""
import threading

import pytest
import torch

from difffea_b200.cuda_mesh import cuda_mesh
from difffea_b200.operators import global_residual, make_A_operator_cuda
from difffea_b200.postprocess import compute_fields
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu
CALLS = [lambda u, th, p: make_A_operator_cuda(u, th, p, "fp32")(u.float()), lambda u, th, p: make_A_operator_cuda(u, th, p)(u),
         global_residual, lambda u, th, p: compute_fields(u, th, p)["mises_n"]]


@pytest.mark.parametrize("et,nx,ny", [("quad4", 400, 300), ("tri6", 120, 90)])
def test_first_use_from_several_streams(et, nx, ny):
    g = torch.Generator().manual_seed(nx)
    for _ in range(3):
        p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device="cuda", build_on_device=True)
        cuda_mesh(p)                                     # packed, nothing built on demand yet
        u = ((torch.rand(p["f"].numel(), dtype=torch.float64, generator=g) - 0.5) * 0.02 / ny).cuda() * p["m"]
        th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).cuda()
        torch.cuda.synchronize()
        out, failed, start = [None] * len(CALLS), [], threading.Barrier(len(CALLS))

        def work(k):
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    start.wait()
                    out[k] = CALLS[k](u, th, p)
                    torch.cuda.current_stream().synchronize()
            except Exception as e:
                failed.append(repr(e))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(CALLS))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed, failed
        for k, call in enumerate(CALLS):
            assert torch.equal(out[k], call(u, th, p)), k
