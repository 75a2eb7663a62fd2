"""What a request holds on the device at its peak is within the estimate that the engine admits it by."""
import gc

import pytest
import torch

from difffea_b200.serving import Request, hbm_estimate, solve_request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et", ["quad4", "quad9"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("preconditioner", ["jacobi", "block_jacobi", "multigrid"])
def test_peak_is_within_the_estimate(et, precision, preconditioner):
    req = Request(0, et, 800, E=1.0, nu=0.3, load=0.01)
    for _ in range(2):                                   # the second time without one-off allocations
        gc.collect()
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        out = solve_request(req, torch.device("cuda"), precision=precision, preconditioner=preconditioner)
        peak = torch.cuda.max_memory_allocated() - before
        del out
    assert peak <= hbm_estimate(req, precision, preconditioner)
