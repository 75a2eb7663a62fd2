"""
Two threads on one stream (every thread's default), each with its own state on a shared mesh: residual, moduli, diagonal,
node blocks, internal force, fields and reactions are those of the thread's own state, bit for bit, in every call.
"""
import threading

import pytest
import torch

from difffea_b200.operators import compute_block_jacobi, global_residual, make_A_operator_cuda
from difffea_b200.postprocess import compute_fields, internal_force, support_reactions
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu


def _quantities(u, th, p):
    A = make_A_operator_cuda(u, th, p)
    fields = compute_fields(u, th, p)
    live = A.moduli.view(A.mesh.n_q * 5, A.mesh.stride, 2)[:, :A.mesh.n_el]
    return [global_residual(u, th, p), live, A.diag, compute_block_jacobi(u, th, p), internal_force(u, th, p),
            *(fields[k] for k in sorted(fields)), support_reactions(u, th, p), A(u)]


@pytest.mark.parametrize("et,nx,ny", [("quad4", 60, 40), ("quad9", 20, 12)])
def test_threads_on_one_stream_keep_their_scratch(et, nx, ny):
    p = build_rectangle_problem(et, nx, ny, nx / ny, 1.0, load=(0.0, -1e-3), device="cuda")
    states = []
    for seed in (1, 2):
        g = torch.Generator().manual_seed(seed)
        u = ((torch.rand(p["f"].numel(), dtype=torch.float64, generator=g) - 0.5) * 0.02 / ny).cuda() * p["m"]
        th = torch.exp(0.3 * torch.randn(p["conn"].shape[0], dtype=torch.float64, generator=g)).cuda()
        states.append((u, th, [t.clone() for t in _quantities(u, th, p)]))      # before any other thread runs
    wrong, failed, start = [], [], threading.Barrier(2)

    def work(k):
        u, th, alone = states[k]
        try:
            start.wait()
            for i in range(200):
                now = _quantities(u, th, p)
                wrong.extend((k, i, j) for j, (a, b) in enumerate(zip(alone, now)) if not torch.equal(a, b))
        except Exception as e:
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and not wrong, (failed, wrong[:5])
