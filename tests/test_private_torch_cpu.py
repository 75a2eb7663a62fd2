"""A torch without one of the private functions that the short way into an op asks: calls go through the dispatcher."""
from types import SimpleNamespace

import pytest
import torch

from difffea_b200 import cuda_mesh, ops

PRIVATE = [(torch._C, "_len_torch_dispatch_stack"), (torch._C, "_len_torch_function_stack"), (torch._C, "_get_tracing_state"),
           (torch._C._functorch, "peek_interpreter_stack"), (torch._C._autograd, "_profiler_enabled"),
           (torch.autograd.forward_ad, "_current_level")]


@pytest.mark.parametrize("owner,name", PRIVATE, ids=[n for _, n in PRIVATE])
def test_a_missing_probe_sends_calls_through_the_dispatcher(monkeypatch, owner, name):
    assert ops._PROBES is not None and not ops._observed(())
    monkeypatch.delattr(owner, name)
    assert ops._interpreter_probes() is None
    monkeypatch.setattr(ops, "_PROBES", ops._interpreter_probes())
    assert ops._observed(())


def test_the_stream_without_its_private_function(monkeypatch):
    monkeypatch.setattr(cuda_mesh, "_RAW_STREAM", None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=1234))
    assert cuda_mesh.stream_handle().value == 1234
