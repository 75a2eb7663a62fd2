"""
The functional ops called without the dispatcher's layers: the same tensors as through it, and every caller that the
dispatcher would serve (modes, tracing, transforms, autograd, tensors elsewhere) still goes through it.
"""
import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils._python_dispatch import TorchDispatchMode

from difffea_b200 import ops
from difffea_b200.adjoint import compute_implicit_vjp
from difffea_b200.operators import global_residual, make_A_operator_cuda, make_tangent_operator
from difffea_b200.postprocess import compute_fields, support_reactions
from difffea_b200.problem import build_rectangle_problem

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(func.name())
        return func(*args, **(kwargs or {}))


def _state(et="quad4", nx=12, ny=7):
    p = build_rectangle_problem(et, nx, ny, float(nx), float(ny), load=(0.0, -1e-3), device=DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    n = p["f"].numel()
    u = 0.05 * torch.randn(n, dtype=torch.float64, device=DEV, generator=g) * p["m"]
    v = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    th = 0.5 + torch.rand(p["conn"].shape[0], dtype=torch.float64, device=DEV, generator=g)
    return p, u, v, th


def _tensors(r):
    if torch.is_tensor(r):
        return [r]
    if isinstance(r, dict):
        r = list(r.values())
    return [t for x in r for t in _tensors(x)] if isinstance(r, (list, tuple)) else []


def _live(A, C):
    """The moduli of the elements (the slots that pad the last tile are not written)."""
    return C.view(-1, A.mesh.stride, 2)[:, :A.mesh.n_el]


def _moduli(p, u, v, th, name):
    A = make_tangent_operator("cuda", u, th, p)
    return _live(A, getattr(A, name))


CALLS = {
    "tangent_apply": lambda p, u, v, th: make_tangent_operator("cuda", u, th, p)(v),
    "frame_moduli": lambda p, u, v, th: _moduli(p, u, v, th, "moduli"),
    "qp_moduli": lambda p, u, v, th: make_A_operator_cuda(u, th, p, precision="fp32")(v.float()),
    "frame_push_forward": lambda p, u, v, th: _moduli(p, u, v, th, "C"),
    "frame_residual": lambda p, u, v, th: global_residual(u, th, p),
    "frame_sensitivity": lambda p, u, v, th: compute_implicit_vjp(u, th, p, v),
    "frame_all_fields": lambda p, u, v, th: compute_fields(u, th, p),
    "frame_reactions": lambda p, u, v, th: support_reactions(u, th, p),
}


@pytest.mark.parametrize("name", CALLS)
def test_direct_calls_give_the_dispatchers_tensors(name):
    p, u, v, th = _state()
    direct = _tensors(CALLS[name](p, u.clone(), v, th))
    with _Seen() as seen:
        through = _tensors(CALLS[name](p, u.clone(), v, th))
    assert "difffea_b200::" + name in seen.names
    assert direct and len(direct) == len(through)
    for a, b in zip(direct, through):
        assert a.dtype == b.dtype and torch.equal(a, b)


def _outcome(f):
    try:
        r = f()
    except Exception as e:
        return type(e)
    return type(r), r.requires_grad, r.shape, r.device.type


def test_observed_calls_go_through_the_dispatcher():
    p, u, v, th = _state()
    A = make_tangent_operator("cuda", u, th, p)
    op = torch.ops.difffea_b200.tangent_apply
    through = lambda t: op(A.mesh_id, A.moduli, t.contiguous())
    y = through(v)
    assert not ops._observed((A.mesh_id, A.moduli, v))
    w = v.clone().requires_grad_()
    assert ops._observed((A.mesh_id, A.moduli, w))
    assert _outcome(lambda: A(w)) == _outcome(lambda: through(w))
    with torch.no_grad():
        assert torch.equal(A(w), y)
    V = torch.stack([v, 2.0 * v])
    assert _outcome(lambda: torch.func.vmap(A)(V)) == _outcome(lambda: torch.func.vmap(through)(V))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(v.clone(), torch.ones_like(v))
        assert ops._observed((dual,))
        assert _outcome(lambda: A(dual)) == _outcome(lambda: through(dual))
    assert _outcome(lambda: A(v.cpu())) == _outcome(lambda: through(v.cpu()))
    part = torch.nn.Parameter(v.clone(), requires_grad=False)
    assert ops._observed((part,)) and torch.equal(A(part), y)
    z = torch.complex(torch.zeros_like(v), -v).conj().imag       # v under a lazy negation
    assert torch.equal(A(z), y)
    graph = make_fx(lambda t: A(t))(v)
    assert any("tangent_apply" in str(n.target) for n in graph.graph.nodes)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        A(v)
    assert any(e.key == "difffea_b200::tangent_apply" for e in prof.key_averages())
