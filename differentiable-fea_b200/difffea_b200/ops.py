"""
PyTorch custom ops over the C ABI (namespace ``difffea_b200``).

Each op is a thin shim: it allocates its outputs through torch's caching allocator and calls one
``extern "C"`` launcher on torch's current stream.  The mesh is referred to by an integer id
(``register_mesh``) because a mesh is a bundle of device arrays, not one tensor.

    torch.ops.difffea_b200.qp_moduli(mesh_id, u, theta, model, scalable, mat_p, fp32, with_diag) -> (C, diag)
    torch.ops.difffea_b200.tangent_apply(mesh_id, C, v, gather=False) -> y   kernel (b)
    torch.ops.difffea_b200.residual(mesh_id, u, theta, model, scalable, mat_p, f, load_factor) -> (R, |R|^2, energy)
    torch.ops.difffea_b200.element_sensitivity(mesh_id, u, lam, model, scalable, mat_p) -> g      kernel (d)
    torch.ops.difffea_b200.element_fields(mesh_id, u, theta, model, scalable, mat_p) -> (7, n_el)
    torch.ops.difffea_b200.node_fields(mesh_id, elem) -> (6, N)
    torch.ops.difffea_b200.internal_force(mesh_id, u, theta, model, scalable, mat_p) -> R_int (2N,)
    torch.ops.difffea_b200.pcg_solve(pcg_id, x, rtol, max_iter) -> [iterations, status]      kernel (c)
    torch.ops.difffea_b200.mg_setup(mg_id, C, moduli_code, diag) -> lambda_max per smoothed level
    torch.ops.difffea_b200.mg_vcycle(mg_id, C, moduli_code, r) -> z
    torch.ops.difffea_b200.mg_pcg(mg_id, C, moduli_code, b, x, rtol, max_iter) -> [iterations, status]
    torch.ops.difffea_b200.newton_solve(ws_id, theta, n_load_steps, tol, max_newton, max_cutbacks,
                                        pcg_max_iter) -> (u, [converged, load factor, Newton, CG, cut-backs])
the same on a mesh with a frame (CudaMesh.ensure_frame), in one element pass and one node pass:
    torch.ops.difffea_b200.frame_moduli / frame_residual / frame_internal_force / frame_sensitivity / frame_fields
    torch.ops.difffea_b200.frame_all_fields / frame_reactions (compute_fields and support_reactions whole)
    torch.ops.difffea_b200.frame_push_forward(mesh_id, C) -> physical moduli
    torch.ops.difffea_b200.frame_residual_out / frame_moduli_out (caller buffers)
and three forms that write into caller buffers, for the solver's preallocated workspace:
    torch.ops.difffea_b200.residual_out(mesh_id, u, theta, model, scalable, mat_p, f, load_factor, R!, scal!, energy)
    torch.ops.difffea_b200.qp_moduli_out(mesh_id, u, theta, model, scalable, mat_p, C!, moduli_code, diag!, blocks!)
    torch.ops.difffea_b200.add_scaled_out(a, alpha, b, out!)                                  out = a + alpha b

The material is (model, scalable, mat_p): the fields of the C ABI's ``dfea_material``
(``material_args`` turns a ``_lib.Material`` into them).  Solver handles -- a device PCG bound to its
buffers (krylov.DevicePCG), a multigrid hierarchy (multigrid.Multigrid), a Newton workspace
(workspace.NewtonWorkspace) -- are referred to by integer ids (``register_handle``) like meshes; the ops that
run them read the buffers the handle is bound to and write the tensors they declare as mutated.
"""
import weakref
from typing import Optional

import torch

from difffea_b200 import _lib
from difffea_b200.cuda_mesh import ptr, stream_handle
from difffea_b200.materials import device_material, get_material, material_of

_MESHES = weakref.WeakValueDictionary()


def register_mesh(mesh):
    """Integer handle of a CudaMesh for the custom ops (kept while the mesh is alive)."""
    key = id(mesh)
    _MESHES[key] = mesh
    return key


_HANDLES = weakref.WeakValueDictionary()


def register_handle(obj):
    """Integer id of a solver handle (DevicePCG, Multigrid, NewtonWorkspace) for the custom ops."""
    key = id(obj)
    _HANDLES[key] = obj
    return key


def _handle(handle_id):
    obj = _HANDLES.get(handle_id)
    if obj is None:
        raise RuntimeError(f"unknown or released solver handle {handle_id}")
    return obj


def _mesh(mesh_id):
    mesh = _MESHES.get(mesh_id)
    if mesh is None:
        raise RuntimeError(f"unknown or released mesh id {mesh_id}")
    return mesh


def _functional_op(name):
    """Register a custom op that mutates nothing; its implementation stays at hand for ``run``."""
    def register(fn):
        op = torch.library.custom_op("difffea_b200::" + name, mutates_args=(), device_types="cuda")(fn)
        op.implementation = fn
        return op
    return register


def _interpreter_probes():
    """The functions of torch that tell _observed what lies on the dispatcher's stacks; None if this torch lacks one."""
    try:
        torch.autograd.forward_ad._current_level
        return (torch.compiler.is_compiling, torch._C._len_torch_dispatch_stack, torch._C._len_torch_function_stack,
                torch._C._autograd._profiler_enabled, torch._C._functorch.peek_interpreter_stack, torch._C._get_tracing_state)
    except AttributeError:
        return None


_PROBES = _interpreter_probes()


def _observed(args):
    """True if the dispatcher has something to do between a call of a functional op and its CUDA implementation: a trace,
    a mode, a functorch or forward-mode level, the profiler, autograd, a tensor subclass, another device.  Also where
    torch does not say: its probes are private."""
    if _PROBES is None:
        return True
    compiling, modes, functions, profiler, functorch, tracing = _PROBES
    if (compiling() or modes() or functions() or functorch() is not None or torch.autograd.forward_ad._current_level >= 0
            or tracing() is not None or profiler()):
        return True
    for t in args:
        if isinstance(t, torch.Tensor) and (type(t) is not torch.Tensor or t.requires_grad or not t.is_cuda or t.is_neg()):
            return True
    return False


def run(op, *args):
    """op(*args); where nothing observes the call, its implementation without the dispatcher's layers (autograd, redispatch
    and Python wrappers: 13 of the 31 us of a small product, whose two launches take 5)."""
    return op(*args) if _observed(args) else op.implementation(*args)


def material_args(mat):
    """(model, scalable, mat_p) of a ``_lib.Material``: the material arguments of the ops."""
    return int(mat.model), int(mat.scalable), [float(x) for x in mat.p]


def _material(model, scalable, mat_p):
    out = _lib.Material()
    out.model, out.scalable = model, scalable
    if len(mat_p) > _lib.MAX_MAT_PARAMS:
        raise ValueError("too many material parameters")
    for k, x in enumerate(mat_p):
        out.p[k] = x
    return out


def _f64(t, mesh, n=None):
    if t.device != mesh.device or t.dtype != torch.float64 or not t.is_contiguous():
        raise ValueError("expected a contiguous float64 tensor on the mesh's device")
    if n is not None and t.numel() != n:
        raise ValueError(f"expected {n} entries, got {t.numel()}")
    return t


@_functional_op("qp_moduli")
def qp_moduli(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
              fp32: bool, with_diag: bool) -> tuple[torch.Tensor, torch.Tensor]:
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    _f64(theta, mesh, mesh.n_el)
    C = torch.empty(mesh.moduli_numel(), dtype=torch.float32 if fp32 else torch.float64, device=mesh.device)
    diag = torch.empty(mesh.n_dof if with_diag else 0, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_qp_moduli_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p), ptr(C),
              _lib.DFEA_F32 if fp32 else _lib.DFEA_F64, ptr(diag) if with_diag else ptr(None), ptr(None),
              stream_handle())
    return C, diag


@qp_moduli.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, fp32, with_diag):
    mesh = _mesh(mesh_id)
    C = u.new_empty(mesh.moduli_numel(), dtype=torch.float32 if fp32 else torch.float64)
    return C, u.new_empty(mesh.n_dof if with_diag else 0)


@_functional_op("tangent_apply")
def tangent_apply(mesh_id: int, C: torch.Tensor, v: torch.Tensor, gather: bool = False) -> torch.Tensor:
    """A(v); ``gather``: physical moduli too in the gather form, which needs the mesh's node incidence."""
    mesh = _mesh(mesh_id)
    fp32 = v.dtype == torch.float32
    if C.dtype == torch.float32:
        mesh.ensure_grad32()
    if v.device != mesh.device or not v.is_contiguous() or v.numel() != mesh.n_dof:
        raise ValueError("v must be a contiguous (2N,) tensor on the mesh's device")
    y = torch.empty_like(v)
    if C.numel() == mesh.moduli_numel_ref():
        # reference-frame moduli: the gather form, with its element results in scratch of this call
        view, keep = mesh.gather_view()
        fe = torch.empty(int(_lib.load().dfea_gather_work_bytes(mesh.view_ref, _lib.DFEA_F64)), dtype=torch.uint8,
                         device=mesh.device)
        code = _lib.DFEA_F64REF if C.dtype == torch.float64 else _lib.DFEA_F32REF
        _lib.call("dfea_tangent_apply_gather", view, ptr(C), code, ptr(v), ptr(y),
                  _lib.DFEA_F32 if fp32 else _lib.DFEA_F64, ptr(fe), stream_handle())
        return y
    dt = _lib.DFEA_F32 if fp32 else _lib.DFEA_F64
    cdt = _lib.DFEA_F32 if C.dtype == torch.float32 else _lib.DFEA_F64
    if gather:
        view, keep = mesh.gather_view()
        # two launches, at every size: FP32 colour / gather us: 65k Tri6 54 / 17, 90k Q4 43 / 13, 640k Q4 74 / 63, 810k Q9
        # 283 / 222, 1M Q4 109 / 97, 4M Q4 356 / 351, 3.9M Tri3 171 / 144
        fe = torch.empty(int(_lib.load().dfea_gather_work_bytes(mesh.view_ref, dt)), dtype=torch.uint8, device=mesh.device)
        _lib.call("dfea_tangent_apply_gather", view, ptr(C), cdt, ptr(v), ptr(y), dt, ptr(fe), stream_handle())
        return y
    _lib.call("dfea_tangent_apply", mesh.view_ref, ptr(C), cdt, ptr(v), ptr(y), dt, stream_handle())
    return y


@tangent_apply.register_fake
def _(mesh_id, C, v, gather=False):
    return torch.empty_like(v)


@_functional_op("residual")
def residual(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
             f: torch.Tensor, load_factor: float) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    _f64(theta, mesh, mesh.n_el)
    _f64(f, mesh, mesh.n_dof)
    R = torch.empty_like(u)
    out = torch.empty(2, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_residual_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p), ptr(f),
              load_factor, ptr(R), ptr(out), ptr(out[1:]), ptr(mesh.reduce_work()), stream_handle())
    return R, out[0].clone(), out[1].clone()


@residual.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, f, load_factor):
    return torch.empty_like(u), u.new_empty(()), u.new_empty(())


@_functional_op("element_sensitivity")
def element_sensitivity(mesh_id: int, u: torch.Tensor, lam: torch.Tensor, model: int, scalable: int,
                        mat_p: list[float]) -> torch.Tensor:
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    _f64(lam, mesh, mesh.n_dof)
    g = torch.empty(mesh.n_el, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_element_sensitivity_mat", mesh.view_ref, ptr(u), ptr(lam), _material(model, scalable, mat_p),
              ptr(g), stream_handle())
    return g


@element_sensitivity.register_fake
def _(mesh_id, u, lam, model, scalable, mat_p):
    return u.new_empty(_mesh(mesh_id).n_el)


# ---------------------------------------------------------------------------------------------
# post-processing
# ---------------------------------------------------------------------------------------------
@_functional_op("element_fields")
def element_fields(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int,
                   mat_p: list[float]) -> torch.Tensor:
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    _f64(theta, mesh, mesh.n_el)
    out = torch.empty(7, mesh.n_el, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_element_fields_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p),
              ptr(out), stream_handle())
    return out


@element_fields.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p):
    return u.new_empty(7, _mesh(mesh_id).n_el)


@torch.library.custom_op("difffea_b200::node_fields", mutates_args=(), device_types="cuda")
def node_fields(mesh_id: int, elem: torch.Tensor) -> torch.Tensor:
    mesh = _mesh(mesh_id)
    if elem.shape != (7, mesh.n_el) or elem.dtype != torch.float64 or not elem.is_contiguous():
        raise ValueError("elem must be the contiguous (7, n_el) float64 output of element_fields")
    view, keep = mesh.gather_view()
    out = torch.empty(6, mesh.n_nodes, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_node_fields", view, ptr(elem), ptr(out), stream_handle())
    return out


@node_fields.register_fake
def _(mesh_id, elem):
    return elem.new_empty(6, _mesh(mesh_id).n_nodes)


@_functional_op("internal_force")
def internal_force(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int,
                   mat_p: list[float]) -> torch.Tensor:
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    _f64(theta, mesh, mesh.n_el)
    R = torch.empty(mesh.n_dof, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_internal_force_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p),
              ptr(R), stream_handle())
    return R


@internal_force.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p):
    return torch.empty_like(u)


# ---------------------------------------------------------------------------------------------
# the same quantities on a mesh with a frame (CudaMesh.ensure_frame): one element pass and one node pass
# ---------------------------------------------------------------------------------------------
def frame_material(params, linear_only=False):
    """
    (model, scalable, mat_p, p_dev, scalable_dev) of a problem for the frame_* ops.  A material whose parameters and
    flags lie on the device is passed as those tensors and read by the kernels: copying it to the host first makes
    every call wait for the GPU (six blocking reads in one linearisation).  ``linear_only``: the op looks at the flags
    on the host unless theta may scale any parameter of the model.
    """
    name, p0, scalable = material_of(params)
    mat = get_material(name)
    n = len(mat["param_names"])
    if (torch.is_tensor(p0) and torch.is_tensor(scalable) and p0.is_cuda
            and p0.device == scalable.device == params["conn"].device
            and p0.dtype == torch.float64 and scalable.dtype == torch.bool and p0.shape == scalable.shape == (n,)
            and p0.is_contiguous() and scalable.is_contiguous()
            and (not linear_only or name in ("neo_hookean", "mooney_rivlin", "saint_venant"))):
        return mat["model"], 0, [], p0.detach(), scalable
    return (*material_args(device_material(params)), None, None)


def _frame_mesh(mesh_id, u, theta=None):
    mesh = _mesh(mesh_id)
    _f64(u, mesh, mesh.n_dof)
    if theta is not None:
        _f64(theta, mesh, mesh.n_el)
    if mesh.frame is None:
        raise ValueError("the mesh has no frame (CudaMesh.ensure_frame)")
    return mesh


def _frame_args(mesh, model, scalable, mat_p, p_dev=None, s_dev=None):
    for t in (p_dev, s_dev):
        if t is not None and t.device != mesh.device:
            raise ValueError("the material's parameters must be on the mesh's device")
    return _material(model, scalable, mat_p), ptr(p_dev), ptr(s_dev)


@_functional_op("frame_moduli")
def frame_moduli(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                 p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor], with_moduli: bool,
                 with_blocks: bool) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """FP64 reference-frame moduli (empty without with_moduli), Jacobi diagonal, inverse node blocks (or empty)."""
    mesh = _frame_mesh(mesh_id, u, theta)
    f64 = dict(dtype=torch.float64, device=mesh.device)
    C = torch.empty(mesh.moduli_numel_ref() if with_moduli else 0, **f64)
    diag = torch.empty(mesh.n_dof, **f64)
    blocks = torch.empty(2 * mesh.n_dof if with_blocks else 0, **f64)
    work = mesh.frame_work()        # a local: the call's own until its launches are made
    _lib.call("dfea_frame_moduli", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev),
              ptr(C if with_moduli else None), _lib.DFEA_F64REF, ptr(diag), ptr(blocks if with_blocks else None),
              ptr(work), stream_handle())
    return C, diag, blocks


@frame_moduli.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev, with_moduli, with_blocks):
    mesh = _mesh(mesh_id)
    return (u.new_empty(mesh.moduli_numel_ref() if with_moduli else 0), u.new_empty(mesh.n_dof),
            u.new_empty(2 * mesh.n_dof if with_blocks else 0))


@_functional_op("frame_residual")
def frame_residual(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                   p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor], f: torch.Tensor,
                   load_factor: float, scalars: bool) -> tuple[torch.Tensor, torch.Tensor]:
    """R and, with scalars, (|R|^2, strain energy) on the device (else empty)."""
    mesh = _frame_mesh(mesh_id, u, theta)
    _f64(f, mesh, mesh.n_dof)
    R = torch.empty_like(u)
    out = torch.empty(2 if scalars else 0, dtype=torch.float64, device=mesh.device)
    work = mesh.frame_work()        # a local: the call's own until its launches are made
    _lib.call("dfea_frame_residual", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev), ptr(f), float(load_factor), ptr(R),
              ptr(out if scalars else None), ptr(out[1:] if scalars else None),
              ptr(work), stream_handle())
    return R, out


@frame_residual.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev, f, load_factor, scalars):
    return torch.empty_like(u), u.new_empty(2 if scalars else 0)


@_functional_op("frame_internal_force")
def frame_internal_force(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int,
                         mat_p: list[float],
                 p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor]) -> torch.Tensor:
    mesh = _frame_mesh(mesh_id, u, theta)
    R = torch.empty(mesh.n_dof, dtype=torch.float64, device=mesh.device)
    work = mesh.frame_work()        # a local: the call's own until its launches are made
    _lib.call("dfea_frame_internal_force", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev),
              ptr(R), ptr(work), stream_handle())
    return R


@frame_internal_force.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev):
    return u.new_empty(_mesh(mesh_id).n_dof)


@_functional_op("frame_sensitivity")
def frame_sensitivity(mesh_id: int, u: torch.Tensor, lam: torch.Tensor, model: int, scalable: int,
                      mat_p: list[float],
                 p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor]) -> torch.Tensor:
    mesh = _frame_mesh(mesh_id, u)
    _f64(lam, mesh, mesh.n_dof)
    g = torch.empty(mesh.n_el, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_frame_sensitivity", mesh.view_ref, ptr(u), ptr(lam),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev), ptr(g),
              stream_handle())
    return g


@frame_sensitivity.register_fake
def _(mesh_id, u, lam, model, scalable, mat_p, p_dev, s_dev):
    return u.new_empty(_mesh(mesh_id).n_el)


@_functional_op("frame_fields")
def frame_fields(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int,
                 mat_p: list[float],
                 p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor]) -> torch.Tensor:
    mesh = _frame_mesh(mesh_id, u, theta)
    out = torch.empty(7, mesh.n_el, dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_frame_fields", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev), ptr(out),
              stream_handle())
    return out


@frame_fields.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev):
    return u.new_empty(7, _mesh(mesh_id).n_el)


@_functional_op("frame_all_fields")
def frame_all_fields(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                     p_dev: Optional[torch.Tensor],
                     s_dev: Optional[torch.Tensor]) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Element rows (7, n_el), nodal rows (7, N; the last is |u|) and (strain energy, smallest J)."""
    mesh = _frame_mesh(mesh_id, u, theta)
    f64 = dict(dtype=torch.float64, device=mesh.device)
    el, nodal, scal = torch.empty(7, mesh.n_el, **f64), torch.empty(7, mesh.n_nodes, **f64), torch.empty(2, **f64)
    work = mesh.frame_work()        # a local: the call's own until its launches are made
    _lib.call("dfea_frame_all_fields", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev), ptr(el), ptr(nodal), ptr(scal),
              ptr(work), stream_handle())
    return el, nodal, scal


@frame_all_fields.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev):
    mesh = _mesh(mesh_id)
    return u.new_empty(7, mesh.n_el), u.new_empty(7, mesh.n_nodes), u.new_empty(2)


@_functional_op("frame_reactions")
def frame_reactions(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                    p_dev: Optional[torch.Tensor], s_dev: Optional[torch.Tensor], fixed: torch.Tensor) -> torch.Tensor:
    mesh = _frame_mesh(mesh_id, u, theta)
    if fixed.dtype != torch.bool or fixed.numel() != mesh.n_dof or not fixed.is_contiguous() or fixed.device != mesh.device:
        raise ValueError("fixed must be the contiguous (2N,) bool flags on the mesh's device")
    out = torch.empty(2, dtype=torch.float64, device=mesh.device)
    work = mesh.frame_work()        # a local: the call's own until its launches are made
    _lib.call("dfea_frame_reactions", mesh.view_ref, ptr(u), ptr(theta),
              *_frame_args(mesh, model, scalable, mat_p, p_dev, s_dev), ptr(fixed), ptr(out), ptr(work),
              stream_handle())
    return out


@frame_reactions.register_fake
def _(mesh_id, u, theta, model, scalable, mat_p, p_dev, s_dev, fixed):
    return u.new_empty(2)


@_functional_op("frame_push_forward")
def frame_push_forward(mesh_id: int, C: torch.Tensor) -> torch.Tensor:
    """The 16 physical moduli per Gauss point (DFEA_F64 layout) of FP64 reference-frame ones."""
    mesh = _mesh(mesh_id)
    _f64(C, mesh, mesh.moduli_numel_ref())
    out = torch.zeros(mesh.moduli_numel(), dtype=torch.float64, device=mesh.device)
    _lib.call("dfea_frame_push_forward", mesh.view_ref, ptr(C), ptr(out), stream_handle())
    return out


@frame_push_forward.register_fake
def _(mesh_id, C):
    return C.new_empty(_mesh(mesh_id).moduli_numel())


@torch.library.custom_op("difffea_b200::frame_residual_out", mutates_args=("R", "scal", "work"), device_types="cuda")
def frame_residual_out(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                       f: torch.Tensor, load_factor: float, R: torch.Tensor, scal: torch.Tensor, energy: bool,
                       work: torch.Tensor) -> None:
    """residual_out on the frame, with its scratch in ``work`` (frame_work of the mesh)."""
    mesh = _frame_mesh(mesh_id, u, theta)
    _f64(R, mesh, mesh.n_dof)
    if scal.dtype != torch.float64 or scal.numel() < 2 or scal.device != mesh.device:
        raise ValueError("scal must hold at least 2 float64 entries on the mesh's device")
    _lib.call("dfea_frame_residual", mesh.view_ref, ptr(u), ptr(theta), *_frame_args(mesh, model, scalable, mat_p), ptr(f),
              float(load_factor), ptr(R), ptr(scal), ptr(scal[1:] if energy else None), ptr(work), stream_handle())


@torch.library.custom_op("difffea_b200::frame_moduli_out", mutates_args=("C", "diag", "blocks", "work"),
                         device_types="cuda")
def frame_moduli_out(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                     C: torch.Tensor, moduli_code: int, diag: torch.Tensor, blocks: torch.Tensor,
                     work: torch.Tensor) -> None:
    """Reference-frame moduli into C, the Jacobi diagonal into diag and, when not empty, the inverse node blocks."""
    mesh = _frame_mesh(mesh_id, u, theta)
    _lib.call("dfea_frame_moduli", mesh.view_ref, ptr(u), ptr(theta), *_frame_args(mesh, model, scalable, mat_p), ptr(C),
              int(moduli_code), ptr(diag), ptr(blocks if blocks.numel() else None), ptr(work), stream_handle())


# ---------------------------------------------------------------------------------------------
# solvers
# ---------------------------------------------------------------------------------------------
def _status_tensor(iters, status):
    return torch.tensor([int(iters), int(status)], dtype=torch.int32)


@torch.library.custom_op("difffea_b200::pcg_solve", mutates_args=("x",), device_types="cuda")
def pcg_solve(pcg_id: int, x: torch.Tensor, rtol: float, max_iter: int) -> torch.Tensor:
    """Run a bound device PCG (kernel (c)) on its right-hand side buffer; x must be its solution buffer."""
    import ctypes
    h = _handle(pcg_id)
    if x.data_ptr() != h.x.data_ptr():
        raise ValueError("x must be the solution buffer the PCG handle is bound to")
    iters, status = ctypes.c_int32(0), ctypes.c_int32(0)
    with torch.cuda.device(h.mesh.device):
        _lib.call("dfea_pcg_solve", h._h, float(rtol), int(max_iter), ctypes.byref(iters), ctypes.byref(status),
                  stream_handle())
    return _status_tensor(iters.value, status.value)


@pcg_solve.register_fake
def _(pcg_id, x, rtol, max_iter):
    return torch.empty(2, dtype=torch.int32)


@torch.library.custom_op("difffea_b200::mg_setup", mutates_args=(), device_types="cuda")
def mg_setup(mg_id: int, C: torch.Tensor, moduli_code: int, diag: torch.Tensor) -> torch.Tensor:
    """Set a multigrid hierarchy up at a linearisation (coarse operators, smoother bounds, coarsest inverse)."""
    mg = _handle(mg_id)
    _lib.call("dfea_mg_setup", mg.mesh.view_ref, mg.ref, ptr(C), int(moduli_code), ptr(diag), stream_handle())
    return torch.tensor([float(mg.h.lam[l]) for l in range(len(mg.levels) - 1)], dtype=torch.float64)


@mg_setup.register_fake
def _(mg_id, C, moduli_code, diag):
    return torch.empty(len(_handle(mg_id).levels) - 1, dtype=torch.float64)


@torch.library.custom_op("difffea_b200::mg_vcycle", mutates_args=(), device_types="cuda")
def mg_vcycle(mg_id: int, C: torch.Tensor, moduli_code: int, r: torch.Tensor) -> torch.Tensor:
    mg = _handle(mg_id)
    _f64(r, mg.mesh, mg.mesh.n_dof)
    z = torch.empty_like(r)
    _lib.call("dfea_mg_vcycle", mg.mesh.view_ref, mg.ref, ptr(C), int(moduli_code), ptr(r), ptr(z), stream_handle())
    return z


@mg_vcycle.register_fake
def _(mg_id, C, moduli_code, r):
    return torch.empty_like(r)


@torch.library.custom_op("difffea_b200::mg_pcg", mutates_args=("x",), device_types="cuda")
def mg_pcg(mg_id: int, C: torch.Tensor, moduli_code: int, b: torch.Tensor, x: torch.Tensor, rtol: float,
           max_iter: int) -> torch.Tensor:
    import ctypes
    mg = _handle(mg_id)
    _f64(b, mg.mesh, mg.mesh.n_dof)
    _f64(x, mg.mesh, mg.mesh.n_dof)
    it, st = ctypes.c_int32(0), ctypes.c_int32(0)
    _lib.call("dfea_mg_pcg", mg.mesh.view_ref, mg.ref, ptr(C), int(moduli_code), ptr(b), ptr(x), float(rtol),
              int(max_iter), ctypes.byref(it), ctypes.byref(st), stream_handle())
    return _status_tensor(it.value, st.value)


@mg_pcg.register_fake
def _(mg_id, C, moduli_code, b, x, rtol, max_iter):
    return torch.empty(2, dtype=torch.int32)


@torch.library.custom_op("difffea_b200::newton_solve", mutates_args=(), device_types="cuda")
def newton_solve(ws_id: int, theta: torch.Tensor, n_load_steps: int, tol: float, max_newton: int, max_cutbacks: int,
                 pcg_max_iter: int) -> tuple[torch.Tensor, torch.Tensor]:
    """One complete Newton-Krylov solve by the library's C++ driver on a workspace's buffers."""
    import ctypes
    ws = _handle(ws_id)
    nw, u = ws._native_args(theta)
    info = _lib.NewtonInfo()
    _lib.call("dfea_newton_solve", ctypes.byref(nw), int(n_load_steps), float(tol), int(max_newton), int(max_cutbacks),
              int(pcg_max_iter), ctypes.byref(info), ws._records, ws.MAX_RECORDS, stream_handle())
    stats = torch.tensor([info.converged, info.load_factor, info.total_newton, info.total_cg, info.n_cutbacks,
                          info.n_records], dtype=torch.float64)
    return u, stats


@newton_solve.register_fake
def _(ws_id, theta, n_load_steps, tol, max_newton, max_cutbacks, pcg_max_iter):
    ws = _handle(ws_id)
    return theta.new_empty(ws.mesh.n_dof), torch.empty(6, dtype=torch.float64)


# ---------------------------------------------------------------------------------------------
# the solver workspace's calls, writing into its buffers
# ---------------------------------------------------------------------------------------------
@torch.library.custom_op("difffea_b200::residual_out", mutates_args=("R", "scal"), device_types="cuda")
def residual_out(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                 f: torch.Tensor, load_factor: float, R: torch.Tensor, scal: torch.Tensor, energy: bool) -> None:
    """R = m (R_int(u) - load_factor f); scal[0] = |R|^2 and, with energy, scal[1] = the strain energy."""
    mesh = _mesh(mesh_id)
    _f64(R, mesh, mesh.n_dof)
    if scal.dtype != torch.float64 or scal.numel() < 2 or scal.device != mesh.device:
        raise ValueError("scal must hold at least 2 float64 entries on the mesh's device")
    _lib.call("dfea_residual_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p), ptr(f),
              float(load_factor), ptr(R), ptr(scal), ptr(scal[1:]) if energy else ptr(None),
              ptr(mesh.reduce_work()), stream_handle())


@torch.library.custom_op("difffea_b200::qp_moduli_out", mutates_args=("C", "diag", "blocks"), device_types="cuda")
def qp_moduli_out(mesh_id: int, u: torch.Tensor, theta: torch.Tensor, model: int, scalable: int, mat_p: list[float],
                  C: torch.Tensor, moduli_code: int, diag: torch.Tensor, blocks: torch.Tensor) -> None:
    """Kernel (a) into C (moduli_code layout; empty: the diagonal alone), diag and, when not empty, the inverse
    2x2 node blocks of block-Jacobi."""
    mesh = _mesh(mesh_id)
    _lib.call("dfea_qp_moduli_mat", mesh.view_ref, ptr(u), ptr(theta), _material(model, scalable, mat_p),
              ptr(C) if C.numel() else ptr(None), int(moduli_code), ptr(diag) if diag.numel() else ptr(None),
              ptr(blocks) if blocks.numel() else ptr(None), stream_handle())


@torch.library.custom_op("difffea_b200::add_scaled_out", mutates_args=("out",), device_types="cuda")
def add_scaled_out(a: torch.Tensor, alpha: float, b: torch.Tensor, out: torch.Tensor) -> None:
    """out = a + alpha b (float64): the Newton trial state of the line search."""
    for t in (a, b, out):
        if t.dtype != torch.float64 or not t.is_contiguous() or t.numel() != a.numel() or t.device != a.device:
            raise ValueError("add_scaled_out: contiguous float64 tensors of one size on one device")
    _lib.call("dfea_add_scaled", a.numel(), ptr(a), float(alpha), ptr(b), ptr(out), stream_handle())
