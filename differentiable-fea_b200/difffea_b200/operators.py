"""
Residual, tangent-operator and preconditioner closures on the GPU (the reference's operators.py API).

    global_residual(u, theta, params, load_factor=1.0)          operators.py:159-220
    make_tangent_operator(kind, u, theta, params)               operators.py:415-435, kind "cuda" / "auto"
    make_AT_operator(u, theta, params)                          operators.py:441-471
    compute_jacobi_diagonal / make_jacobi_preconditioner        operators.py:477-570
    make_preconditioner(kind, u, theta, params)                 operators.py:702-710, "jacobi" / "block_jacobi" /
                                                                "multigrid" (structured quad meshes, multigrid.py)
    make_block_jacobi_preconditioner(u, theta, params)          operators.py:586-625
    precompute_geometry(params)                                 operators.py:85-120

Every closure has the reference's semantics -- A(v) = m * J(u)(m * v) + (1 - m) * v, symmetric, the
identity on fixed DOFs -- and runs on the device of ``u`` through the kernels of libdifffea_b200.so.
``"cuda"`` is the stored-moduli variant: kernel (a) evaluates the Gauss-point moduli C once per
linearisation point, kernel (b) applies them.  The reference's own variants (jvp, linearize, qp, qp_ew)
are PyTorch programs of the reference package and are not re-implemented here.
"""
import weakref

import torch

from difffea_b200 import _lib, ops
from difffea_b200.cuda_mesh import _require_cuda, cuda_mesh
from difffea_b200.materials import device_material
from difffea_b200.problem import precompute_geometry  # noqa: F401  (re-exported, as in the reference)

TANGENT_OPERATORS = ("auto", "cuda")
REFERENCE_TANGENT_VARIANTS = ("jvp", "linearize", "qp", "qp_ew")
PRECONDITIONERS = ("jacobi", "block_jacobi", "multigrid")


def _prepare(u, theta, params):
    _require_cuda(u, theta)
    mesh = cuda_mesh(params)
    if u.device != mesh.device:
        raise RuntimeError("u and params must be on the same device")
    return mesh, ops.register_mesh(mesh)


def _f64c(t):
    return t.detach().to(torch.float64).contiguous()


# ---------------------------------------------------------------------------------------------
# residual
# ---------------------------------------------------------------------------------------------
def global_residual(u, theta, params, load_factor=1.0):
    """R(u) = m * (R_int(u, theta) - load_factor * f), shape (2N,)."""
    return _residual(u, theta, params, load_factor, False)[0]


def _residual(u, theta, params, load_factor, scalars):
    """(R, (|R|^2, strain energy) on the device with ``scalars``)."""
    mesh, mid = _prepare(u, theta, params)
    u, theta, f = _f64c(u), _f64c(theta), _f64c(params["f"])
    if mesh.ensure_frame():
        return ops.run(ops.frame_residual, mid, u, theta, *ops.frame_material(params), f, float(load_factor), scalars)
    R, n2, W = ops.run(ops.residual, mid, u, theta, *ops.material_args(device_material(params)), f, float(load_factor))
    return R, (n2, W)


def residual_and_norm(u, theta, params, load_factor=1.0):
    """(R, ||R||) with the norm reduced on the device in fixed order (one scalar read-back)."""
    R, (n2, _) = _residual(u, theta, params, load_factor, True)
    return R, float(n2) ** 0.5


def strain_energy(u, theta, params):
    """Total strain energy sum_e sum_q w detJ psi(F), the ``strain_energy`` of compute_fields."""
    return _residual(u, theta, params, 0.0, True)[1][1]


# ---------------------------------------------------------------------------------------------
# tangent operator
# ---------------------------------------------------------------------------------------------
def _versions(*tensors):
    """The tensors' version counters (0 for what is no tensor), or None where torch keeps none (inference mode)."""
    try:
        return tuple([t._version for t in tensors])
    except AttributeError:
        return _versions(*(t for t in tensors if torch.is_tensor(t)))
    except RuntimeError:
        return None


class _Linearisation:
    """
    The point (u, theta, material) an operator or preconditioner was made at: what its physical moduli, diagonal or
    blocks are computed from when a solve asks for them later.  Holds the tensors themselves; ``unchanged`` is False
    once one of them was written to (or where torch keeps no version of it).
    """
    __slots__ = ("u", "theta", "keys", "values", "versions", "__weakref__")
    MATERIAL, LEGACY = ("mat_p", "mat_scalable", "material"), ("nodes", "mu0", "lmbda0")

    def __init__(self, u, theta, params):
        self.u = u.detach() if u.requires_grad else u
        self.theta = theta.detach() if theta.requires_grad else theta
        self.keys = self.MATERIAL if "material" in params else self.LEGACY
        a, b, c = self.keys
        self.values = a, b, c = params[a], params[b], params[c]
        self.versions = _versions(u, theta, a, b) if c.__class__ is str else _versions(u, theta, a, b, c)

    @property
    def unchanged(self):
        a, b, c = self.values
        now = _versions(self.u, self.theta, a, b) if c.__class__ is str else _versions(self.u, self.theta, a, b, c)
        return now is not None and now == self.versions

    def holds(self, params):
        """Whether this is a point of the problem's material, none of it written to since."""
        (a, b, c), (x, y, z) = self.keys, self.values
        return (params.get(a) is x and params.get(b) is y and params.get(c) is z
                and ("material" in params) == (self.keys is self.MATERIAL) and self.unchanged)

    @property
    def material(self):
        return dict(zip(self.keys, self.values))

    def physical(self, mesh_id):
        """(the 16 physical moduli per Gauss point, the Jacobi diagonal) by the kernels that read dN/dX."""
        return ops.run(ops.qp_moduli, mesh_id, _f64c(self.u), _f64c(self.theta),
                       *ops.material_args(device_material(self.material)), False, True)

    def physical_preconditioner(self, mesh, mesh_id, with_blocks):
        """(diag, blocks or None) by the same kernels, without storing moduli."""
        diag = torch.empty(mesh.n_dof, dtype=torch.float64, device=mesh.device)
        blocks = torch.empty(2 * mesh.n_dof if with_blocks else 0, dtype=torch.float64, device=mesh.device)
        torch.ops.difffea_b200.qp_moduli_out(mesh_id, _f64c(self.u), _f64c(self.theta),
                                             *ops.material_args(device_material(self.material)),
                                             torch.empty(0, dtype=torch.float64, device=mesh.device), _lib.DFEA_F64, diag,
                                             blocks)
        return diag, blocks if with_blocks else None


class CudaTangentOperator:
    """
    v -> A(v) from moduli stored at the Gauss points (kernel (b)).  Holds the moduli of its linearisation point
    (``moduli``, layout ``code``: FP64 in the element reference frame where the mesh has one, else the 16 physical
    entries) and the Jacobi diagonal computed in the same pass of kernel (a); ``point`` is that linearisation point, where
    the operator was made from one.  ``gather``: physical moduli are applied in the gather form; chosen when the operator
    is made, so that its sums are grouped alike for as long as it lives.
    """

    def __init__(self, mesh, mesh_id, moduli, diag, precision="fp64", point=None, gather=False):
        self.mesh, self.mesh_id, self.moduli, self.diag, self.precision = mesh, mesh_id, moduli, diag, precision
        self.point, self.gather = point, gather
        self._indefinite = None
        self.code = (_lib.DFEA_F32 if moduli.dtype == torch.float32 else
                     _lib.DFEA_F64REF if moduli.numel() == mesh.moduli_numel_ref() else _lib.DFEA_F64)
        self._physical = None if self.code == _lib.DFEA_F64REF else moduli
        self._pcg = None
        self._pcg_diag_src = None
        self.last_status = None

    @property
    def C(self):
        """The 16 physical moduli per Gauss point; from the reference-frame ones on first use."""
        if self._physical is None:
            self._physical = ops.run(ops.frame_push_forward, self.mesh_id, self.moduli)
        return self._physical

    def __call__(self, v):
        """A(v); FP32 moduli apply to FP32 vectors, or to FP64 vectors with FP64 arithmetic."""
        if v.dtype != self.dtype and not (self.dtype == torch.float32 and v.dtype == torch.float64):
            raise ValueError(f"this operator applies {self.dtype} vectors, got {v.dtype}")
        return ops.run(ops.tangent_apply, self.mesh_id, self.moduli, v.contiguous(), self.gather)

    @property
    def dtype(self):
        return self.moduli.dtype

    def pcg_solve(self, b, diag, rtol, max_iter, preconditioner="jacobi", diag_point=None):
        """
        PCG on the device (kernel (c)) with this operator; returns (x in b's dtype, iterations).  ``diag`` is
        the Jacobi diagonal, or with preconditioner="block_jacobi" the (4N,) inverse node blocks, and ``diag_point`` the
        linearisation point it was made at.
        """
        from difffea_b200.krylov import DevicePCG
        from difffea_b200.workspace import pcg_form_for
        if self._indefinite is not None and self._indefinite[0] is diag and self._indefinite[1] == _versions(diag):
            return self._run_pcg(self._indefinite[2], b, rtol, max_iter)
        vt = b.dtype if self.dtype == torch.float32 else torch.float64   # FP32 moduli: FP64 or FP32 vectors
        if preconditioner == "block_jacobi":
            vt = torch.float64
        if (self._pcg is None or self._pcg_diag_src is not diag or self._pcg.vec_dtype != vt
                or self._pcg.preconditioner != preconditioner):
            d = diag.detach().to(vt).contiguous()
            n = self.mesh.n_dof
            bb = torch.empty(n, dtype=vt, device=self.mesh.device)
            xx = torch.empty(n, dtype=vt, device=self.mesh.device)
            if self._pcg is not None:
                self._pcg.close()
            ref = {}
            if self.code == _lib.DFEA_F64REF:
                ref = dict(form=pcg_form_for(self.mesh), moduli="ref", use_graph=2, cluster=True)
            self._pcg = DevicePCG(self.mesh, self.moduli, d, bb, xx, preconditioner=preconditioner, **ref)
            self._pcg_diag_src = diag
        out = self._run_pcg(self._pcg, b, rtol, max_iter)
        if self.last_status == "negative_curvature" and self.code == _lib.DFEA_F64REF:
            physical = self._physical_pcg(diag, preconditioner, diag_point)
            if physical is not None:
                self._indefinite = (diag, _versions(diag), physical)
                return self._run_pcg(physical, b, rtol, max_iter)
        return out

    def _run_pcg(self, solver, b, rtol, max_iter):
        solver.b.copy_(b)
        iters, status = solver.solve(rtol, max_iter)
        self.last_status = status
        return solver.x.to(b.dtype, copy=True), iters

    def _physical_pcg(self, diag, preconditioner, diag_point):
        """
        The solver of an operator that is not positive definite: physical moduli, one launch per colour.  On such an
        operator the iterate at the first non-positive curvature is amplified rounding -- two orders of summation
        leave 1e-4 to 1 of it different -- so the forms of a solve would give different answers.  All of them end
        here instead, with one answer.  None (the first solve's answer stands) where the point the operator was made
        at is gone or there is no memory for its physical moduli.
        """
        from difffea_b200.krylov import DevicePCG
        if self.point is None or not self.point.unchanged:
            return None
        try:
            C, own = self.point.physical(self.mesh_id)
            d = diag.detach().to(torch.float64).contiguous()
            as_made = _versions(diag) == (0,)           # not a diagonal the caller has written to
            if as_made and diag is self.diag:
                d = own
            elif as_made and diag_point is not None and diag_point.unchanged:
                blocks = preconditioner == "block_jacobi"
                d = diag_point.physical_preconditioner(self.mesh, self.mesh_id, blocks)[1 if blocks else 0]
            n = self.mesh.n_dof
            b, x = (torch.empty(n, dtype=torch.float64, device=self.mesh.device) for _ in range(2))
            return DevicePCG(self.mesh, C, d, b, x, preconditioner=preconditioner)
        except torch.cuda.OutOfMemoryError:
            return None


# (weakref(u), u._version, weakref(theta), theta._version, mesh id) -> diag and point of the last linearisation,
# so that make_preconditioner right after make_tangent_operator at the same point reuses kernel (a)'s pass
_LAST_DIAG = {}


def _diag_key(u, theta, mesh):
    return (id(u), u._version, id(theta), theta._version, id(mesh))


def make_A_operator_cuda(u, theta, params, precision="fp64"):
    """The stored-moduli tangent operator at (u, theta); precision "fp64" or "fp32" (moduli and vectors)."""
    if precision not in ("fp64", "fp32"):
        raise ValueError("precision must be 'fp64' or 'fp32'")
    mesh, mid = _prepare(u, theta, params)
    if precision == "fp32":
        mesh.ensure_grad32()
    framed = precision == "fp64" and mesh.ensure_frame()
    gather = mesh.ensure_gather()
    if framed:
        C, diag, _ = ops.run(ops.frame_moduli, mid, _f64c(u), _f64c(theta), *ops.frame_material(params), True, False)
    else:
        C, diag = ops.run(ops.qp_moduli, mid, _f64c(u), _f64c(theta), *ops.material_args(device_material(params)),
                          precision == "fp32", True)
    _LAST_DIAG.clear()
    point = _Linearisation(u, theta, params)
    _LAST_DIAG[_diag_key(u, theta, mesh)] = (weakref.ref(u), weakref.ref(theta), diag, weakref.ref(point))
    return CudaTangentOperator(mesh, mid, C, diag, precision, point, gather)


def make_tangent_operator(kind, u, theta, params):
    """
    Build the forward tangent operator by name: one of ``TANGENT_OPERATORS``.  "auto" picks "cuda"
    for CUDA tensors (the reference picks qp_ew there and qp on the CPU; its CPU variants stay in the
    reference package).
    """
    if kind == "auto":
        if not u.is_cuda:
            raise RuntimeError("'auto' on a CPU tensor selects the reference's CPU variant 'qp', which lives "
                               "in the reference package; difffea_b200 runs on CUDA devices only")
        kind = "cuda"
    if kind == "cuda":
        return make_A_operator_cuda(u, theta, params)
    if kind in REFERENCE_TANGENT_VARIANTS:
        raise ValueError(f"tangent '{kind}' is one of the reference's PyTorch variants; difffea_b200 provides "
                         f"{TANGENT_OPERATORS}")
    raise ValueError(f"Unknown tangent operator '{kind}'. Choose one of {TANGENT_OPERATORS}.")


def make_AT_operator(u, theta, params):
    """A^T: the hyperelastic tangent is symmetric, so this is the same stored-moduli operator."""
    return make_A_operator_cuda(u, theta, params)


# ---------------------------------------------------------------------------------------------
# Jacobi preconditioner
# ---------------------------------------------------------------------------------------------
class CudaJacobiPreconditioner:
    """r -> r / diag(K) with diag clamped to >= 1e-6 on free DOFs and 1 on fixed DOFs."""

    def __init__(self, mesh, diag, point=None):
        self.mesh, self.diag, self.point = mesh, diag, point

    def __call__(self, r):
        return r / self.diag.to(r.dtype)


def compute_jacobi_diagonal(u, theta, params):
    """diag(K) without forming K (kernel (a)'s element diagonals, summed at the nodes), shape (2N,)."""
    return _jacobi(u, theta, params)[1]


def _jacobi(u, theta, params):
    """(mesh, diagonal, the point it was made at)."""
    mesh, mid = _prepare(u, theta, params)
    hit = _LAST_DIAG.get(_diag_key(u, theta, mesh))
    if hit is not None and hit[0]() is u and hit[1]() is theta:
        point = hit[3]()
        if point is not None and point.holds(params):
            return mesh, hit[2], point
    return mesh, _preconditioner_data(mesh, mid, u, theta, params, False)[0], _Linearisation(u, theta, params)


def _preconditioner_data(mesh, mid, u, theta, params, with_blocks):
    """(diag, blocks or None) at (u, theta), without storing moduli."""
    if mesh.ensure_frame():
        _, diag, blocks = ops.run(ops.frame_moduli, mid, _f64c(u), _f64c(theta), *ops.frame_material(params), False, with_blocks)
        return diag, blocks
    return _Linearisation(u, theta, params).physical_preconditioner(mesh, mid, with_blocks)


def make_jacobi_preconditioner(u, theta, params):
    return CudaJacobiPreconditioner(*_jacobi(u, theta, params))


class CudaBlockJacobiPreconditioner:
    """
    r -> Binv r per node, Binv the inverse of the node's 2x2 tangent block with identity rows/columns on
    fixed DOFs and + 1e-12 I (operators.py:598-625); ``blocks`` = (Binv00, Binv01, Binv11, 0) per node.
    """

    def __init__(self, mesh, blocks, point=None):
        self.mesh, self.blocks, self.point = mesh, blocks, point

    def __call__(self, r):
        B = self.blocks.view(-1, 4).to(r.dtype)
        rn = r.view(-1, 2)
        return torch.stack([B[:, 0] * rn[:, 0] + B[:, 1] * rn[:, 1], B[:, 1] * rn[:, 0] + B[:, 2] * rn[:, 1]],
                           dim=1).reshape(-1)


def compute_block_jacobi(u, theta, params):
    """The (4N,) inverse 2x2 node blocks of the tangent at (u, theta) (kernel (a) with the coupling term)."""
    mesh, mid = _prepare(u, theta, params)
    return _preconditioner_data(mesh, mid, u, theta, params, True)[1]


def make_block_jacobi_preconditioner(u, theta, params):
    mesh = cuda_mesh(params)
    return CudaBlockJacobiPreconditioner(mesh, compute_block_jacobi(u, theta, params), _Linearisation(u, theta, params))


class CudaMultigridPreconditioner:
    """
    r -> one V-cycle of the geometric multigrid of a structured mesh (multigrid.py), set up at (u, theta).

    The hierarchy's buffers are shared by every preconditioner of the same mesh (one ``Multigrid`` per mesh),
    while each closure keeps the moduli and diagonal of its own linearisation point: when another set-up
    has overwritten the coarse operators since this closure was made, the call sets them up again from its
    own moduli first, so closures made at different states stay independent, as the reference's are.
    """

    def __init__(self, mg, A):
        self.mg, self.A = mg, A
        self.mesh = mg.mesh
        self.generation = mg.generation

    def refresh(self):
        """Set the shared hierarchy up at this closure's linearisation again if another set-up replaced it."""
        if self.mg.generation != self.generation:
            self.mg.setup(self.A.moduli, self.A.code, self.A.diag)
            self.generation = self.mg.generation

    def __call__(self, r):
        self.refresh()
        return self.mg(r.to(torch.float64))


_MG = {}


def multigrid_for(mesh, params):
    """The (cached) Multigrid hierarchy of a mesh."""
    from difffea_b200.multigrid import Multigrid
    key = id(mesh)
    hit = _MG.get(key)
    if hit is None or hit[0]() is not mesh:
        hit = (weakref.ref(mesh), Multigrid(mesh, params))
        _MG.clear()
        _MG[key] = hit
    return hit[1]


def make_multigrid_preconditioner(u, theta, params):
    A = make_A_operator_cuda(u, theta, params)
    mg = multigrid_for(A.mesh, params)
    mg.setup(A.moduli, A.code, A.diag)
    return CudaMultigridPreconditioner(mg, A)


def make_preconditioner(kind, u, theta, params):
    """Build a preconditioner by name: one of ``PRECONDITIONERS``."""
    if kind == "jacobi":
        return make_jacobi_preconditioner(u, theta, params)
    if kind == "multigrid":
        return make_multigrid_preconditioner(u, theta, params)
    if kind == "block_jacobi":
        return make_block_jacobi_preconditioner(u, theta, params)
    if kind == "ilu":
        raise ValueError("preconditioner 'ilu' factorises the assembled matrix on the CPU (SciPy); it is not "
                         "built on the device: use 'jacobi' or 'block_jacobi'")
    raise ValueError(f"Unknown preconditioner '{kind}'. Choose one of {PRECONDITIONERS}.")
