"""
The work this package is timed on: its public entry points over the range of sizes, element types, materials
and precisions they are used with.

    product     A(v) with a stored tangent operator -- what a caller's own Krylov loop, eigenvalue solver or
                operator study does thousands of times per linearisation
    linearise   one Newton linearisation: residual, tangent operator, Jacobi preconditioner, and one use of each
    pcg         one preconditioned linear solve on the device
    solve       a whole Newton-Krylov solve of a rectangle from problem dictionary to displacement
    plate       the same on the mapped quarter plate with a hole (Q9, mixed precision, multigrid)
    gradient    compliance and its gradient by the adjoint, the step of a design loop
    fields      post-processing of a solution: element and nodal fields, support reactions
    serve       a backlog of requests through the continuous-batching engine

States, stiffness scales and loads are seeded; the problems' sizes are the case's.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "differentiable-fea_b200"))

from difffea_b200.autograd import compliance  # noqa: E402
from difffea_b200.newton_krylov import newton_krylov_solve, pcg  # noqa: E402
from difffea_b200.operators import (global_residual, make_preconditioner, make_tangent_operator)  # noqa: E402
from difffea_b200.postprocess import compute_fields, support_reactions  # noqa: E402
from difffea_b200.problem import build_quarter_plate_problem, build_rectangle_problem  # noqa: E402
from difffea_b200.serving import Request, ServingEngine  # noqa: E402
from difffea_b200.workspace import NewtonWorkspace  # noqa: E402

DEV = "cuda"
NEN = {"tri3": 3, "tri6": 6, "quad4": 4, "quad8": 8, "quad9": 9}
NQ = {"tri3": 1, "tri6": 6, "quad4": 4, "quad8": 9, "quad9": 9}
MATERIALS = {"neo_hookean": None, "mooney_rivlin": {"c10": 0.2, "c01": 0.05, "kappa": 0.7},
             "saint_venant": {"mu": 0.4, "lmbda": 0.6}}


def listed():
    return [
        # the smallest call: the mesh of the smallest serving request, where launches and host time count
        dict(name="product_q4_tiny", kind="product", element="quad4", nx=16, ny=4, precision="fp64"),
        # the size the tangent product is judged at: a million Q4 elements
        dict(name="product_q4_1m", kind="product", element="quad4", nx=1024, ny=1024, precision="fp64"),
        # a quadratic mesh with odd cell counts
        dict(name="product_q9_ragged", kind="product", element="quad9", nx=317, ny=203, precision="fp64"),
        # FP32 operator and vectors on triangles
        dict(name="product_tri6_fp32", kind="product", element="tri6", nx=251, ny=130, precision="fp32"),
        # a Newton step's set-up on a large Q4 mesh and, with another material, on an ordinary Q9 one
        dict(name="linearise_q4", kind="linearise", element="quad4", nx=800, ny=800, material="neo_hookean"),
        dict(name="linearise_q9_mooney", kind="linearise", element="quad9", nx=150, ny=91, material="mooney_rivlin"),
        # a long Jacobi-PCG solve on a mid-sized mesh
        dict(name="pcg_q4", kind="pcg", element="quad4", nx=256, ny=64, preconditioner="jacobi"),
        # the plain reference workload: 100 x 100 Q4, three load steps, Jacobi-PCG
        dict(name="solve_q4_plain", kind="solve", element="quad4", nx=100, ny=100, precision="fp64",
             preconditioner="jacobi", steps=3),
        # mixed precision with multigrid on the quarter plate
        dict(name="plate_q9_mixed", kind="plate", n=128, steps=2),
        # one step of a design loop: forward solve, adjoint, gradient
        dict(name="gradient_q4", kind="gradient", nx=384, ny=384),
        # post-processing of a Q9 solution
        dict(name="fields_q9", kind="fields", element="quad9", nx=256, ny=256),
        # a backlog of serving requests, Q4 and Q9 cantilevers of uneven sizes
        dict(name="serve_backlog", kind="serve", requests=32, nx_max=256, stream=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, element, lo, hi):
    """nx, ny of a mesh with a log-uniform number of elements in [lo, hi] and an aspect ratio of up to 4."""
    n_el = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    cells = n_el / 2 if element.startswith("tri") else n_el
    aspect = math.exp(rng.uniform(0.0, math.log(4.0)))
    return max(4, int(math.sqrt(cells * aspect))), max(2, int(math.sqrt(cells / aspect)))


def draw(rng):
    kind = rng.choice(["product", "product", "linearise", "pcg", "solve", "plate", "gradient", "fields", "serve"])
    if kind == "product":
        element = rng.choice(sorted(NEN))
        nx, ny = _cells(rng, element, 64, 1_000_000 if NEN[element] <= 4 else 100_000)
        return dict(kind=kind, element=element, nx=nx, ny=ny, precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "linearise":
        element = rng.choice(sorted(NEN))
        nx, ny = _cells(rng, element, 1_000, 600_000 if NEN[element] <= 4 else 100_000)
        return dict(kind=kind, element=element, nx=nx, ny=ny, material=rng.choice(sorted(MATERIALS)))
    if kind == "pcg":
        element = rng.choice(["tri3", "quad4", "quad9"])
        nx = _log_int(rng, 16, 100 if element == "quad9" else 256)
        return dict(kind=kind, element=element, nx=nx, ny=max(2, nx // rng.choice([2, 3, 4])),
                    preconditioner=rng.choice(["jacobi", "jacobi", "block_jacobi"]))
    if kind == "solve":
        element = rng.choice(["tri3", "tri6", "quad4", "quad9"])
        nx = _log_int(rng, 8, 40 if NEN[element] > 4 else 100)
        multigrid = rng.random() < 0.4
        return dict(kind=kind, element=element, nx=nx, ny=max(4, nx // rng.choice([1, 2, 4])),
                    precision=rng.choice(["fp64", "fp32"]), preconditioner="multigrid" if multigrid else "jacobi",
                    steps=rng.choice([1, 2, 3]))
    if kind == "plate":
        return dict(kind=kind, n=2 * _log_int(rng, 8, 60), steps=rng.choice([1, 2]))
    if kind == "gradient":
        nx = _log_int(rng, 32, 380)
        return dict(kind=kind, nx=nx, ny=max(8, nx // rng.choice([1, 2])))
    if kind == "fields":
        element = rng.choice(sorted(NEN))
        nx, ny = _cells(rng, element, 100, 400_000 if NEN[element] <= 4 else 60_000)
        return dict(kind=kind, element=element, nx=nx, ny=ny)
    return dict(kind=kind, requests=rng.choice([4, 8, 16, 32]), nx_max=4 * _log_int(rng, 8, 64),
                stream=rng.randrange(1 << 20))


# ---------------------------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------------------------
def _theta(n_el, gen):
    """A log-normal per-element stiffness scale (mu = 0, sigma = 0.3)."""
    return torch.exp(0.3 * torch.randn(n_el, dtype=torch.float64, generator=gen, device=DEV))


def _mesh(case, load=(0.0, -1e-3), material="neo_hookean", unit=False):
    """A rectangle of unit-sized cells (the operator cases), or the unit-height body of the solves."""
    nx, ny = case["nx"], case["ny"]
    w, h = (nx / ny, 1.0) if unit else (float(nx), float(ny))
    return build_rectangle_problem(case["element"], nx, ny, w, h, E=1.0, nu=0.3, load=load, device=DEV,
                                   build_on_device=True, material=material, material_params=MATERIALS[material])


def _state(p, gen, element):
    """Seeded nodal displacements uniform in +- 0.05 node spacings, zero at the supports."""
    h = 1.0 if NEN[element] <= 4 else 0.5
    u = (2.0 * torch.rand(p["f"].numel(), dtype=torch.float64, generator=gen, device=DEV) - 1.0) * 0.05 * h
    return u * p["m"]


def _requests(case, seed):
    sizes, values = random.Random(case["stream"]), random.Random(seed)
    out = []
    for i in range(case["requests"]):
        nx = 4 * sizes.randint(4, max(4, case["nx_max"] // 4))
        out.append(Request(i, sizes.choice(["quad4", "quad9"]), nx, E=math.exp(values.uniform(math.log(0.5), math.log(2.0))),
                           nu=values.uniform(0.2, 0.45), load=values.uniform(0.01, 0.05)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    s = dict(case=case)
    if kind == "serve":
        s["engine"] = ServingEngine(n_slots=16, order="largest_first", hbm_budget=32 << 30)
        s["requests"] = _requests(case, seed)
        return s
    if kind == "plate":
        p = build_quarter_plate_problem("quad9", n_theta=case["n"], n_radial=case["n"], traction=0.05 * case["steps"],
                                        device=DEV)
        s.update(p=p, theta=_theta(p["conn"].shape[0], gen), tol=1e-10 * float(torch.linalg.vector_norm(p["f"])))
        return s
    if kind in ("solve", "gradient"):
        case = dict(case, element=case.get("element", "quad4"))
        load = (0.1, 0.0) if kind == "solve" else (0.0, -0.0072 * (case["ny"] / case["nx"]) ** 2)
        p = _mesh(case, load=load, unit=True)
        s.update(p=p, theta=_theta(p["conn"].shape[0], gen), tol=1e-10 * float(torch.linalg.vector_norm(p["f"])))
        if kind == "gradient":                       # a design loop keeps its buffers from step to step
            s["workspace"] = NewtonWorkspace(p, preconditioner="multigrid")
        return s
    p = _mesh(case, material=case.get("material", "neo_hookean"), unit=kind == "pcg")
    s.update(p=p, theta=_theta(p["conn"].shape[0], gen), u=_state(p, gen, case["element"]))
    if kind == "pcg":
        s["u"] = s["u"] / case["ny"]
    if kind in ("product", "linearise"):
        s["v"] = torch.randn(p["f"].numel(), dtype=torch.float64, generator=gen, device=DEV)
    if kind == "product":
        if case["precision"] == "fp32":
            from difffea_b200.operators import make_A_operator_cuda
            s["A"] = make_A_operator_cuda(s["u"], s["theta"], p, precision="fp32")
            s["v"] = s["v"].to(torch.float32)
        else:
            s["A"] = make_tangent_operator("cuda", s["u"], s["theta"], p)
    if kind == "pcg":
        s["A"] = make_tangent_operator("cuda", s["u"], s["theta"], p)
        s["Minv"] = make_preconditioner(case["preconditioner"], s["u"], s["theta"], p)
        s["b"] = p["m"] * torch.randn(p["f"].numel(), dtype=torch.float64, generator=gen, device=DEV)
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
PCG_RTOL = 1e-12


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "product":
        return s["A"](s["v"])
    if kind == "linearise":
        R = global_residual(s["u"], s["theta"], s["p"])
        A = make_tangent_operator("cuda", s["u"], s["theta"], s["p"])
        Minv = make_preconditioner("jacobi", s["u"], s["theta"], s["p"])
        return R, Minv(R), A(s["v"])
    if kind == "pcg":
        return pcg(s["A"], s["b"], s["Minv"], rtol=PCG_RTOL, max_iter=20000)[0]
    if kind == "solve":
        return newton_krylov_solve(s["p"], s["theta"], case["steps"], s["tol"], verbose=False, pcg_max_iter=5000,
                                   precision=case["precision"], preconditioner=case["preconditioner"])[0]
    if kind == "plate":
        return newton_krylov_solve(s["p"], s["theta"], case["steps"], s["tol"], verbose=False, pcg_max_iter=5000,
                                   precision="fp32", preconditioner="multigrid", driver="native")[0]
    if kind == "gradient":
        theta = s["theta"].detach().requires_grad_(True)
        L = compliance(theta, s["p"], n_load_steps=1, tol=s["tol"], preconditioner="multigrid",
                       workspace=s["workspace"], adjoint_preconditioner="multigrid")
        L.backward()
        return L.detach(), theta.grad
    if kind == "fields":
        return compute_fields(s["u"], s["theta"], s["p"]), support_reactions(s["u"], s["theta"], s["p"])
    return [r.u for r in s["engine"].run(s["requests"])]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _sizes(element, nx, ny):
    k = 1 if NEN[element] <= 4 else 2
    n_el = nx * ny * (2 if element.startswith("tri") else 1)
    nodes = (k * nx + 1) * (k * ny + 1) - (nx * ny if element == "quad8" else 0)
    return n_el, nodes


def _operator(element, nx, ny, word=8):
    """Bytes and operations of one product: state, input and output vectors, nodes, connectivity, theta; per
    Gauss point the gradient of v, the 4 x 4 moduli, the element forces."""
    n_el, nodes = _sizes(element, nx, ny)
    nen, nq = NEN[element], NQ[element]
    return dict(bytes=nodes * (32 + 4 * word) + n_el * (4 * nen + 8), flops=n_el * nq * (16 * nen + 32))


def _request_work(element, nx, steps):
    w = _operator(element, nx, nx // 4)
    return dict(bytes=steps * w["bytes"], flops=steps * w["flops"])


def work(case):
    kind = case["kind"]
    if kind == "product":
        return _operator(case["element"], case["nx"], case["ny"], 4 if case["precision"] == "fp32" else 8)
    if kind == "linearise":      # residual, moduli and product; u, v, f, nodes read, three vectors written
        w = _operator(case["element"], case["nx"], case["ny"])
        n_el, nodes = _sizes(case["element"], case["nx"], case["ny"])
        return dict(bytes=w["bytes"] + 48 * nodes, flops=2 * w["flops"] + n_el * NQ[case["element"]] * 150)
    if kind == "fields":         # u, nodes, theta, connectivity read; 6 element and 9 nodal fields written
        n_el, nodes = _sizes(case["element"], case["nx"], case["ny"])
        nen, nq = NEN[case["element"]], NQ[case["element"]]
        return dict(bytes=nodes * (32 + 72) + n_el * (4 * nen + 8 + 56), flops=n_el * nq * (24 * nen + 100))
    if kind == "serve":          # about 12 V-cycles of ~6 products each, or as many iterations' worth
        ws = [_request_work(r.element_type, r.nx, 80) for r in _requests(case, 0)]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    if kind == "plate":
        w, n = _operator("quad9", case["n"], case["n"]), 100 * case["steps"]
    elif kind == "gradient":
        w, n = _operator("quad4", case["nx"], case["ny"]), 200
    elif kind == "pcg":          # iterations grow with the cells across
        w, n = _operator(case["element"], case["nx"], case["ny"]), 6 * case["nx"]
    else:
        w = _operator(case["element"], case["nx"], case["ny"])
        n = 60 * case["steps"] if case["preconditioner"] == "multigrid" else 13 * case["nx"] * case["steps"]
    return dict(bytes=n * w["bytes"], flops=n * w["flops"])


# ---------------------------------------------------------------------------------------------
# the same values in plain torch, 64 bits (the problem dictionaries' arrays are inputs)
# ---------------------------------------------------------------------------------------------
def _psi(name, F, q):
    """Energy density of the plane-strain embedding; q: the parameters, (n_el, 1, n_params)."""
    J = F[..., 0] * F[..., 3] - F[..., 1] * F[..., 2]
    lnJ = torch.log(J)
    I1 = (F * F).sum(-1) + 1.0
    if name == "neo_hookean":
        return 0.5 * q[..., 0] * (I1 - 3.0 - 2.0 * lnJ) + 0.5 * q[..., 1] * lnJ ** 2
    if name == "mooney_rivlin":
        C = torch.stack([F[..., 0] ** 2 + F[..., 2] ** 2, F[..., 0] * F[..., 1] + F[..., 2] * F[..., 3],
                         F[..., 1] ** 2 + F[..., 3] ** 2], -1)
        trC2 = C[..., 0] ** 2 + 2.0 * C[..., 1] ** 2 + C[..., 2] ** 2 + 1.0
        I2 = 0.5 * (I1 ** 2 - trC2)
        return (q[..., 0] * (J ** (-2.0 / 3.0) * I1 - 3.0) + q[..., 1] * (J ** (-4.0 / 3.0) * I2 - 3.0)
                + 0.5 * q[..., 2] * lnJ ** 2)
    E00 = 0.5 * (F[..., 0] ** 2 + F[..., 2] ** 2 - 1.0)
    E11 = 0.5 * (F[..., 1] ** 2 + F[..., 3] ** 2 - 1.0)
    E01 = 0.5 * (F[..., 0] * F[..., 1] + F[..., 2] * F[..., 3])
    return 0.5 * q[..., 1] * (E00 + E11) ** 2 + q[..., 0] * (E00 ** 2 + E11 ** 2 + 2.0 * E01 ** 2)


class _Plain:
    """Residual, moduli and products of a problem at (u, theta) by autodiff of the energy."""

    def __init__(self, s):
        p = s["p"]
        self.p, self.conn, self.G, self.w = p, p["conn"], p["dN_dX"], p["w_detJ"]
        scal = p["mat_scalable"].to(DEV)
        self.q = torch.where(scal[None, :], s["theta"][:, None], torch.ones_like(s["theta"])[:, None]) * p["mat_p"].to(DEV)
        self.q = self.q[:, None, :]
        self.F = (torch.einsum("eai,eqaj->eqij", s["u"].view(-1, 2)[self.conn], self.G)
                  + torch.eye(2, dtype=torch.float64, device=DEV)).flatten(-2).requires_grad_(True)
        self.psi = _psi(p["material"], self.F, self.q)
        self.P = torch.autograd.grad(self.psi.sum(), self.F, create_graph=True)[0]

    def scatter(self, stress):
        """Nodal forces of the stresses (n_el, n_q, 2, 2), at every DOF."""
        fe = torch.einsum("eq,eqij,eqaj->eai", self.w, stress.view(*self.w.shape, 2, 2), self.G)
        out = torch.zeros(self.p["f"].numel() // 2, 2, dtype=torch.float64, device=DEV)
        return out.index_add_(0, self.conn.reshape(-1), fe.reshape(-1, 2)).reshape(-1)

    def residual(self):
        return self.p["m"] * (self.scatter(self.P.detach()) - self.p["f"])

    def moduli(self):
        rows = [torch.autograd.grad(self.P[..., r].sum(), self.F, retain_graph=True)[0] for r in range(4)]
        return torch.stack(rows, -2)

    def product(self, C, v):
        m = self.p["m"]
        g = torch.einsum("eai,eqaj->eqij", (m * v).view(-1, 2)[self.conn], self.G).flatten(-2)
        return m * self.scatter(torch.einsum("eqrc,eqc->eqr", C, g)) + (1.0 - m) * v

    def node_blocks(self, C):
        """(N, 2, 2) diagonal blocks of the tangent, unmasked."""
        K = torch.einsum("eq,eqiJkL,eqaJ,eqaL->eaik", self.w, C.view(*self.w.shape, 2, 2, 2, 2), self.G, self.G)
        out = torch.zeros(self.p["f"].numel() // 2, 2, 2, dtype=torch.float64, device=DEV)
        return out.index_add_(0, self.conn.reshape(-1), K.reshape(-1, 2, 2))

    def diagonal(self, C):
        d = torch.diagonal(self.node_blocks(C), dim1=1, dim2=2).reshape(-1)
        return torch.where(self.p["m"] > 0, d.clamp(min=1e-6), torch.ones_like(d))


def _solve_exact(A, b, diag):
    """Jacobi-PCG of plain torch operations to the rounding floor."""
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, nb = z.clone(), torch.dot(r, z), torch.linalg.vector_norm(b)
    for k in range(20000):
        Ap = A(p)
        a = rz / torch.dot(p, Ap)
        x += a * p
        r -= a * Ap
        if k % 50 == 0 and float(torch.linalg.vector_norm(r) / nb) < 2e-14:
            break
        z = r / diag
        rz_new = torch.dot(r, z)
        p = z + (rz_new / rz) * p
        rz = rz_new
    return x


def _fields_exact(s):
    p, plain = s["p"], _Plain(s)
    F, P = plain.F.detach(), plain.P.detach()
    J = F[..., 0] * F[..., 3] - F[..., 1] * F[..., 2]
    sxx = (P[..., 0] * F[..., 0] + P[..., 1] * F[..., 1]) / J
    syy = (P[..., 2] * F[..., 2] + P[..., 3] * F[..., 3]) / J
    sxy = (P[..., 0] * F[..., 2] + P[..., 1] * F[..., 3]) / J
    szz = plain.q[..., 1] * torch.log(J) / J                        # neo-Hookean, F33 = 1
    area = plain.w.sum(1)
    mean = lambda t: (plain.w * t).sum(1) / area  # noqa: E731
    mJ, a, b, c, z, e = (mean(t) for t in (J, sxx, syy, sxy, szz, plain.psi.detach()))
    mises = torch.sqrt(0.5 * ((a - b) ** 2 + (b - z) ** 2 + (z - a) ** 2) + 3.0 * c ** 2)
    el = dict(J=mJ, sxx=a, syy=b, sxy=c, mises=mises, energy_density=e)
    N, conn = p["nodes"].shape[0], p["conn"].reshape(-1)
    count = torch.zeros(N, dtype=torch.float64, device=DEV).index_add_(0, conn, torch.ones(conn.numel(), dtype=torch.float64, device=DEV))
    un = s["u"].view(N, 2)
    out = dict(el, ux=un[:, 0], uy=un[:, 1], u_mag=torch.sqrt((un ** 2).sum(1)), strain_energy=(e * area).sum(), min_J=mJ.min())
    for k in ("ux", "uy", "u_mag"):
        out[k + "_n"] = out[k]
    for k, t in el.items():
        spread = t[:, None].expand(-1, p["conn"].shape[1]).reshape(-1)
        out[k + "_n"] = torch.zeros(N, dtype=torch.float64, device=DEV).index_add_(0, conn, spread) / count
    R = plain.scatter(P).view(-1, 2)
    return out, torch.where(p["fixed"].view(-1, 2), R, torch.zeros_like(R)).sum(0)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "plate", "gradient", "serve"):
        return None                        # thousands of plain products: over the time a check has
    s = prepare(case, seed)
    if kind == "fields":
        return _fields_exact(s)
    plain = _Plain(s)
    if kind == "product":
        return plain.product(plain.moduli(), s["v"].double())
    C = plain.moduli()
    if kind == "linearise":
        R = plain.residual()
        return R, R / plain.diagonal(C), plain.product(C, s["v"])
    return _solve_exact(lambda v: plain.product(C, v), s["b"], plain.diagonal(C))
