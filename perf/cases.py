"""Performance cases of the matrix-free Neo-Hookean tangent operator and its
solvers, timed through the public Python entry points: the tangent vmult over
the cachings, element degrees, precisions and mesh sizes in use, the operator
update of a Newton iteration (cache + diagonal), the residual, preconditioned
linear solves with and without the multigrid set-up, and the adjoint pass.

Fields are what a Newton iteration meets: shear moduli drawn from {1, 10}
per cell (log-normal in the solves), a smooth displacement with det F well
above zero, random source and right-hand-side vectors.  exact() restates the
operator in plain torch in 64 bits: the tangent is the directional derivative
of the internal force.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "large-strain-matrix-free_b200"))
import lsmf  # noqa: E402

NU = 0.3
VARIANTS = [("tensor4", 1), ("tensor2", 1), ("scalar", 1), ("scalar", 0), ("scalar_referential", 1), ("tensor4_ns", 1)]


def _case(name, kind, coarse, refinements=0, degree=2, caching="tensor4", formulation=1, precision="fp64",
          geometry="box", voids=0):
    c = {"kind": kind, "geometry": geometry, "nx": coarse[0], "ny": coarse[1], "nz": coarse[2],
         "refinements": refinements, "degree": degree, "caching": caching, "formulation": formulation,
         "precision": precision, "voids": voids}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the Cook membrane of the small example (8x8x1 cells refined twice): one
        # operator application of its CG, bound by launches and latency
        _case("vmult_cook_q2_small", "vmult", (8, 8, 1), 2, geometry="cook"),
        # operator throughput benchmark: unit cube, 64^3 Q2, the default caching
        _case("vmult_tensor4_q2_64", "vmult", (64, 64, 64)),
        # the finest multigrid level of the voids problem: FP32 level operator
        _case("vmult_tensor4_q2_fp32_60", "vmult", (15, 15, 15), 2, precision="fp32"),
        # the smaller cachings of the operator benchmark, ragged mesh sizes
        _case("vmult_tensor2_q2_ragged", "vmult", (61, 63, 67), caching="tensor2"),
        _case("vmult_scalar_q2_fp32_ragged", "vmult", (63, 61, 65), caching="scalar", precision="fp32"),
        # formulation 0 on linear elements (the reference's linear Cook example), at scale
        _case("vmult_scalar_f0_q1_ragged", "vmult", (95, 93, 97), degree=1, caching="scalar", formulation=0),
        # high-order run: 48^3 Q4, the largest number of unknowns
        _case("vmult_tensor4_q4_48", "vmult", (48, 48, 48), degree=4),
        # what a Newton iteration does to the outer operator before a Jacobi-CG
        _case("update_tensor4_q2_60", "update", (15, 15, 15), 2),
        # right-hand side of a Newton iteration with a surface load
        _case("residual_q2_60", "residual", (15, 15, 15), 2),
        # another right-hand side at a tangent whose multigrid is set up: CG with
        # all-FP64 V-cycles, 15^3 coarse cells and one refinement
        _case("gmg_cg_fp64_q2_15to30", "gmg_cg", (15, 15, 15), 1),
        # linear step of a Newton iteration of the voids problem at its own size:
        # cache, multigrid set-up (FP32 levels) and CG to 1e-8
        _case("newton_linear_step_voids_60", "gmg_solve", (15, 15, 15), 2, precision="fp32", voids=16),
        # adjoint pass of the shear-modulus gradient on the reduced voids mesh
        _case("adjoint_backward_voids_32", "adjoint", (8, 8, 8), 2, voids=16),
    ]


# cells a drawn vmult / update may have, per degree (the listed sizes bound them)
_MAX_CELLS = {1: 800000, 2: 262144, 3: 120000, 4: 100000}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_box(rng, cells):
    """Three sides of about `cells` cells in all, none over three times another."""
    side = cells ** (1.0 / 3.0)
    a, b = (math.exp(rng.uniform(-0.35, 0.35)) for _ in range(2))
    return tuple(max(1, int(round(s))) for s in (side * a, side * b, side / (a * b)))


def draw(rng):
    kind = rng.choice(["vmult"] * 10 + ["update"] * 3 + ["residual"] * 2 + ["jacobi_solve", "gmg_cg", "gmg_solve", "gmg_solve"])
    caching, formulation = rng.choice(VARIANTS)
    degree = rng.choice([1, 2, 2, 2, 3, 4])
    precision = rng.choice(["fp64", "fp32"])
    if kind in ("vmult", "update"):
        if rng.random() < 0.25:  # non-affine cells
            n = _log_int(rng, 3, 24)
            return _case(None, kind, (n, n, rng.randint(1, 3)), 1 if degree > 2 else 2, degree, caching, formulation,
                         precision, "cook")
        box = _draw_box(rng, _log_int(rng, 64, _MAX_CELLS[degree]))
        return _case(None, kind, box, 0, degree, caching, formulation, precision)
    if kind == "residual":
        box = _draw_box(rng, _log_int(rng, 64, 200000 // degree))
        return _case(None, kind, box, 0, degree, "scalar", rng.choice([0, 1]), "fp64")
    if kind == "jacobi_solve":
        box = _draw_box(rng, _log_int(rng, 64, 6000))
        return _case(None, kind, box, 0, rng.choice([1, 2]), caching, formulation, "fp64")
    # multigrid hierarchies
    n = rng.randint(3, 15)
    refinements = rng.choice([1, 2]) if n <= 10 else 1
    degree = rng.choice([1, 2, 2]) if n > 7 else rng.choice([1, 2, 3])
    return _case(None, kind, (n, rng.randint(3, n), rng.randint(3, n)), refinements, degree, caching, formulation, precision)


# ------------------------------------------------------------------ geometry
def _domain(case):
    if case["geometry"] == "cook":
        return (0.0, 0.0, -5.0), (48.0, 44.0, 5.0)
    return (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)


def _fine_cells(case):
    return [case[k] << case["refinements"] for k in ("nx", "ny", "nz")]


def _n_cells(case):
    a, b, c = _fine_cells(case)
    return a * b * c


def _n_nodes(case):
    p = case["degree"]
    a, b, c = _fine_cells(case)
    return (p * a + 1) * (p * b + 1) * (p * c + 1)


def _basis(p):
    """Gauss points (p + 1) on [0, 1], weights, nodes, values and derivatives [q][i]."""
    x, w = np.polynomial.legendre.leggauss(p + 1)
    x, w = 0.5 * (x + 1), 0.5 * w
    inner = {1: [], 2: [0.0], 3: [-math.sqrt(0.2), math.sqrt(0.2)], 4: [-math.sqrt(3 / 7), 0.0, math.sqrt(3 / 7)]}[p]
    nodes = np.array([0.0] + [0.5 * (1 + t) for t in inner] + [1.0])
    val, der = np.zeros((p + 1, p + 1)), np.zeros((p + 1, p + 1))
    for i in range(p + 1):
        others = [j for j in range(p + 1) if j != i]
        den = np.prod([nodes[i] - nodes[j] for j in others])
        for q in range(p + 1):
            val[q, i] = np.prod([x[q] - nodes[j] for j in others]) / den
            der[q, i] = sum(np.prod([x[q] - nodes[j] for j in others if j != k]) for k in others) / den
    return x, w, nodes, val, der


def _nodes(case):
    """Node coordinates [n_nodes, 3] in lattice order, x fastest (meshes without voids)."""
    p = case["degree"]
    gll = _basis(p)[2]
    lo, hi = _domain(case)
    axes = []
    for d, n in enumerate(_fine_cells(case)):
        t = np.append((np.arange(n)[:, None] + gll[None, :p]).reshape(-1), n) / n
        axes.append(torch.tensor(lo[d] + (hi[d] - lo[d]) * t, device="cuda"))
    z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    if case["geometry"] == "cook":
        theta = y / 44.0
        y = (1 - theta) * (44.0 / 48.0) * x + theta * (44.0 + (16.0 / 48.0) * x)
    return torch.stack([x, y, z], -1).reshape(-1, 3).contiguous()


def _cell_nodes(case):
    p = case["degree"]
    a, b, c = _fine_cells(case)
    n1 = torch.arange(p + 1, device="cuda")
    nx, ny = p * a + 1, p * b + 1
    local = (n1[:, None, None] * ny + n1[None, :, None]) * nx + n1[None, None, :]
    i, j, k = torch.arange(a, device="cuda"), torch.arange(b, device="cuda"), torch.arange(c, device="cuda")
    base = p * ((k[:, None, None] * ny + j[None, :, None]) * nx + i[None, None, :])
    return base.reshape(-1, 1) + local.reshape(1, -1)


def _constrained(case, X):
    """Clamped dofs: the face x = 0 of the Cook membrane, the bottom of a box
    (and the z component of the top where a face is displaced)."""
    if case["geometry"] == "cook":
        return (X[:, 0:1] == 0.0).expand(-1, 3).reshape(-1).clone()
    m = (X[:, 2:3] == 0.0).expand(-1, 3).clone()
    if case["voids"]:
        m[:, 2] |= X[:, 2] == 1.0
    return m.reshape(-1)


def _dirichlet(case):
    if case["geometry"] == "cook":
        return [(1, 7)]
    return [(4, 7), (5, 4)] if case["voids"] else [(4, 7)]


def _void_mask(case):
    """Coarse cells left when `voids` spheres of radius 0.08 are cut out of the unit cube."""
    rng = np.random.default_rng(2024)
    centres = []
    while len(centres) < case["voids"]:
        p = rng.uniform(0.08, 0.92, 3)
        if all(np.linalg.norm(p - q) >= 0.2 for q in centres):
            centres.append(p)
    n = [case[k] for k in ("nx", "ny", "nz")]
    z, y, x = np.meshgrid(*[(np.arange(m) + 0.5) / m for m in reversed(n)], indexing="ij")
    keep = np.ones(x.shape, dtype=np.uint8)
    for q in centres:
        keep[(x - q[0]) ** 2 + (y - q[1]) ** 2 + (z - q[2]) ** 2 < 0.08 ** 2] = 0
    return keep.reshape(-1)


# -------------------------------------------------------------------- inputs
def _fields(case, seed, X, n_cells):
    """mu [n_cells] (host), u and a random vector [n_dofs] in 64 bits."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    solve = case["kind"] in ("gmg_cg", "gmg_solve", "jacobi_solve")
    scale = 80.194 if case["geometry"] == "cook" else 1.0
    mu = scale * (np.exp(0.3 * rng.normal(size=n_cells)) if solve else rng.choice([1.0, 10.0], size=n_cells))
    size = 60.0 if case["geometry"] == "cook" else 1.0  # the membrane reaches up to y = 60
    amplitude = 0.001 if solve else 0.01  # solves: strains of a load step, a definite tangent
    u = torch.zeros_like(X)
    for c in range(3):
        for _ in range(3):
            k = rng.integers(0, 3, 3)
            phase = (X / size) @ torch.tensor(2 * np.pi * k, dtype=torch.float64, device="cuda")
            u[:, c] += (amplitude * size / 3) * torch.sin(phase + rng.uniform(0, 2 * np.pi))
    v = 2.0 * torch.rand(X.numel(), generator=gen, dtype=torch.float64, device="cuda") - 1.0
    return mu, u.reshape(-1), v


def _mesh(case):
    lo, hi = _domain(case)
    m = lsmf.Mesh(case["geometry"], (case["nx"], case["ny"], case["nz"]), case["refinements"], lo, hi,
                  degree=case["degree"], coarse_active=_void_mask(case) if case["voids"] else None)
    m.set_dirichlet(_dirichlet(case))
    return m


def _prm(sections):
    out = []
    for name, keys in sections:
        out += ["subsection " + name] + ["  set %s = %s" % kv for kv in keys] + ["end"]
    return "\n".join(out) + "\n"


def _problem_prm(case, preconditioner, residual=1e-10):
    box = [("Dimension", 3), ("Type", "Box"), ("Box cells", "%d, %d, %d" % (case["nx"], case["ny"], case["nz"])),
           ("Global refinement", case["refinements"])]
    if case["voids"]:
        box.append(("Void spheres", "%d, 0.08, 2024" % case["voids"]))
    return _prm([
        ("Finite element system", [("Polynomial degree", case["degree"]), ("Quadrature order", case["degree"] + 1)]),
        ("Geometry", box),
        ("Material properties", [("Shear modulus", 1.0), ("Poisson's ratio", NU), ("Formulation", case["formulation"])]),
        ("Linear solver", [("Solver type", "MF_CG"), ("Residual", residual), ("Preconditioner type", preconditioner),
                           ("MF caching", case["caching"])]),
        ("Nonlinear solver", [("Max iterations Newton-Raphson", 25), ("Tolerance force", 1e-11),
                              ("Tolerance displacement", 1e-10), ("Absolute tolerance force", 1e-17),
                              ("Absolute tolerance displacement", 1e-17)]),
        ("Boundary conditions", [("Dirichlet IDs and expressions", "4:0,0,0"),
                                 ("Dirichlet IDs and component mask", "4:true,true,true"),
                                 ("Neumann IDs and expressions", "5:0.02*t,0,-0.05*t")]),
        ("Time", [("End time", 1), ("Time step size", 1)])])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "residual":
        problem = lsmf.Problem(_problem_prm(case, "jacobi"))
        mu, u, _ = _fields(case, seed, _nodes(case), problem.n_cells)
        problem.set_mu(mu)
        return {"kind": kind, "problem": problem, "u": u, "R": torch.empty_like(u)}
    if kind == "adjoint":
        problem = lsmf.Problem(_problem_prm(case, "gmg"))
        rng = np.random.default_rng(seed)
        theta = rng.normal(0.0, 0.3, problem.n_cells)
        target = rng.uniform(-1e-3, 1e-3, problem.n_dofs)
        problem.adjoint_forward(theta, target, 5)
        return {"kind": kind, "problem": problem}

    mesh = _mesh(case)
    X = torch.tensor(mesh.arrays()[0], device="cuda") if case["voids"] else _nodes(case)
    mu, u, v = _fields(case, seed, X, mesh.info()[0])
    state = {"kind": kind, "mesh": mesh}
    if kind in ("vmult", "update"):
        op = lsmf.NeoHookOperator(mesh, case["caching"], case["formulation"], case["precision"])
        op.set_material(mu, NU)
        state.update(op=op, u=u.to(op.dtype))
        if kind == "vmult":
            op.cache(state["u"])
            src = v.to(op.dtype)
            state.update(src=src, dst=torch.empty_like(src))
        return state

    # linear solves: homogeneous Dirichlet right-hand side
    v[_constrained(case, X)] = 0.0
    state.update(u=u, b=v, x=torch.zeros_like(v), tol=1e-8 * float(v.norm()))
    op = lsmf.NeoHookOperator(mesh, case["caching"], case["formulation"], "fp64")
    op.set_material(mu, NU)
    state["op"] = op
    if kind == "jacobi_solve":
        op.cache(u)
        op.compute_diagonal()
        return state
    gmg = lsmf.GMG(mesh, case["caching"], case["formulation"], case["precision"])
    gmg.set_material(mu, NU)
    state["gmg"] = gmg
    if kind == "gmg_cg":
        op.cache(u)
        gmg.setup(u)
    return state


def run(state):
    kind = state["kind"]
    if kind == "vmult":
        state["op"].vmult(state["dst"], state["src"])
        return state["dst"]
    if kind == "update":
        state["op"].cache(state["u"])
        state["op"].compute_diagonal()
        return state["op"].get_matrix_diagonal_inverse()
    if kind == "residual":
        norm = state["problem"].residual(state["u"], 1.0, state["R"])
        return {"R": state["R"], "norm": norm}
    if kind == "adjoint":
        return state["problem"].adjoint_backward()
    state["x"].zero_()
    if kind == "jacobi_solve":
        lsmf.cg_solve(state["op"], state["x"], state["b"], state["tol"], 20000, "jacobi", omega=1.0)
        return state["x"]
    if kind == "gmg_solve":  # the linear part of a Newton iteration at the displacement u
        state["op"].cache(state["u"])
        state["gmg"].setup(state["u"])
    lsmf.cg_solve(state["op"], state["x"], state["b"], state["tol"], 1000, "gmg", state["gmg"])
    return state["x"]


# ---------------------------------------------------------------------- work
def _level_work(case, caching, precision, cells, nodes):
    """Bytes and flops of one operator application: src, dst (and u for the
    scalar caching) once, the values a point needs once; flops of the three
    sweeps each way and of the point's physics."""
    p = case["degree"]
    q = (p + 1) ** 3
    size = 8 if precision == "fp64" else 4
    per_point = {"tensor4": 9 + 6 + 21, "tensor2": 17, "scalar": 11, "scalar_referential": 14,
                 "tensor4_ns": 9 + 45}[caching]
    fields = 3 if caching == "scalar" else 2
    bytes_ = size * (3 * fields * nodes + per_point * q * cells) + 4 * q * cells
    sweeps = 2 * 3 * 8 * (p + 1) * q * (3 if caching == "scalar" else 2)
    return bytes_, (sweeps + 250 * q) * cells


def work(case):
    kind, p = case["kind"], case["degree"]
    cells, nodes = _n_cells(case), _n_nodes(case)
    q = (p + 1) ** 3
    if kind == "vmult":
        b, f = _level_work(case, case["caching"], case["precision"], cells, nodes)
        return {"bytes": b, "flops": f}
    if kind == "update":
        b, f = _level_work(case, case["caching"], case["precision"], cells, nodes)
        return {"bytes": b + 24 * nodes, "flops": 4 * f}
    if kind == "residual":
        return {"bytes": 8 * 9 * nodes + (4 * q + 8) * cells, "flops": (2 * 3 * 8 * (p + 1) * 3 + 250) * q * cells}
    if kind == "jacobi_solve":
        b, f = _level_work(case, case["caching"], "fp64", cells, nodes)
        its = 4 * (cells ** (1 / 3)) * p
        return {"bytes": its * b, "flops": its * f}
    # V-cycles of two smoothings of degree 5 and a residual on each refined
    # level; the coarse solve is left out, so this is a lower bound
    cyc_b = cyc_f = 0
    for l in range(1, case["refinements"] + 1):
        sub = dict(case, refinements=l)
        b, f = _level_work(sub, case["caching"], case["precision"], _n_cells(sub), _n_nodes(sub))
        cyc_b, cyc_f = cyc_b + 11 * b, cyc_f + 11 * f
    b, f = _level_work(case, case["caching"], "fp64", cells, nodes)
    # a solve to 1e-8: about 8 CG iterations; a set-up: 30 eigenvalue iterations a level
    setup = 0 if kind == "gmg_cg" else 3
    return {"bytes": 8 * (cyc_b + b) + setup * cyc_b, "flops": 8 * (cyc_f + f) + setup * cyc_f}


# --------------------------------------------------------------------- exact
def _inverse(F):
    a, b, c = F[..., 0, :], F[..., 1, :], F[..., 2, :]
    cof = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)
    det = (a * cof[..., :, 0]).sum(-1)
    return cof / det[..., None, None], det


def _piola(F, mu, formulation):
    """First Piola-Kirchhoff stress of the two compressible Neo-Hookean forms (mu broadcasts over points)."""
    Fi, det = _inverse(F)
    Fit = Fi.transpose(-1, -2)
    lam = 2 * mu * NU / (1 - 2 * NU)
    if formulation == 1:
        return mu[..., None, None] * F - (mu - 2 * lam * torch.log(det))[..., None, None] * Fit
    kappa = 2 * mu * (1 + NU) / (3 * (1 - 2 * NU))
    s = mu * det ** (-2.0 / 3.0)
    tr = s * (F * F).sum((-1, -2))
    return s[..., None, None] * F + (0.5 * kappa * (det * det - 1.0) - tr / 3.0)[..., None, None] * Fit


class _Exact:
    """The cell integrals in 64 bits, in chunks of cells."""

    def __init__(self, case, mu):
        self.case, p = case, case["degree"]
        self.X = _nodes(case)
        self.cn = _cell_nodes(case)
        self.mu = torch.tensor(mu, device="cuda")
        _, w, _, val, der = _basis(p)
        N, D = (torch.tensor(m, device="cuda") for m in (val, der))
        n1 = p + 1
        # dN[q, a, e]: reference gradients of the shape functions at the points
        def grad(z, y, x):
            return torch.einsum("kc,jb,ia->kjicba", z, y, x).reshape(n1 ** 3, n1 ** 3)
        self.dN = torch.stack([grad(N, N, D), grad(N, D, N), grad(D, N, N)], -1)
        self.w = torch.tensor((w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1), device="cuda")
        self.constrained = _constrained(case, self.X)
        self.chunk = max(1, (1 << 20) // (n1 ** 6))

    def chunks(self):
        for s in range(0, self.cn.shape[0], self.chunk):
            idx = self.cn[s:s + self.chunk]
            J = torch.einsum("cad,qae->cqde", self.X[idx], self.dN)
            Ji, det = _inverse(J)
            gN = torch.einsum("qae,cqed->cqad", self.dN, Ji)  # physical gradients
            yield idx, gN, det * self.w, self.mu[s:s + self.chunk, None].expand(-1, self.w.numel())

    def force(self, u, direction=None):
        """Internal force of u, or its derivative along `direction`."""
        out = torch.zeros_like(self.X)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        U, V = u.reshape(-1, 3), None if direction is None else direction.reshape(-1, 3)
        for idx, gN, jxw, mu in self.chunks():
            F = torch.einsum("cak,cqad->cqkd", U[idx], gN) + eye
            stress = lambda f: _piola(f, mu, self.case["formulation"])  # noqa: E731
            if V is None:
                P = stress(F)
            else:
                P = torch.func.jvp(stress, (F,), (torch.einsum("cak,cqad->cqkd", V[idx], gN),))[1]
            f = torch.einsum("cqkd,cqad,cq->cak", P, gN, jxw)
            out.index_add_(0, idx.reshape(-1), f.reshape(-1, 3))
        return out.reshape(-1)

    def vmult(self, u, src):
        free = torch.where(self.constrained, torch.zeros_like(src), src)
        return torch.where(self.constrained, src, self.force(u, free))

    def diagonal(self, u):
        out = torch.zeros_like(self.X)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        U = u.reshape(-1, 3)
        for idx, gN, jxw, mu in self.chunks():
            F = torch.einsum("cak,cqad->cqkd", U[idx], gN) + eye
            stress = lambda f: _piola(f, mu, self.case["formulation"])  # noqa: E731
            d = []
            for k in range(3):
                cols = []
                for l in range(3):
                    E = torch.zeros_like(F)
                    E[..., k, l] = 1.0
                    cols.append(torch.func.jvp(stress, (F,), (E,))[1][..., k, :])
                A = torch.stack(cols, -1)  # [c, q, j, l]
                d.append(torch.einsum("cqaj,cqjl,cqal,cq->ca", gN, A, gN, jxw))
            out.index_add_(0, idx.reshape(-1), torch.stack(d, -1).reshape(-1, 3))
        return torch.where(self.constrained, torch.ones_like(u), out.reshape(-1))


def exact(case, seed):
    kind = case["kind"]
    # meshes with voids and large solves are left out
    if case["voids"] or kind == "adjoint":
        return None
    if kind in ("gmg_cg", "gmg_solve", "jacobi_solve") and _n_nodes(case) > 40000:
        return None
    X = _nodes(case)
    mu, u, v = _fields(case, seed, X, _n_cells(case))
    if kind in ("vmult", "update") and case["precision"] == "fp32":
        u, v = u.float().double(), v.float().double()
    e = _Exact(case, mu)
    if kind == "vmult":
        return e.vmult(u, v)
    if kind == "update":
        return 1.0 / e.diagonal(u)
    if kind == "residual":
        # dead load (0.02, 0, -0.05) on the top face
        p = case["degree"]
        _, w, _, val, _ = _basis(p)
        line = w @ val
        a, b, _ = _fine_cells(case)
        sides = []
        for n in (a, b):
            s = np.zeros(p * n + 1)
            for i in range(n):
                s[p * i:p * i + p + 1] += line / n
            sides.append(torch.tensor(s, device="cuda"))
        load = torch.zeros_like(X)
        load[-sides[0].numel() * sides[1].numel():] = (sides[1][:, None] * sides[0][None, :]).reshape(-1, 1) * \
            torch.tensor([0.02, 0.0, -0.05], dtype=torch.float64, device="cuda")
        R = torch.where(e.constrained, torch.zeros_like(u), load.reshape(-1) - e.force(u))
        return {"R": R, "norm": float(R.norm())}
    # solves: Jacobi-CG in 64 bits, far below the tolerance of the run
    b = torch.where(e.constrained, torch.zeros_like(v), v)
    inv = 1.0 / e.diagonal(u)
    x = torch.zeros_like(b)
    r = b.clone()
    z = inv * r
    d, rz, stop = z.clone(), r @ z, 1e-12 * float(b.norm())
    for _ in range(3000):
        q = e.vmult(u, d)
        alpha = rz / (d @ q)
        x += alpha * d
        r -= alpha * q
        if float(r.norm()) <= stop:
            break
        z = inv * r
        rz_new = r @ z
        d = z + (rz_new / rz) * d
        rz = rz_new
    return x
