"""Performance cases of the framework: what a user's program calls, over the sizes it is called at.

Every case solves, assembles or differentiates ``-div(k grad u) = 1`` with u = 0 on the boundary (the
transient ones ``u_t - div(k grad u) = 1``) on a Kuhn-tetrahedral box or a triangulated rectangle with
jittered interior vertices and a lognormal coefficient, through ``jno_b200``'s public surface.

Fields of a case: ``path`` (what is called, below), ``nx, ny, nz`` (cells per axis; nz = 0: a rectangle of
triangles), ``order`` (1 or 2), ``numbering`` ("lattice": the structured constructors' order; "shuffled":
vertices and cells in random order, as a mesh file may hold them) and per path:

* ``solve``    evaluate the parametric system and solve it: ``solver`` cg | mixed | bicgstab, ``tol``
* ``matfree``  the same solve on the matrix-free operator (cg)
* ``gradient`` misfit of a solve and its gradient with respect to log k (forward and adjoint solve)
* ``assemble`` evaluate alone, with the backward pass of a loss of A's values; ``param`` p0 | nodal
* ``march``    a transient solve over ``steps`` theta steps (``theta``)
* ``batch``    ``count`` independent P1 cubes of sides in [nx, ny], one launch; ``solver`` cg | mixed
"""

import math

import numpy as np
import torch

import jno_b200 as jno
from jno_b200.batch import BatchedPoisson

KUHN = ((0, 4, 6, 7), (0, 4, 5, 7), (0, 2, 6, 7), (0, 2, 3, 7), (0, 1, 5, 7), (0, 1, 3, 7))
DT = 1e-3  # time step of the transient cases
LAUNCH = {"tile_rows": 64, "blocks_per_sm": 2}  # the batched launch's schedule, kept from an earlier tuning


def listed():
    def case(name, path, nx, ny, nz, order=1, numbering="lattice", **more):
        return dict(name=name, path=path, nx=nx, ny=ny, nz=nz, order=order, numbering=numbering, **more)

    return [
        # a coarse model inside an optimisation loop: a few hundred unknowns, launches and latency
        case("p1_tiny_cg", "solve", 8, 7, 9, solver="cg", tol=1e-8),
        # the plain method at a desktop size: 32^3 hexes, 35,937 unknowns
        case("p1_32_cg", "solve", 32, 32, 32, solver="cg", tol=1e-8),
        # the production size: 128^3 hexes, 12.6M tetrahedra, 2.1M unknowns
        case("p1_128_cg", "solve", 128, 128, 128, solver="cg", tol=1e-8),
        # the same with FP32 inner iterations, refined to 1e-10
        case("p1_128_mixed", "solve", 128, 128, 128, solver="mixed", tol=1e-10),
        # no room for a matrix: the operator recomputed per element, an uneven box
        case("p1_matfree", "matfree", 92, 104, 87, tol=1e-8),
        # second-order elements: 64^3 hexes, 2.1M unknowns, rows of up to 65 entries
        case("p2_64_mixed", "solve", 64, 64, 64, order=2, solver="mixed", tol=1e-10),
        # second-order elements in FP64 on an odd box
        case("p2_odd_cg", "solve", 37, 45, 41, order=2, solver="cg", tol=1e-10),
        # one step of an inverse problem: value and gradient with respect to 1.57M coefficients
        case("gradient_64", "gradient", 64, 64, 64, tol=1e-10),
        # assembly for a program with its own solver, forward and backward
        case("assemble_p1", "assemble", 100, 97, 104, param="p0"),
        # a triangle mesh from a file (no lattice order), second order, the default steady solver
        case("tri_p2_general", "solve", 131, 118, 0, order=2, numbering="shuffled", solver="bicgstab", tol=1e-12),
        # heat conduction in time, Crank-Nicolson
        case("heat_march", "march", 44, 40, 47, theta=0.5, steps=12),
        # many small problems of uneven size at once
        case("batch_96", "batch", 8, 48, 0, count=96, solver="cg", tol=1e-8),
    ]


def draw(rng):
    """One more case of the ranges above: sizes log-uniform per path, uneven sides."""
    path = rng.choice(["solve"] * 6 + ["matfree", "matfree", "gradient", "gradient", "assemble", "march", "batch"])
    order, nz, c = 1, 1, {}
    numbering = rng.choice(["lattice", "lattice", "shuffled"])
    lo, hi = 5, 64
    if path == "solve":
        order = rng.choice([1, 1, 2])
        nz = rng.choice([0, 1, 1, 1])
        solver = rng.choice(["cg", "cg", "cg", "mixed", "bicgstab"])
        if solver == "mixed" and nz == 0:
            solver = "cg"  # FP32 inner iterations are for well-conditioned systems
        c = dict(solver=solver, tol=1e-12 if solver == "bicgstab" or nz == 0 else (1e-10 if order == 2 or solver == "mixed" else 1e-8))
        lo, hi = {(1, 0): (10, 260), (2, 0): (8, 120), (1, 1): (4, 110), (2, 1): (3, 48)}[(order, min(nz, 1))]
    elif path == "matfree":
        order = rng.choice([1, 1, 2])
        lo, hi = (8, 80) if order == 1 else (5, 40)
        c = dict(tol=1e-8 if order == 1 else 1e-10)
    elif path == "gradient":
        lo, hi = 6, 60
        c = dict(tol=1e-10)
    elif path == "assemble":
        order = rng.choice([1, 1, 2])
        lo, hi = (10, 90) if order == 1 else (6, 44)
        c = dict(param=rng.choice(["p0", "p0", "nodal"]) if order == 1 else "p0")
    elif path == "march":
        lo, hi = 6, 40
        c = dict(theta=rng.choice([1.0, 0.5]), steps=rng.randint(3, 12))
    else:
        n0 = rng.randint(6, 14)
        c = dict(count=rng.randint(5, 80), solver=rng.choice(["cg", "mixed"]))
        c["tol"] = 1e-8 if c["solver"] == "cg" else 1e-10
        return dict(path=path, nx=n0, ny=n0 + rng.randint(4, 30), nz=0, order=1, numbering="lattice", **c)
    side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax = [max(2, round(side * math.exp(rng.uniform(-0.15, 0.15)))) for _ in range(3)]
    return dict(path=path, nx=ax[0], ny=ax[1], nz=ax[2] if nz else 0, order=order, numbering=numbering, **c)


# ---------------------------------------------------------------------------------------------- inputs
def _mesh(nx, ny, nz, numbering, seed):
    """(points f64[nv, dim], cells i64[T, dim + 1]) of the unit box or rectangle, interior vertices moved
    by up to a tenth of the spacing."""
    rng = np.random.default_rng(seed)
    dims = (nx, ny, nz) if nz else (nx, ny)
    dim = len(dims)
    shape = tuple(d + 1 for d in dims)
    stride = [int(np.prod(shape[a + 1:])) for a in range(dim)]
    points = np.empty(shape + (dim,))
    for a, d in enumerate(dims):
        points[..., a] = np.linspace(0.0, 1.0, d + 1).reshape([-1 if b == a else 1 for b in range(dim)])
    inner = tuple(slice(1, -1) for _ in dims)
    move = rng.uniform(-0.1, 0.1, tuple(d - 1 for d in dims) + (dim,)) / np.asarray(dims, dtype=np.float64)
    points[inner] += move
    base = sum(np.arange(d, dtype=np.int64).reshape([-1 if b == a else 1 for b in range(dim)]) * stride[a]
               for a, d in enumerate(dims)).reshape(-1)
    if dim == 3:
        corner = np.asarray([(c >> 2 & 1) * stride[0] + (c >> 1 & 1) * stride[1] + (c & 1) for c in range(8)])
        local = corner[np.asarray(KUHN)]
    else:
        local = np.asarray([[0, stride[0], stride[0] + 1], [0, stride[0] + 1, 1]])
    points = points.reshape(-1, dim)
    cells = (base[:, None, None] + local[None]).reshape(-1, dim + 1)
    if numbering == "shuffled":
        perm = rng.permutation(len(points))  # new id of each vertex
        moved = np.empty_like(points)
        moved[perm] = points
        points, cells = moved, perm[cells][rng.permutation(len(cells))]
    return points, cells


def _sides(case):
    """Sides of a batch's cubes: log-uniform in [nx, ny], in no order of size."""
    at = (np.random.default_rng(case["count"]).permutation(case["count"]) + 0.5) / case["count"]
    return np.rint(case["nx"] * (case["ny"] / case["nx"]) ** at).astype(int).tolist()


def _log_field(size, seed):
    """log k ~ N(0, 0.5^2) per element (or vertex), on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return 0.5 * torch.randn(size, dtype=torch.float64, device="cuda", generator=gen)


class _Built:
    """What a mesh constructor returns: points [nv, 3] and cells."""

    def __init__(self, points, cells):
        if points.shape[1] == 2:
            points = np.column_stack([points, np.zeros(len(points))])
        self.points, self.tets = points, cells


def _system(case, points, cells, time=None):
    """The user's FEM object for ``exp(logk) grad u . grad v - v`` (plus ``u_t v``), u = 0 on the boundary."""
    dim = points.shape[1]
    domain = jno.domain(lambda geo: (_Built(points, cells), dim, 1.0 / max(case["nx"], case["ny"])), time=time)
    u, v = domain.fem_symbols(order=case["order"])
    if case.get("param", "p0") == "nodal":
        sym = domain.fem_symbols(order=1)[0]
    else:
        sym = domain.fem_symbols(space="P0")[0]
    k = jno.np.exp(jno.np.parameter(sym, name="logk"))
    at = dict(zip("xyz", domain.variable("interior")))
    edge = domain.variable("boundary")[:dim]
    if time is not None:
        at["t"] = domain.variable("interior")[-1]
    ui, vi = u.bind(**at), v.bind(**at)
    grad = ui.x * vi.x + ui.y * vi.y
    if dim == 3:
        grad = grad + ui.z * vi.z
    terms = [k * grad - 1.0 * vi, u(*edge) - 0.0]
    if time is not None:
        start = domain.variable("initial")
        hill = jno.np.sin(math.pi * start[0]) * jno.np.sin(math.pi * start[1]) * jno.np.sin(math.pi * start[2])
        terms = [ui.t * vi + terms[0], terms[1], u(*start[:dim]) - hill]
    return jno.fem(terms)


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        meshes = [_mesh(n, n, n, "lattice", [seed, i]) for i, n in enumerate(_sides(case))]
        batch = BatchedPoisson(meshes)
        return dict(case=case, batch=batch, logk=_log_field(int(batch.tet_off[-1]), seed))
    points, cells = _mesh(case["nx"], case["ny"], case["nz"], case["numbering"], seed)
    if path == "march":
        fem = _system(case, points, cells, time=(0.0, DT * case["steps"], case["steps"] + 1))
    else:
        fem = _system(case, points, cells)
    nodal = case.get("param") == "nodal"
    state = dict(case=case, fem=fem, logk=_log_field(len(points) if nodal else len(cells), seed))
    if path == "gradient":  # the observation that the misfit compares with, and its weights
        state["target"] = _log_field(fem.dofs, seed + 1) * 0.1
        state["mass"] = fem.plan.lumped_mass()
    if path == "assemble":  # the cotangent that a user's own loss sends back into the matrix
        state["cotangent"] = _log_field(fem.plan.nnz, seed + 1)
    return state


# ------------------------------------------------------------------------------------------------ runs
def _solver(case):
    if case.get("solver") == "bicgstab":
        return jno.solve.bicgstab(tol=case["tol"])
    return jno.solve.cg(tol=case["tol"], precision="mixed" if case.get("solver") == "mixed" else "fp64")


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "solve":
        A, b = state["fem"].operator.evaluate({"logk": state["logk"]})
        return {"data": A.data, "b": b, "u": _solver(case)(A, b, M=jno.precond.jacobi())}
    if path == "matfree":
        A, b = state["fem"].matrix_free({"logk": state["logk"]})
        return {"b": b, "u": _solver(case)(A, b, M=jno.precond.jacobi())}
    if path == "gradient":
        logk = state["logk"].detach().requires_grad_(True)
        A, b = state["fem"].operator.evaluate({"logk": logk})
        u = _solver(case)(A, b, M=jno.precond.jacobi())
        loss = 0.5 * torch.sum(state["mass"] * (u - state["target"]) ** 2)
        (grad,) = torch.autograd.grad(loss, logk)
        return {"u": u.detach(), "loss": loss.detach(), "grad": grad}
    if path == "assemble":
        logk = state["logk"].detach().requires_grad_(True)
        A, b = state["fem"].operator.evaluate({"logk": logk})
        (grad,) = torch.autograd.grad(A.data, logk, grad_outputs=state["cotangent"])
        return {"data": A.data.detach(), "b": b.detach(), "grad": grad}
    if path == "march":
        sol = state["fem"].solve(args={"logk": state["logk"]}, linear=jno.solve.bicgstab(tol=1e-12),
                                 time=jno.solve.theta(case["theta"]))
        return {"trajectory": sol.fn()}
    vals, b = state["batch"].assemble(state["logk"])
    x, _, _ = state["batch"].solve(vals, b, tol=case["tol"], schedule=LAUNCH,
                                   precision="mixed" if case["solver"] == "mixed" else "fp64")
    return {"data": vals, "b": b, "u": x}


def _sizes(case):
    """(elements, unknowns, stored matrix entries) of a box or rectangle."""
    nx, ny, nz, p = case["nx"], case["ny"], case["nz"], case["order"]
    if nz:
        n = (p * nx + 1) * (p * ny + 1) * (p * nz + 1)
        return 6 * nx * ny * nz, n, n * (15 if p == 1 else 28.5)
    n = (p * nx + 1) * (p * ny + 1)
    return 2 * nx * ny, n, n * (7 if p == 1 else 11.5)


def work(case):
    """Bytes and operations of one pass: the coefficient read and the results written once, and for a solve
    the iterations of Jacobi-CG at these sizes, each reading one triangle of the matrix and updating three
    vectors (a matrix-free one the coordinates, the coefficient and the vectors)."""
    path, p = case["path"], case["order"]
    if path == "batch":
        ns = range(case["nx"], case["ny"] + 1)
        w = [math.log((n + 0.5) / (n - 0.5)) for n in ns]
        each = [work(dict(case, path="solve", nx=n, ny=n, nz=n)) for n in ns]
        return {k: case["count"] * sum(a * e[k] for a, e in zip(w, each)) / sum(w) for k in ("bytes", "flops")}
    T, n, nnz = _sizes(case)
    nd = {(1, 0): 3, (2, 0): 6, (1, 1): 4, (2, 1): 10}[(p, 1 if case["nz"] else 0)]
    mean = n ** (1.0 / (3 if case["nz"] else 2))
    out = {"bytes": 8.0 * (T + nnz + 2 * n), "flops": 60.0 * T + 2.0 * nd * nd * T}
    tol = case.get("tol", 1e-12)
    its = mean * (3.6 if case["nz"] else 3.4) * math.log(1 / tol) / math.log(1e8)
    if path == "assemble":
        out["bytes"] += 8.0 * (T + nnz)
        out["flops"] += 2.0 * nd * nd * T
        return out
    half = case.get("solver") == "mixed"
    step = {"bytes": (4.0 if half else 8.0) * ((nnz + n) / 2 + 6 * n), "flops": 2.0 * nnz + 10.0 * n}
    if path == "matfree":
        out["bytes"] = 8.0 * (T + 2 * n)
        step = {"bytes": 8.0 * (T + 3 * n / p ** 3 + 6 * n), "flops": T * (40.0 + 2.0 * nd * nd) + 10.0 * n}
    if path == "march":
        its = case["steps"] * 2.0 * mean * 0.55
        out["bytes"] += 8.0 * (nnz + case["steps"] * n)
    if path == "gradient":
        its *= 2.0
        out["bytes"] += 8.0 * (2 * T + 4 * n)
    return {k: out[k] + its * step[k] for k in out}


# ----------------------------------------------------------------------------------------- exact values
def _dofs(points, cells, order):
    """(cells of unknowns i64[T, nd], number of unknowns), midpoints numbered as the cells first meet them."""
    nv = len(points)
    cells = torch.as_tensor(cells, device="cuda")
    if order == 1:
        return cells, nv
    pairs = [(2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1)] if points.shape[1] == 3 else [(1, 2), (0, 2), (0, 1)]
    ends = torch.stack([torch.stack([cells[:, a], cells[:, b]], 1) for a, b in pairs], 1).reshape(-1, 2)
    key = ends.min(1).values * nv + ends.max(1).values
    found, inverse = torch.unique(key, return_inverse=True)
    first = torch.full((found.numel(),), key.numel(), dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inverse, torch.arange(key.numel(), device="cuda"), "amin")
    number = torch.empty_like(first)
    number[torch.argsort(first)] = torch.arange(found.numel(), device="cuda")
    mids = nv + number[inverse].reshape(len(cells), len(pairs))
    return torch.cat([cells, mids], 1), nv + found.numel()


def _on_boundary(points, cells, dofs, order, n):
    """Mask of the unknowns on facets that one cell alone owns."""
    nvl = points.shape[1] + 1
    cells = torch.as_tensor(cells, device="cuda")
    keep = [[j for j in range(nvl) if j != i] for i in range(nvl)]
    facets = torch.stack([torch.sort(cells[:, k], 1).values for k in keep], 1).reshape(-1, nvl - 1)
    key = facets[:, 0]
    for j in range(1, nvl - 1):
        key = key * len(points) + facets[:, j]
    _, inverse, count = torch.unique(key, return_inverse=True, return_counts=True)
    alone = (count[inverse] == 1).reshape(-1, nvl)
    mask = torch.zeros(n, dtype=torch.bool, device="cuda")
    pairs = [(2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1)] if nvl == 4 else [(1, 2), (0, 2), (0, 1)]
    for i, k in enumerate(keep):
        here = dofs[alone[:, i]]
        local = k + ([nvl + e for e, (a, b) in enumerate(pairs) if a in k and b in k] if order == 2 else [])
        mask[here[:, local].reshape(-1)] = True
    return mask


def _elements(points, cells, order):
    """Unit-coefficient stiffness f64[T, nd, nd], mass f64[T, nd, nd] (order 1) and load f64[T, nd]."""
    dim = points.shape[1]
    X = torch.as_tensor(points, device="cuda")[torch.as_tensor(cells, device="cuda")]
    J = (X[:, 1:] - X[:, :1]).transpose(1, 2)
    vol = torch.linalg.det(J).abs() / math.factorial(dim)
    G = torch.linalg.inv(J)
    G = torch.cat([-G.sum(1, keepdim=True), G], 1)  # gradients of the barycentric coordinates
    nvl = dim + 1
    if order == 1:
        K = vol[:, None, None] * (G @ G.transpose(1, 2))
        M = vol[:, None, None] * (torch.ones(nvl, nvl) + torch.eye(nvl)).to(vol) / ((dim + 1) * (dim + 2))
        return K, M, (vol / nvl)[:, None].expand(-1, nvl)
    # points that integrate quadratics exactly, gradients of the second-order basis there
    b = (5 + 3 * math.sqrt(5)) / 20 if dim == 3 else 2 / 3
    a = (1 - b) / dim
    pairs = [(2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1)] if dim == 3 else [(1, 2), (0, 2), (0, 1)]
    K = 0.0
    for q in range(nvl):
        lam = [b if i == q else a for i in range(nvl)]
        D = [(4 * lam[i] - 1) * G[:, i] for i in range(nvl)]
        D += [4 * (lam[i] * G[:, j] + lam[j] * G[:, i]) for i, j in pairs]
        D = torch.stack(D, 1)
        K = K + (vol / nvl)[:, None, None] * (D @ D.transpose(1, 2))
    ends, mid = ((-0.05, 0.2) if dim == 3 else (0.0, 1.0 / 3.0))
    F = vol[:, None] * torch.tensor([ends] * nvl + [mid] * len(pairs), dtype=torch.float64, device="cuda")
    return K, None, F


def _pattern(dofs, n):
    """(inverse of every element entry into the stored entries, their rows, their columns)."""
    key = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    key, inverse = torch.unique(key, return_inverse=True)
    return inverse, key // n, key % n


def _csr(rows, cols, vals, n):
    crow = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    crow[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(crow, cols, vals, (n, n))


def _cg(A, diag, b, x=None):
    """A x = b (symmetric positive definite) as far as 64 bits go."""
    x = torch.zeros_like(b) if x is None else x.clone()
    stop = 1e-28 * torch.dot(b, b)
    for _ in range(2):  # the second round starts from the residual of the first
        r = b - A @ x
        z = r / diag
        p, rz = z.clone(), torch.dot(r, z)
        for k in range(40000):
            if k % 20 == 0 and bool(torch.dot(r, r) <= stop):
                break
            q = A @ p
            alpha = rz / torch.dot(p, q)
            x += alpha * p
            r -= alpha * q
            z = r / diag
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
    return x


def _scatter(inverse, size, values):
    return torch.zeros(size, dtype=torch.float64, device="cuda").index_add_(0, inverse, values.reshape(-1))


def _assembled(dofs, n, fixed, K, F, k):
    """(rows, cols, values, load, inverse) of the system with the boundary rows and columns eliminated."""
    inverse, rows, cols = _pattern(dofs, n)
    free = (~fixed).to(torch.float64)
    mask = free[dofs]
    vals = _scatter(inverse, rows.numel(), k[:, None, None] * K * mask[:, :, None] * mask[:, None, :])
    vals[(rows == cols) & fixed[rows]] = 1.0
    load = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dofs.reshape(-1), (F * mask).reshape(-1))
    return rows, cols, vals, load, inverse


def exact(case, seed):
    path, order = case["path"], case["order"]
    if path == "batch":
        parts = [_mesh(n, n, n, "lattice", [seed, i]) for i, n in enumerate(_sides(case))]
        offset = np.cumsum([0] + [len(p) for p, _ in parts])
        points = np.concatenate([p for p, _ in parts])
        cells = np.concatenate([c + o for (_, c), o in zip(parts, offset)])
    else:
        points, cells = _mesh(case["nx"], case["ny"], case["nz"], case["numbering"], seed)
    dofs, n = _dofs(points, cells, order)
    fixed = _on_boundary(points, cells, dofs, order, n)
    K, M, F = _elements(points, cells, order)
    if case.get("param") == "nodal":
        p = _log_field(len(points), seed)[dofs]
        b = (5 + 3 * math.sqrt(5)) / 20 if points.shape[1] == 3 else 2 / 3
        a = (1 - b) / points.shape[1]
        at = torch.exp(a * p.sum(1, keepdim=True) + (b - a) * p)  # k at the points of the degree-2 rule
        k = at.mean(1)
    else:
        k = torch.exp(_log_field(len(cells), seed))
    if path == "march":
        return {"trajectory": _march(case, points, dofs, n, fixed, K, M, F, k)}
    rows, cols, vals, load, inverse = _assembled(dofs, n, fixed, K, F, k)
    if path == "assemble":
        mask = (~fixed).to(torch.float64)[dofs]
        back = _log_field(rows.numel(), seed + 1)[inverse].reshape(K.shape)
        S = (back * K * mask[:, :, None] * mask[:, None, :]).sum((1, 2))
        if case["param"] == "nodal":
            # d k / d p_i: every point of the rule weighs vertex i by its barycentric coordinate
            grad_k = (a * at.sum(1, keepdim=True) + (b - a) * at) / at.shape[1]
            grad = torch.zeros(len(points), dtype=torch.float64, device="cuda")
            grad.index_add_(0, dofs.reshape(-1), (S[:, None] * grad_k).reshape(-1))
        else:
            grad = S * k
        return {"data": vals, "b": load, "grad": grad}
    diag = vals[rows == cols]
    A = _csr(rows, cols, vals, n)
    u = _cg(A, diag, load)
    if path == "gradient":
        target = _log_field(n, seed + 1) * 0.1
        mass = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dofs.reshape(-1), F.reshape(-1))
        loss = 0.5 * torch.sum(mass * (u - target) ** 2)
        lam = _cg(A, diag, mass * (u - target))
        free = (~fixed).to(torch.float64)
        grad = -k * torch.einsum("ea,eab,eb->e", (free * lam)[dofs], K, (free * u)[dofs])
        return {"u": u, "loss": loss, "grad": grad}
    if path == "matfree":
        return {"b": load, "u": u}
    return {"data": vals, "b": load, "u": u}


def _march(case, points, dofs, n, fixed, K, M, F, k):
    """The theta steps on the free unknowns (the boundary stays at its initial value, zero)."""
    theta, dt = case["theta"], DT
    inverse, rows, cols = _pattern(dofs, n)
    free = (~fixed).to(torch.float64)
    both = free[rows] * free[cols]
    stiff = _scatter(inverse, rows.numel(), k[:, None, None] * K) * both
    mass = _scatter(inverse, rows.numel(), M) * both
    load = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dofs.reshape(-1), F.reshape(-1)) * free
    left = mass + theta * dt * stiff
    left[(rows == cols) & fixed[rows]] = 1.0
    S, R = _csr(rows, cols, left, n), _csr(rows, cols, mass - (1 - theta) * dt * stiff, n)
    diag = left[rows == cols]
    u = torch.sin(math.pi * torch.as_tensor(points, device="cuda")).prod(1)
    states = [u]
    for _ in range(case["steps"]):
        u = _cg(S, diag, R @ (free * u) + dt * load, free * u)
        states.append(u)
    return torch.stack(states)
