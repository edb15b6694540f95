"""The performance cases of the library: what a program that discretizes and solves with it spends its
time on, each through the Python entry points, over the sizes the tests, the benchmark and ordinary
use give them. `listed()` names them, `draw(rng)` gives another case of the same ranges.

Every kind of case is one pass of a user's inner loop on given coefficients:

  elliptic  assemble -div(kappa grad u) = f with Dirichlet constraints, then solve (FP64 or mixed)
  apply     assemble the operator and the load vector, then one matrix-vector product
  mesh      the same as elliptic on an unstructured tetrahedral mesh
  q2        order-2 elements with the diffusion at the quadrature points, assemble and solve
  adjoint   SWIPDG forward solve and the log-kappa gradient of 0.5 |u - u_d|^2 (adjoint solve)
  batch     a parameter sweep over meshes of uneven size, assembled and solved in one call
  fv        explicit finite-volume time stepping (one state or a batch of states)
"""
import importlib
import itertools
import math

import numpy as np
import torch

gdt = importlib.import_module("dune-gdt_gb300")

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------------------------- the cases ---
def listed():
    return [
        # The reference's introductory problem, the stationary heat equation on 64^2 squares: a few thousand
        # unknowns, where latency and launches are the whole cost. Parameter studies and tests repeat it
        # (unit diffusion, a source per element).
        {"name": "heat_2d_q1_64_fp64", "kind": "elliptic", "element": "q1", "nx": 64, "ny": 64, "nz": 0,
         "mapped": False, "kappa": "one", "precision": "fp64", "tol": 1e-10},
        # 3D heterogeneous diffusion at the benchmark's size, in both precisions a caller can choose.
        {"name": "heat_3d_q1_128_fp64", "kind": "elliptic", "element": "q1", "nx": 128, "ny": 128, "nz": 128,
         "mapped": False, "kappa": "lognormal", "precision": "fp64", "tol": 1e-11},
        {"name": "heat_3d_q1_128_mixed", "kind": "elliptic", "element": "q1", "nx": 128, "ny": 128, "nz": 128,
         "mapped": False, "kappa": "lognormal", "precision": "mixed", "tol": 1e-11},
        # An ordinary production size with odd extents, on simplices, as most runs that are not benchmarks.
        {"name": "heat_3d_p1_45x64x51_fp64", "kind": "elliptic", "element": "p1", "nx": 45, "ny": 64, "nz": 51,
         "mapped": False, "kappa": "lognormal", "precision": "fp64", "tol": 1e-11},
        # A curved (mapped) hexahedral grid: geometry per element, mixed precision on the assembled values.
        {"name": "heat_3d_mapped_67x60x72_mixed", "kind": "elliptic", "element": "q1", "nx": 67, "ny": 60, "nz": 72,
         "mapped": True, "kappa": "lognormal", "precision": "mixed", "tol": 1e-11},
        # Assembly and one product, as in time stepping, reduced bases and outer solvers of the caller's own.
        {"name": "assemble_apply_3d_q1_96x101x90", "kind": "apply", "element": "q1", "nx": 96, "ny": 101, "nz": 90},
        # An imported tetrahedral mesh whose vertex numbers carry no lattice order.
        {"name": "heat_mesh_tets_40", "kind": "mesh", "cells": 40, "tol": 1e-11},
        # Order-2 elements with a coefficient that varies inside the elements.
        {"name": "heat_3d_q2_28", "kind": "q2", "nx": 28, "ny": 28, "nz": 28, "tol": 1e-10},
        # Forward and backward: the gradient of a misfit with respect to a high-contrast SWIPDG coefficient.
        {"name": "adjoint_swipdg_128", "kind": "adjoint", "cells": 128, "tol": 1e-12},
        # Parametric sweep over meshes of uneven size in one call (the sides of the benchmark's sweep).
        {"name": "batch_p1_64_fp64", "kind": "batch", "element": "p1", "problems": 64, "sides": "64,128,256,512",
         "kappa": "quadrants", "precision": "fp64", "tol": 1e-10},
        # 2D Burgers, local Lax-Friedrichs, SSP-RK2 on one large state; linear transport with upwinding on a
        # batch of small ones (in- and outflow boundaries), where a step is a launch or two.
        {"name": "fv_burgers_2d_2048_ssp2", "kind": "fv", "nx": 2048, "ny": 2048, "nz": 0, "flux": "burgers",
         "numflux": "lf", "method": "ssp2", "steps": 20, "batch": 1, "boundary": "periodic"},
        {"name": "fv_transport_2d_16x120x97_euler", "kind": "fv", "nx": 120, "ny": 97, "nz": 0, "flux": "transport",
         "numflux": "upwind", "method": "euler", "steps": 50, "batch": 16, "boundary": "inflow"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["elliptic", "elliptic", "elliptic", "apply", "mesh", "q2", "adjoint", "batch", "fv", "fv"])
    if kind in ("elliptic", "apply"):
        dim = rng.choice([2, 3, 3])
        mean = _log_int(rng, 24, 400) if dim == 2 else _log_int(rng, 10, 112)
        ext = [max(4, int(mean * rng.uniform(0.85, 1.14))) for _ in range(dim)] + [0] * (3 - dim)
        case = {"kind": kind, "element": rng.choice(["q1", "q1", "p1"]), "nx": ext[0], "ny": ext[1], "nz": ext[2]}
        if kind == "elliptic":
            case["mapped"] = rng.random() < 0.25
            case["kappa"] = rng.choice(["lognormal", "lognormal", "one"])
            case["precision"] = rng.choice(["fp64", "mixed"])
            case["tol"] = 1e-11
        return case
    if kind == "mesh":
        return {"kind": "mesh", "cells": _log_int(rng, 6, 44), "tol": 1e-11}
    if kind == "q2":
        m = _log_int(rng, 5, 26)
        return {"kind": "q2", "nx": m, "ny": max(2, int(m * rng.uniform(0.8, 1.2))),
                "nz": max(2, int(m * rng.uniform(0.8, 1.2))), "tol": 1e-10}
    if kind == "adjoint":
        return {"kind": "adjoint", "cells": _log_int(rng, 12, 128), "tol": 1e-12}
    if kind == "batch":
        kappa = rng.choice(["quadrants", "elements"])  # quadrants take even sides
        sides = sorted(_log_int(rng, 20, 400) for _ in range(rng.randint(1, 4)))
        sides = [s + s % 2 for s in sides] if kappa == "quadrants" else sides
        return {"kind": "batch", "element": rng.choice(["p1", "p1", "q1"]), "problems": rng.randint(4, 64),
                "sides": ",".join(str(s) for s in sides), "kappa": kappa,
                "precision": rng.choice(["fp64", "fp64", "mixed"]), "tol": 1e-10}
    dim = rng.choice([1, 2, 2, 2, 3])
    cells = _log_int(rng, 2000, 3000000)  # per state
    side = cells ** (1.0 / dim)
    ext = [max(4, int(side * rng.uniform(0.8, 1.2))) for _ in range(dim)] + [0] * (3 - dim)
    batch = rng.choice([1, 1, 4, 16]) if cells < 200000 else 1
    return {"kind": "fv", "nx": ext[0], "ny": ext[1], "nz": ext[2], "flux": rng.choice(["burgers", "transport"]),
            "numflux": rng.choice(["lf", "upwind"]), "method": rng.choice(["ssp2", "euler"]),
            "steps": rng.randint(8, 40), "batch": batch, "boundary": rng.choice(["periodic", "inflow"])}


# ------------------------------------------------------------------------------ inputs from the seed ---
def _extents(case):
    return [case[k] for k in ("nx", "ny", "nz") if case.get(k, 0) > 0]


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, sum(case["kind"].encode())])


def _dev(a):
    return torch.tensor(a, device=DEVICE)


def _lattice(n):
    """Vertices of the unit cube's grid with n[a] cells per axis, x fastest."""
    axes = [np.linspace(0.0, 1.0, k + 1) for k in n]
    grids = np.meshgrid(*axes[::-1], indexing="ij")[::-1]
    return np.stack([g.reshape(-1) for g in grids], -1)


def _wavy(n):
    """The lattice moved by x_a -> x_a + 0.04 sin(2 pi x_a)(1 + x_{a+1}): a curved grid of the same box."""
    X = _lattice(n)
    Y = X.copy()
    for a in range(len(n)):
        Y[:, a] += 0.04 * np.sin(2 * np.pi * X[:, a]) * (1.0 + X[:, (a + 1) % len(n)])
    return Y


def _corners(n):
    """Vertex numbers of every cube [ncubes, 2^d], corner bit a = offset along axis a."""
    idx = np.indices(n[::-1]).reshape(len(n), -1)[::-1]  # idx[a] of every cube, x fastest
    strides = np.cumprod([1] + [k + 1 for k in n[:-1]])
    base = sum(i * s for i, s in zip(idx, strides))
    off = [sum(((c >> a) & 1) * strides[a] for a in range(len(n))) for c in range(2 ** len(n))]
    return base[:, None] + np.array(off)[None, :]


def _simplices(n):
    """Vertex numbers of the Kuhn split [ncubes * d!, d + 1]: element = cube * d! + permutation."""
    c, d = _corners(n), len(n)
    parts = []
    for perm in itertools.permutations(range(d)):
        corner = [sum(1 << a for a in perm[:m]) for m in range(d + 1)]
        parts.append(c[:, corner])
    return np.stack(parts, 1).reshape(-1, d + 1)


def _kappa(case, seed, ne):
    if case.get("kappa") == "one":
        return np.ones(ne)
    return np.exp(_rng(case, seed).standard_normal(ne))


def _source(case, seed, ne):
    """The source: one value per element where the diffusion is the unit one, else 1."""
    if case.get("kappa") == "one":
        return 1.0 + 0.5 * _rng(case, seed).uniform(-1, 1, ne)
    return np.ones(ne)


def _elements(case):
    n = _extents(case)
    return math.prod(n) * (math.factorial(len(n)) if case["element"] == "p1" else 1)


def _mesh(case, seed):
    """Jittered Kuhn tetrahedra of the unit cube, vertices renumbered by a random permutation:
    coordinates, element vertex lists, boundary vertices, kappa per element."""
    n = case["cells"]
    rng = _rng(case, seed)
    X, cells = _lattice([n] * 3), _simplices([n] * 3)
    inner = np.all((X > 0) & (X < 1), axis=1)
    moved = X.copy()
    moved[inner] += (0.2 / n) * rng.uniform(-1, 1, (int(inner.sum()), 3))
    perm = rng.permutation(len(X))
    xyz, boundary = np.empty_like(moved), np.empty(len(X), dtype=bool)
    xyz[perm], boundary[perm] = moved, ~inner
    return xyz, perm[cells], boundary, np.exp(rng.standard_normal(len(cells)))


def _q2_kappa(case, seed, points):
    """kappa at points [element, q, 3]: lognormal per element times a smooth factor."""
    ke = _rng(case, seed).standard_normal(points.shape[0])
    s = torch.sin(2 * math.pi * points)
    return torch.exp(torch.tensor(ke, device=points.device))[:, None] * (1 + 0.5 * s[..., 0] * s[..., 1] * s[..., 2])


def _adjoint_inputs(case, seed):
    """log kappa ~ N(0, 1) with random 8-cell-wide horizontal channels of contrast 1e4, and a target."""
    n = case["cells"]
    rng = _rng(case, seed)
    ne = 2 * n * n
    channel = rng.random((n + 7) // 8) < 0.5
    stripe = channel[((np.arange(ne) // 2) // n) // 8]
    logk = rng.standard_normal(ne) + stripe * math.log(1e4)
    target = 0.05 * rng.standard_normal(3 * ne)
    return logk, target


def _sides(case):
    s = [int(v) for v in case["sides"].split(",")]
    return [s[i % len(s)] for i in range(case["problems"])]


def _batch_kappa(case, seed):
    """Per problem: mu of the four quadrants, or lognormal values per element."""
    rng = _rng(case, seed)
    if case["kappa"] == "quadrants":
        return list(rng.uniform(0.1, 10.0, (case["problems"], 4)))
    per_cell = 2 if case["element"] == "p1" else 1
    return [np.exp(rng.standard_normal(per_cell * s * s)) for s in _sides(case)]


FV_INFLOW = 0.25
FV_VELOCITY = (0.7, -0.4, 0.3)


def _fv_state(case, seed):
    """Sums of eight seeded Gaussian bumps of both signs per state, flattened with x fastest."""
    n = _extents(case)
    rng = _rng(case, seed)
    out = []
    for _ in range(case["batch"]):
        u = np.zeros(n[::-1])
        for _ in range(8):
            w, term = rng.uniform(0.02, 0.15), rng.uniform(-1, 1)
            for a, k in enumerate(n):
                x = (np.arange(k) + 0.5) / k - rng.uniform(0, 1)
                x -= np.round(x)
                shape = [1] * len(n)
                shape[len(n) - 1 - a] = k
                term = term * np.exp(-x * x / (2 * w * w)).reshape(shape)
            u += term
        out.append(u.reshape(-1))
    return np.concatenate(out)


def _fv_dt(case):
    """Half of the bound for speeds up to one per axis (a few bumps can add up to about two)."""
    return 0.2 / sum(_extents(case))


# ---------------------------------------------------------------------------------- prepare and run ---
def _laplace(grid, space, kappa):
    op = gdt.MatrixOperator(grid, space)
    op += gdt.LocalElementIntegralBilinearForm(gdt.LocalLaplaceIntegrand(kappa))
    return op


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("elliptic", "apply"):
        n = _extents(case)
        grid = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, simplex=case["element"] == "p1")
        if case.get("mapped"):
            grid.map_vertices(_wavy(n))
        space = gdt.ContinuousLagrangeSpace(grid, 1)
        kappa = 1.0 if case.get("kappa") == "one" else _dev(_kappa(case, seed, grid.num_elements))
        s["op"] = _laplace(grid, space, kappa)
        s["rhs"] = torch.zeros(space.num_DoFs, dtype=torch.float64, device=DEVICE)
        if kind == "apply":
            s["x"] = _dev(_rng(case, seed + 1).standard_normal(space.num_DoFs))
            s["y"] = torch.zeros_like(s["rhs"])
        else:
            s["opts"] = {"tol": case["tol"], "precision": case["precision"]}
        s["force"] = _dev(_source(case, seed, grid.num_elements)) if case.get("kappa") == "one" else 1.0
    elif kind == "mesh":
        xyz, cells, _, kappa = _mesh(case, seed)
        mesh = gdt.make_simplex_mesh(xyz, cells)
        space = gdt.ContinuousLagrangeSpace(mesh, 1)
        s["op"] = _laplace(mesh, space, _dev(kappa))
        s["rhs"] = torch.zeros(space.num_DoFs, dtype=torch.float64, device=DEVICE)
        s["opts"] = {"tol": case["tol"]}
    elif kind == "q2":
        grid = gdt.make_cube_grid([0.0] * 3, [1.0] * 3, _extents(case))
        space = gdt.ContinuousLagrangeSpace(grid, 2)
        s["op"] = _laplace(grid, space, _q2_kappa(case, seed, space.quadrature_points()).contiguous())
        s["rhs"] = torch.zeros(space.num_DoFs, dtype=torch.float64, device=DEVICE)
        s["opts"] = {"tol": case["tol"]}
    elif kind == "adjoint":
        n = case["cells"]
        grid = gdt.make_cube_grid([0.0, 0.0], [1.0, 1.0], [n, n], simplex=True)
        logk, target = _adjoint_inputs(case, seed)
        s["problem"] = gdt.DiffusionProblem(grid, dg=True, solver_opts={"tol": case["tol"], "max_iter": 400000})
        s["logk"], s["target"] = _dev(logk), _dev(target)
    elif kind == "batch":
        s["batch"] = gdt.BatchedDiffusion(_sides(case), element=case["element"])
        kappa = _dev(np.concatenate(_batch_kappa(case, seed)))
        s["kappa"] = {"mu": kappa} if case["kappa"] == "quadrants" else {"kappa": kappa}
    elif kind == "fv":
        n = _extents(case)
        grid = gdt.make_cube_grid([0.0] * len(n), [1.0] * len(n), n, periodic=case["boundary"] == "periodic")
        space = gdt.FiniteVolumeSpace(grid)
        flux = gdt.BurgersFlux() if case["flux"] == "burgers" else gdt.LinearTransportFlux(FV_VELOCITY[:len(n)])
        num = {"lf": gdt.NumericalLaxFriedrichsFlux, "upwind": gdt.NumericalUpwindFlux}[case["numflux"]](flux)
        op = gdt.AdvectionFvOperator(grid, num, space)
        if case["boundary"] == "inflow":  # a prescribed state on the lower sides, outflow on the upper ones
            op.append(gdt.BoundaryTreatmentByCustomExtrapolation(FV_INFLOW), filter=["-x", "-y", "-z"][:len(n)])
            op.append(gdt.BoundaryTreatmentByCustomExtrapolation(), filter=["+x", "+y", "+z"][:len(n)])
        s["u0"] = _dev(_fv_state(case, seed))
        s["stepper"] = gdt.ExplicitRungeKuttaTimeStepper(op, torch.zeros_like(s["u0"]), method=case["method"])
        s["dt"] = _fv_dt(case)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        op = state["op"]
        op.assemble(rhs=state["rhs"], force=1.0, dirichlet=True)
        op.apply(state["x"], state["y"])
        values = op.csr()[2]
        values.owner = op  # a view of the operator's memory: it lives as long as the operator
        return {"values": values, "rhs": state["rhs"], "y": state["y"]}
    if kind in ("elliptic", "mesh", "q2"):
        op = state["op"]
        op.assemble(rhs=state["rhs"], force=state.get("force", 1.0), dirichlet=True)
        return {"rhs": state["rhs"], "u": op.apply_inverse(state["rhs"], opts=state["opts"])}
    if kind == "adjoint":
        logk = state["logk"].detach().clone().requires_grad_(True)
        u = gdt.DiffusionSolve.apply(logk, state["problem"])
        misfit = 0.5 * torch.sum((u - state["target"]) ** 2)
        misfit.backward()
        return {"u": u.detach(), "gradient": logk.grad}
    if kind == "batch":
        return {"u": state["batch"].solve(**state["kappa"], precision=case["precision"], tol=case["tol"])}
    stepper = state["stepper"]
    stepper.u.copy_(state["u0"])
    stepper.step(state["dt"], case["steps"])
    return {"u": stepper.u}


# ----------------------------------------------------------------------------------------- the work ---
def work(case):
    """Inputs read once and outputs written once. Operations: the assembly (one multiply-add per entry of
    every element matrix) and, for solves, CG with Jacobi: its iterations grow with the cells per axis
    (measured factors: 3.4 in 3D and 2 in 2D with lognormal or unit kappa, 12 for SWIPDG with channels, 6 for
    order 2, 4.2 for the sweep), each a multiply-add per nonzero and about ten operations per unknown."""
    kind = case["kind"]

    def solve(iterations, nnz, ndof):
        return iterations * (2.0 * nnz + 10.0 * ndof)

    if kind in ("elliptic", "apply"):
        n, ne = _extents(case), _elements(case)
        d = len(n)
        ndof = math.prod(k + 1 for k in n)
        L = d + 1 if case["element"] == "p1" else 2 ** d
        nnz = ndof * ((7 if d == 2 else 15) if case["element"] == "p1" else 3 ** d)
        if kind == "apply":
            return {"bytes": 8.0 * (ne + nnz + 3 * ndof), "flops": 2.0 * L * L * ne + 2.0 * nnz}
        its = (2.0 if d == 2 else 3.4) * max(n)
        return {"bytes": 8.0 * (ne + 2 * ndof),
                "flops": 2.0 * L * L * ne + solve(its, nnz, ndof)}
    if kind == "mesh":
        ne, ndof = 6 * case["cells"] ** 3, (case["cells"] + 1) ** 3
        return {"bytes": 8.0 * (ne * 3 + ndof * 5), "flops": 32.0 * ne + solve(3.4 * case["cells"], 15 * ndof, ndof)}
    if kind == "q2":
        n = _extents(case)
        ne, ndof = math.prod(n), math.prod(2 * k + 1 for k in n)
        return {"bytes": 8.0 * (64 * ne + 2 * ndof), "flops": 2.0 * 27 * 27 * ne + solve(6.0 * max(n), 64 * ndof, ndof)}
    if kind == "adjoint":
        ne = 2 * case["cells"] ** 2
        return {"bytes": 8.0 * (2 * ne + 6 * ne), "flops": 800.0 * ne + 2 * solve(12.0 * case["cells"], 36 * ne, 3 * ne)}
    if kind == "batch":
        width = 7 if case["element"] == "p1" else 9
        dofs = [(s + 1) ** 2 for s in _sides(case)]
        values = 4 * len(dofs) if case["kappa"] == "quadrants" else 2 * sum(dofs)
        return {"bytes": 8.0 * (sum(dofs) + values),
                "flops": sum(solve(4.2 * s, width * m, m) for s, m in zip(_sides(case), dofs))}
    cells = math.prod(_extents(case)) * case["batch"]
    stages = 2 if case["method"] == "ssp2" else 1
    return {"bytes": 16.0 * cells, "flops": cells * case["steps"] * stages * (2.0 + 5.0 * len(_extents(case)))}


# --------------------------------------------------------------------- the same in plain torch, 64 bits ---
def _csr(dofs, Ke, ndof, boundary):
    """Sparse matrix of the element matrices Ke [ne, L, L] with unit rows and columns at the boundary."""
    L = dofs.shape[1]
    rows = dofs[:, :, None].expand(-1, L, L).reshape(-1)
    cols = dofs[:, None, :].expand(-1, L, L).reshape(-1)
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), Ke.reshape(-1), (ndof, ndof)).coalesce()
    (i, j), v = A.indices(), A.values().clone()
    if boundary is not None:
        v[boundary[i] | boundary[j]] = 0.0
        v[boundary[i] & (i == j)] = 1.0
    rp = torch.zeros(ndof + 1, dtype=torch.int64, device=v.device)
    rp[1:] = torch.cumsum(torch.bincount(i, minlength=ndof), 0)
    dv = v[i == j]
    return torch.sparse_csr_tensor(rp, j, v, (ndof, ndof)), dv


def _cg(A, diag, b, max_iter=40000):
    """Jacobi-preconditioned CG to the rounding level, restarted from the true residual."""
    x, dinv = torch.zeros_like(b), 1.0 / diag
    r, target, done = b.clone(), 1e-15 * b.norm(), 0
    for _ in range(3):
        z = dinv * r
        p, rz = z.clone(), torch.dot(r, z)
        while done < max_iter:
            for _ in range(25):
                q = A @ p
                alpha = rz / torch.dot(p, q)
                x = torch.addcmul(x, alpha, p)
                r = torch.addcmul(r, -alpha, q)
                z = dinv * r
                new = torch.dot(r, z)
                p = torch.addcmul(z, new / rz, p)
                rz = new
            done += 25
            if not bool(r.norm() > target) or not bool(rz > 0):
                break
        r = b - A @ x
        if not bool(r.norm() > 4 * target):
            break
    return x


def _simplex_stiffness(X, kappa):
    """Element matrices [ne, d+1, d+1] and volumes of P1 on corners X [ne, d+1, d]."""
    d = X.shape[2]
    J = (X[:, 1:, :] - X[:, :1, :]).transpose(1, 2)
    ref = torch.cat([-torch.ones(1, d), torch.eye(d)]).to(X)
    G = ref[None] @ torch.linalg.inv(J)
    vol = torch.linalg.det(J).abs() / math.factorial(d)
    return (kappa * vol)[:, None, None] * (G @ G.transpose(1, 2)), vol


def _cube_basis(x):
    """Values [2^d] and gradients [2^d, d] of the multilinear basis at one reference point."""
    d = len(x)
    f = [[(1 - x[a], x[a])[(c >> a) & 1] for a in range(d)] for c in range(2 ** d)]
    df = [[(-1.0, 1.0)[(c >> a) & 1] for a in range(d)] for c in range(2 ** d)]
    grad = [[math.prod(df[c][b] if b == a else f[c][b] for b in range(d)) for a in range(d)] for c in range(2 ** d)]
    return np.array([math.prod(v) for v in f]), np.array(grad)


def _cube_stiffness(X, kappa):
    """Element matrices and midpoint |det J| of Q1 on corners X [ne or 1, 2^d, d], 2 Gauss points per axis."""
    d = X.shape[2]
    Ke = 0.0
    for q in itertools.product([0.5 - math.sqrt(1 / 12), 0.5 + math.sqrt(1 / 12)], repeat=d):
        ref = torch.tensor(_cube_basis(q)[1]).to(X)
        J = torch.einsum("ecr,ck->erk", X, ref)
        G = ref[None] @ torch.linalg.inv(J)
        Ke = Ke + (torch.linalg.det(J).abs() / 2 ** d)[:, None, None] * (G @ G.transpose(1, 2))
    mid = torch.tensor(_cube_basis([0.5] * d)[1]).to(X)
    return kappa[:, None, None] * Ke, torch.linalg.det(torch.einsum("ecr,ck->erk", X, mid)).abs()


def _load(dofs, per_element, ndof, boundary):
    b = torch.zeros(ndof, dtype=torch.float64, device=dofs.device)
    b.index_add_(0, dofs.reshape(-1), per_element[:, None].expand(-1, dofs.shape[1]).reshape(-1))
    b[boundary] = 0.0
    return b


def _exact_structured(case, seed):
    n = _extents(case)
    d = len(n)
    X = _dev(_wavy(n) if case.get("mapped") else _lattice(n))
    lat = _lattice(n)
    boundary = _dev(np.any((lat == 0) | (lat == 1), axis=1))
    kappa = _dev(_kappa(case, seed, _elements(case)))
    if case["element"] == "p1":
        dofs = _dev(_simplices(n))
        Ke, vol = _simplex_stiffness(X[dofs], kappa)
        share = vol / (d + 1)
    else:
        dofs = _dev(_corners(n))
        corners = X[dofs] if case.get("mapped") else torch.tensor(
            [[[((c >> a) & 1) / n[a] for a in range(d)] for c in range(2 ** d)]], dtype=torch.float64, device=DEVICE)
        Ke, det = _cube_stiffness(corners, kappa)
        share = (det / 2 ** d).expand(len(dofs))
    A, diag = _csr(dofs, Ke, len(X), boundary)
    return A, diag, _load(dofs, share * _dev(_source(case, seed, len(dofs))), len(X), boundary)


def _q2_numbering(n):
    """DoF of every point of the half-step lattice (x fastest): cells, faces, edges and vertices, cells and
    vertices in their own order, faces and edges by first appearance in the walk over the elements."""
    points = [(x, y, z) for z, y, x in itertools.product(range(3), repeat=3)]
    m = [2 * k + 1 for k in n]
    cell = np.indices(n[::-1]).reshape(3, -1)[::-1]
    dof, at = np.empty(math.prod(m), dtype=np.int64), 0
    for codim in range(3):
        o = np.array([p for p in points if sum(c != 1 for c in p) == codim])
        pts = [2 * cell[a][:, None] + o[None, :, a] for a in range(3)]
        keys, first = np.unique((pts[0] + m[0] * (pts[1] + m[1] * pts[2])).reshape(-1), return_index=True)
        dof[keys[np.argsort(first)]] = at + np.arange(len(keys))
        at += len(keys)
    vertex = np.indices([k + 1 for k in n[::-1]]).reshape(3, -1)[::-1]
    dof[2 * vertex[0] + m[0] * (2 * vertex[1] + m[1] * 2 * vertex[2])] = at + np.arange(vertex.shape[1])
    return dof


def _exact_q2(case, seed):
    n = _extents(case)
    m = [2 * k + 1 for k in n]
    cell = np.indices(n[::-1]).reshape(3, -1)[::-1]
    local = list(itertools.product(range(3), repeat=3))  # (z, y, x) offsets of the 27 lattice points
    lattice = np.stack([2 * cell[0] + x + m[0] * (2 * cell[1] + y + m[1] * (2 * cell[2] + z)) for z, y, x in local], 1)
    number = _dev(_q2_numbering(n))
    g, w = np.polynomial.legendre.leggauss(4)
    g, w = (g + 1) / 2, w / 2
    val = np.stack([(1 - g) * (1 - 2 * g), 4 * g * (1 - g), g * (2 * g - 1)])
    der = np.stack([4 * g - 3, 4 - 8 * g, 4 * g - 1])
    pts = _dev(np.array([(g[i], g[j], g[k]) for k in range(4) for j in range(4) for i in range(4)]))
    wq = np.array([w[i] * w[j] * w[k] for k in range(4) for j in range(4) for i in range(4)])
    grads = [_dev(np.stack([np.einsum("k,j,i->kji", *[(der if a == ax else val)[o] for ax, o in ((2, z), (1, y), (0, x))]
                                      ).reshape(-1) for z, y, x in local]) * n[a]) for a in range(3)]
    h = _dev(1.0 / np.array(n))
    kappa = _q2_kappa(case, seed, (_dev(cell.T.astype(np.float64))[:, None, :] + pts[None]) * h)
    pairs = sum(G[:, None, :] * G[None, :, :] for G in grads) * _dev(wq / math.prod(n))
    Ke = (kappa @ pairs.reshape(27 * 27, 64).T).reshape(-1, 27, 27)
    i = np.stack(np.unravel_index(np.arange(math.prod(m)), m[::-1])[::-1], 1)
    edge = _dev(np.any((i == 0) | (i == np.array(m) - 1), axis=1))
    boundary = torch.zeros_like(edge)
    boundary[number] = edge
    dofs = number[_dev(lattice)]
    b1 = val @ w  # integrals of the 1D basis
    load = _dev(np.array([b1[z] * b1[y] * b1[x] for z, y, x in local]) / math.prod(n))
    b = torch.zeros(math.prod(m), dtype=torch.float64, device=DEVICE)
    b.index_add_(0, dofs.reshape(-1), load[None].expand(len(dofs), -1).reshape(-1))
    b[boundary] = 0.0
    A, diag = _csr(dofs, Ke, math.prod(m), boundary)
    return A, diag, b


def _exact_adjoint(case, seed):
    """SWIPDG (symmetric, weights and penalties from kappa, sigma 8 inside and 14 on the boundary, h = |face|)
    on the Kuhn triangles: every face adds outer products over the six (three) unknowns beside it."""
    n = case["cells"]
    logk, target = (_dev(a) for a in _adjoint_inputs(case, seed))
    cells, lat = _simplices([n, n]), _lattice([n, n])
    ne = len(cells)
    X = _dev(lat)[_dev(cells)]
    unit, vol = _simplex_stiffness(X, torch.ones(ne, dtype=torch.float64, device=DEVICE))
    G = torch.linalg.inv((X[:, 1:, :] - X[:, :1, :]).transpose(1, 2))
    G = torch.cat([-G.sum(1, keepdim=True), G], 1)  # [ne, 3, 2]
    ends = np.array([(0, 1), (0, 2), (1, 2)])
    sides = np.sort(cells[:, ends], axis=2).reshape(-1, 2)
    order = np.lexsort((sides[:, 1], sides[:, 0]))
    same = np.all(sides[order[1:]] == sides[order[:-1]], axis=1)
    first, second = order[:-1][same], order[1:][same]
    alone = np.setdiff1d(order, np.concatenate([first, second]))

    def trace(side, v0):
        """Of a side: element, traces [f, 3, 2] at its two vertices in order (v0 first), inner data."""
        e, k = side // 3, side % 3
        t = np.zeros((len(side), 3, 2))
        lo = np.where(cells[e, ends[k, 0]] == v0, ends[k, 0], ends[k, 1])
        hi = ends[k, 0] + ends[k, 1] - lo
        t[np.arange(len(side)), lo, 0] = t[np.arange(len(side)), hi, 1] = 1.0
        return e, _dev(t)

    def geometry(side):
        p = _dev(lat)[_dev(sides[side])]
        along = p[:, 1] - p[:, 0]
        length = along.norm(dim=1)
        normal = torch.stack([along[:, 1], -along[:, 0]], 1) / length[:, None]
        e = _dev(side // 3)
        out = ((p[:, 0] - X[e].mean(1)) * normal).sum(1)
        return length, normal * torch.sign(out)[:, None]

    edge_mass = torch.tensor([[2.0, 1.0], [1.0, 2.0]], dtype=torch.float64, device=DEVICE) / 6
    half = torch.full((2,), 0.5, dtype=torch.float64, device=DEVICE)
    ei, ti = trace(first, sides[first, 0])
    eo, to = trace(second, sides[first, 0])
    li, ni = geometry(first)
    eb, tb = trace(alone, sides[alone, 0])
    lb, nb = geometry(alone)
    gi, go = (G[_dev(ei)] * ni[:, None, :]).sum(2), (G[_dev(eo)] * ni[:, None, :]).sum(2)
    gb = (G[_dev(eb)] * nb[:, None, :]).sum(2)
    jump = torch.cat([ti, -to], 1)  # [f, 6, 2]
    jump_mean, tb_mean = jump @ half, tb @ half
    jump_mass, tb_mass = jump @ edge_mass @ jump.transpose(1, 2), tb @ edge_mass @ tb.transpose(1, 2)
    dof = torch.arange(3 * ne, device=DEVICE).reshape(ne, 3)
    dof_f = torch.cat([dof[_dev(ei)], dof[_dev(eo)]], 1)
    dof_b = dof[_dev(eb)]

    def blocks(k):
        kin, kout, kb = k[_dev(ei)], k[_dev(eo)], k[_dev(eb)]
        half_harmonic = kin * kout / (kin + kout)  # weight_minus kin = weight_plus kout
        mean = half_harmonic[:, None] * torch.cat([gi, go], 1)
        c = (li[:, None] * mean)[:, :, None] * jump_mean[:, None, :]
        inner = -(c + c.transpose(1, 2)) + (8.0 * half_harmonic)[:, None, None] * jump_mass
        c = (lb * kb)[:, None, None] * gb[:, :, None] * tb_mean[:, None, :]
        outer = -(c + c.transpose(1, 2)) + (14.0 * kb)[:, None, None] * tb_mass
        return k[:, None, None] * unit, inner, outer

    kappa = torch.exp(logk)
    parts = [sum_part.detach() for sum_part in blocks(kappa)]
    idx, val = [], []
    for d, K in zip((dof, dof_f, dof_b), parts):
        L = d.shape[1]
        idx.append(torch.stack([d[:, :, None].expand(-1, L, L).reshape(-1), d[:, None, :].expand(-1, L, L).reshape(-1)]))
        val.append(K.reshape(-1))
    A = torch.sparse_coo_tensor(torch.cat(idx, 1), torch.cat(val), (3 * ne, 3 * ne)).coalesce()
    diag = A.values()[A.indices()[0] == A.indices()[1]]
    A = A.to_sparse_csr()
    b = (vol / 3)[:, None].expand(-1, 3).reshape(-1).contiguous()
    u = _cg(A, diag, b)
    lam = _cg(A, diag, u - target)
    lk = logk.clone().requires_grad_(True)
    energy = 0.0
    with torch.enable_grad():
        for d, K in zip((dof, dof_f, dof_b), blocks(torch.exp(lk))):
            energy = energy + torch.einsum("fi,fij,fj->", lam[d], K, u[d])
        energy.backward()
    return {"u": u, "gradient": -lk.grad}


def _exact_batch(case, seed):
    """All problems as one block-diagonal system."""
    at, dofs_all, Ke_all, bnd_all, load_all = 0, [], [], [], []
    for side, k in zip(_sides(case), _batch_kappa(case, seed)):
        n = [side, side]
        if case["kappa"] == "quadrants":
            cx, cy = np.arange(side * side) % side, np.arange(side * side) // side
            k = k[(cx >= side // 2).astype(int) + 2 * (cy >= side // 2).astype(int)]
            k = np.repeat(k, 2) if case["element"] == "p1" else k
        lat, k = _lattice(n), _dev(k)
        if case["element"] == "p1":
            dofs = _dev(_simplices(n))
            Ke, vol = _simplex_stiffness(_dev(lat)[dofs], k)
            load = vol / 3
        else:
            dofs = _dev(_corners(n))
            Ke, det = _cube_stiffness(_dev(np.array([[(0, 0), (1, 0), (0, 1), (1, 1)]]) / side), k)
            load = (det / 4).expand(len(dofs))
        dofs_all.append(dofs + at)
        Ke_all.append(Ke)
        load_all.append(load)
        bnd_all.append(_dev(np.any((lat == 0) | (lat == 1), axis=1)))
        at += len(lat)
    dofs, boundary = torch.cat(dofs_all), torch.cat(bnd_all)
    A, diag = _csr(dofs, torch.cat(Ke_all), at, boundary)
    return {"u": _cg(A, diag, _load(dofs, torch.cat(load_all), at, boundary))}


def _exact_fv(case, seed):
    n, d = _extents(case), len(_extents(case))
    u = _dev(_fv_state(case, seed)).reshape([case["batch"]] + n[::-1])
    burgers, lf, inflow = case["flux"] == "burgers", case["numflux"] == "lf", case["boundary"] == "inflow"

    def flux(v, a):
        return 0.5 * v * v if burgers else FV_VELOCITY[a] * v

    def speed(v):
        return v.abs() if burgers else torch.full_like(v, max(abs(c) for c in FV_VELOCITY[:d]))

    def operator(v):
        out = torch.zeros_like(v)
        for a in range(d):
            ax, k = d - a, n[a]
            if inflow:
                lo, hi = torch.full_like(v.narrow(ax, 0, 1), FV_INFLOW), v.narrow(ax, k - 1, 1)
            else:
                lo, hi = v.narrow(ax, k - 1, 1), v.narrow(ax, 0, 1)
            w = torch.cat([lo, v, hi], ax)
            left, right = w.narrow(ax, 0, k + 1), w.narrow(ax, 1, k + 1)
            if lf:
                g = 0.5 * (flux(left, a) + flux(right, a)) + 0.5 * torch.maximum(speed(left), speed(right)) * (left - right)
            else:
                m = (left + right) / 2
                g = flux(torch.where((m if burgers else torch.full_like(m, FV_VELOCITY[a])) > 0, left, right), a)
            out += (g.narrow(ax, 1, k) - g.narrow(ax, 0, k)) * k
        return out

    dt = _fv_dt(case)
    for _ in range(case["steps"]):
        k0 = operator(u)
        if case["method"] == "euler":
            u = u - dt * k0
        else:
            u = u - 0.5 * dt * (k0 + operator(u - dt * k0))
    return {"u": u.reshape(-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fv":
        return _exact_fv(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "mesh":
        xyz, cells, boundary, kappa = (_dev(a) for a in _mesh(case, seed))
        Ke, vol = _simplex_stiffness(xyz[cells], kappa)
        A, diag = _csr(cells, Ke, len(xyz), boundary)
        b = _load(cells, vol / 4, len(xyz), boundary)
    elif kind == "q2":
        A, diag, b = _exact_q2(case, seed)
    else:
        A, diag, b = _exact_structured(case, seed)
    if kind == "apply":
        x = _dev(_rng(case, seed + 1).standard_normal(len(b)))
        return {"values": A.values(), "rhs": b, "y": A @ x}
    return {"rhs": b, "u": _cg(A, diag, b)}
