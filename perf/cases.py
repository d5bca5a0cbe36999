"""The solve path's cases: what a user of this package has it do, through its public entry points.

A case is one of three uses:

* ``whole``: ``LinearElasticSolver.solve`` on a model just built (ordering, pattern, assembly, supports, PCG,
  reactions, element and nodal fields), as a program that analyses one model calls it;
* ``solve``: ``ElasticProblem.solve`` with new element moduli on a mesh that stays (assembly, supports, PCG), the
  forward step of a design or calibration loop;
* ``gradient``: the same and the adjoint solve, through ``torch.autograd``, for a weighted sum of displacements.

Meshes are the package's own workloads at other sizes: the clamped cantilever and the jittered two-material beam
with gravity and pressure, from a few elements to 1000x1000, with log-normal element moduli.  Displacements come back by node ID, whatever the ordering.

Whole analyses stop at the default 1e-10, FP64 solves at the workloads' 1e-8, mixed ones at 3e-10, about what FP64 round-off leaves of the residual on
the larger meshes, so that the refinement runs its whole course and u is settled to nine digits.
"""

from __future__ import annotations

import numpy as np
import torch

from lightfem_gb300 import mesh
from lightfem_gb300.adjoint import ElasticProblem, displacements
from lightfem_gb300.model import PLANE_STRAIN, PLANE_STRESS, SolverSettings
from lightfem_gb300.solver import LinearElasticSolver

WHOLE_TOLERANCE = 1e-10
FP64_TOLERANCE = 1e-8
MIXED_TOLERANCE = 3e-10
EXACT_FLOPS = 9e12  # block elimination beyond this takes too long for a reference value


def _case(name, use, shape, nx, ny, precision, storage, preconditioner, *, plane="stress", order="none",
          assembly="coloring"):
    case = {"use": use, "shape": shape, "nx": nx, "ny": ny, "plane": plane, "order": order, "assembly": assembly,
            "precision": precision, "storage": storage, "preconditioner": preconditioner}
    return dict(case, name=name) if name else case


def listed():
    return [
        # A few elements, as in unit tests, teaching and patch studies: only launches and latency count.
        _case("whole 8x8 fp64", "whole", "cantilever", 8, 8, "fp64", "csr", "jacobi"),
        # A coarse part model, odd sizes, analysed once with all its fields.
        _case("whole 121x59 beam fp64", "whole", "beam", 121, 59, "fp64", "bsr", "block", order="rcm"),
        # Coarse design loops re-solve small meshes many times.
        _case("solve 41x37 mixed", "solve", "cantilever", 41, 37, "mixed", "bsr", "block"),
        # The 200x200 plane-stress workload (the reference's README mesh) in its default storage, both precisions.
        _case("solve 200x200 fp64", "solve", "cantilever", 200, 200, "fp64", "csr", "jacobi"),
        _case("solve 200x200 mixed", "solve", "cantilever", 200, 200, "mixed", "csr", "jacobi"),
        # The two-material beam workload at a third of its size, odd and ragged, RCM, 2x2 blocks.
        _case("solve 351x173 beam fp64", "solve", "beam", 351, 173, "fp64", "bsr", "block", order="rcm"),
        # Middle of the plane-strain range.
        _case("solve 500x500 mixed", "solve", "cantilever", 500, 500, "mixed", "csr", "jacobi", plane="strain",
              order="rcm"),
        _case("solve 640x640 fp64", "solve", "cantilever", 640, 640, "fp64", "bsr", "jacobi", plane="strain",
              order="rcm"),
        # The headline workload: 1000x1000, 2,004,002 unknowns, FP32 inner PCG with FP64 refinement.
        _case("solve 1000x1000 mixed", "solve", "cantilever", 1000, 1000, "mixed", "bsr", "jacobi", plane="strain",
              order="rcm"),
        # Calibration of element moduli: forward and adjoint solve, atomic assembly.
        _case("gradient 150x150 mixed", "gradient", "cantilever", 150, 150, "mixed", "csr", "block",
              assembly="atomic"),
        # The stronger preconditioners: incomplete Cholesky and the reference's default 64-node blocks.
        _case("solve 96x96 ic0 fp64", "solve", "cantilever", 96, 96, "fp64", "csr", "ic0", order="rcm"),
        _case("solve 180x160 subdomain fp64", "solve", "cantilever", 180, 160, "fp64", "csr", "subdomain"),
    ]


def _log_uniform(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    use = rng.choice(["solve"] * 7 + ["whole"] * 2 + ["gradient"] * 2)
    precision = rng.choice(["fp64", "mixed"]) if use != "whole" else "fp64"
    preconditioner = rng.choice(["jacobi"] * 5 + ["block"] * 4 + ["ic0", "subdomain"])
    largest = {"whole": 160, "gradient": 240}.get(use, 1000 if precision == "mixed" else 640)
    if preconditioner == "ic0":
        largest = 96 if use == "solve" else 48
    elif preconditioner == "subdomain":
        largest = 180 if use == "solve" else 110
    nx = _log_uniform(rng, 6, largest)
    ny = max(4, min(largest, int(round(nx * rng.uniform(0.4, 1.0)))))
    return _case(None, use, rng.choice(["cantilever", "beam"]), nx, ny, precision, rng.choice(["csr", "bsr"]),
                 preconditioner, plane=rng.choice(["stress", "strain"]), order=rng.choice(["none", "rcm"]),
                 assembly=rng.choice(["coloring"] * 3 + ["atomic"]))


def _moduli(case, seed):
    return mesh.lognormal_moduli(case["nx"] * case["ny"], seed=seed, scale=70e9, sigma=0.5)


def _model(case, seed):
    tolerance = (WHOLE_TOLERANCE if case["use"] == "whole"
                 else MIXED_TOLERANCE if case["precision"] == "mixed" else FP64_TOLERANCE)
    settings = SolverSettings(
        tolerance=tolerance, max_iterations=200000,
        reordering=case["order"], assembly=case["assembly"], storage=case["storage"], precision=case["precision"],
        preconditioner="block" if case["preconditioner"] == "subdomain" else case["preconditioner"],
        subdomain_nodes=1 if case["preconditioner"] == "block" else 64)
    plane = PLANE_STRAIN if case["plane"] == "strain" else PLANE_STRESS
    young = _moduli(case, seed)
    if case["shape"] == "beam":
        model = mesh.perturbed_beam(case["nx"], case["ny"], seed=seed, plane_mode=plane, per_element_young=young,
                                    settings=settings)
    else:
        model = mesh.cantilever(case["nx"], case["ny"], poisson=0.33, plane_mode=plane, per_element_young=young,
                                settings=settings)
    model.sort_and_index()
    return model


def _weights(case, seed):
    """Weights of the displacement objective, by node ID: a smooth average over the mesh with measurement noise."""
    rng = np.random.default_rng([seed, 7])
    return 1.0 + 0.1 * rng.standard_normal(2 * (case["nx"] + 1) * (case["ny"] + 1))


def prepare(case, seed):
    model = _model(case, seed)
    if case["use"] == "whole":
        # The program's solver stays; the model is new.  RCM renumbers the model in place, so a pass takes a copy.
        return {"use": "whole", "model": model, "solver": LinearElasticSolver(retain_matrix=False)}
    problem = ElasticProblem(model)
    rank = np.argsort(problem.node_ids, kind="stable")  # the place of each node ID in the solve's order
    state = {"use": case["use"], "problem": problem, "rank": None if case["order"] == "none" else rank,
             "young": _moduli(case, seed + 1000003)}
    if case["use"] == "gradient":
        dofs = np.empty(2 * rank.size, np.int64)
        dofs[0::2], dofs[1::2] = 2 * rank, 2 * rank + 1
        state["dofs"] = torch.from_numpy(dofs)
        state["weights"] = torch.from_numpy(_weights(case, seed))
    return state


def _by_node(values, rank):
    return values if rank is None else values.reshape(rank.size, -1)[rank].reshape(-1)


def run(state):
    if state["use"] == "whole":
        model = state["model"].copy()
        result = state["solver"].solve(model)
        rank = np.argsort(model.node_ids, kind="stable")
        return {"u": _by_node(result.displacement, rank), "reaction": _by_node(result.reaction, rank),
                "elements": result.element_results, "nodes": result.node_results[rank]}
    problem = state["problem"]
    if state["use"] == "solve":
        return {"u": _by_node(problem.solve(state["young"]), state["rank"])}
    young = torch.from_numpy(state["young"]).requires_grad_(True)
    u = displacements(young, problem)[state["dofs"]]
    u.mul(state["weights"]).sum().backward()
    return {"u": u.detach(), "gradient": young.grad}


def work(case):
    """Bytes and operations of one pass: PCG iterations a mesh of this size takes, each reading the matrix and the
    iteration's vectors once and writing the three it updates, in the working precision."""
    nodes = (case["nx"] + 1) * (case["ny"] + 1)
    blocks = (3 * case["nx"] + 1) * (3 * case["ny"] + 1)  # 2x2 node blocks of the stiffness matrix
    size = 4 if case["precision"] == "mixed" else 8
    span = max(case["nx"], case["ny"])
    iterations = (7.0 if case["shape"] == "beam" else 12.0) * span
    if case["precision"] == "mixed":
        iterations *= 1.5
    vectors = 8 * 2 * nodes
    flops = 8 * blocks + 14 * 2 * nodes
    entries = 4 * blocks
    if case["preconditioner"] == "ic0":
        iterations *= 0.17
        entries, flops = 2 * entries, 2 * flops
    elif case["preconditioner"] == "subdomain":
        iterations *= 0.4
        entries, flops = entries + 128 * 2 * nodes, flops + 256 * 2 * nodes
    if case["use"] == "gradient":
        iterations *= 2
    return {"bytes": iterations * size * (entries + vectors), "flops": iterations * flops}


# ------------------------------------------------------------------ reference values in 64 bits
GAUSS = 1.0 / 3.0 ** 0.5
CORNERS = ((-1.0, -1.0), (1.0, -1.0), (1.0, 1.0), (-1.0, 1.0))


def _strain_operators(xy, xi, eta):
    """The 3x8 strain matrix and the Jacobian of every element at one point; xy is [E, 4, 2]."""
    dxi = xy.new_tensor([0.25 * a * (1 + b * eta) for a, b in CORNERS])
    deta = xy.new_tensor([0.25 * b * (1 + a * xi) for a, b in CORNERS])
    j = torch.stack([torch.einsum("a,eac->ec", dxi, xy), torch.einsum("a,eac->ec", deta, xy)], 1)  # [E, 2, 2]
    det = j[:, 0, 0] * j[:, 1, 1] - j[:, 0, 1] * j[:, 1, 0]
    dx = (j[:, 1, 1, None] * dxi - j[:, 0, 1, None] * deta) / det[:, None]
    dy = (j[:, 0, 0, None] * deta - j[:, 1, 0, None] * dxi) / det[:, None]
    b = xy.new_zeros(xy.shape[0], 3, 8)
    b[:, 0, 0::2] = dx
    b[:, 1, 1::2] = dy
    b[:, 2, 0::2] = dy
    b[:, 2, 1::2] = dx
    return b, det


def _elasticity(model, young):
    nu, one = torch.as_tensor(model["nu"]).to(young), torch.ones_like(young)
    d = young.new_zeros(young.shape[0], 3, 3)
    if model["strain"]:
        f = young / ((1 + nu) * (1 - 2 * nu))
        d[:, 0, 0] = d[:, 1, 1] = f * (1 - nu)
        d[:, 0, 1] = d[:, 1, 0] = f * nu
        d[:, 2, 2] = f * (1 - 2 * nu) / 2
    else:
        f = young / (1 - nu * nu)
        d[:, 0, 0] = d[:, 1, 1] = f * one
        d[:, 0, 1] = d[:, 1, 0] = f * nu
        d[:, 2, 2] = f * (1 - nu) / 2
    return d


class _Elimination:
    """K = sum of element matrices, eliminated by grid lines (the shorter side): block tridiagonal Cholesky."""

    def __init__(self, nx, ny, nodes, ke, fixed):
        self.lines, self.width, self.by_column = (nx + 1, ny + 1, True) if ny <= nx else (ny + 1, nx + 1, False)
        i, j = nodes % (nx + 1), nodes // (nx + 1)
        line, place = (i, j) if self.by_column else (j, i)
        self.line_of = torch.stack([line, line], -1).reshape(line.shape[0], -1)              # [E, 8]
        self.place_of = torch.stack([2 * place, 2 * place + 1], -1).reshape(line.shape[0], -1)
        self.nx, self.size, self.fixed = nx, 2 * self.width, fixed
        self.ke = ke
        self.first = line.min(1).values
        order = torch.argsort(self.first, stable=True)
        begin = torch.searchsorted(self.first[order], torch.arange(self.lines, device=nodes.device))
        self.sets = [order[begin[k]: begin[k + 1]] for k in range(self.lines - 1)]
        free = ~self._lines(fixed)
        n, new = self.size, ke.new_zeros
        self.l, self.w = [], []
        diag = new(n, n)
        for k in range(self.lines):
            nxt, off = new(n, n), new(n, n)
            if k < self.lines - 1:
                self._add(k, diag, off, nxt)
            keep = free[k].to(ke.dtype)
            d = diag * keep[:, None] * keep[None, :] + torch.diag(1 - keep)
            low = torch.linalg.cholesky(d)
            self.l.append(low)
            if k < self.lines - 1:
                off = off * keep[:, None] * free[k + 1].to(ke.dtype)[None, :]
                w = torch.linalg.solve_triangular(low, off, upper=False)
                self.w.append(w)
                diag = nxt - w.T @ w
        self.free = free

    def _add(self, k, here, off, there):
        e = self.sets[k]
        line, place, n = self.line_of[e], self.place_of[e], self.size
        for target, a, b in ((here, k, k), (off, k, k + 1), (there, k + 1, k + 1)):
            on = (line[:, :, None] == a) & (line[:, None, :] == b)
            flat = (place[:, :, None] * n + place[:, None, :])[on]
            target.view(-1).index_add_(0, flat, self.ke[e][on])

    def _lines(self, v):
        """A vector by node ID, two values a node, as [lines, 2 * width]."""
        grid = v.reshape(-1, self.nx + 1, 2)
        return (grid.transpose(0, 1) if self.by_column else grid).reshape(self.lines, self.size)

    def _flat(self, lines):
        grid = lines.reshape(self.lines, self.width, 2)
        return (grid.transpose(0, 1) if self.by_column else grid).reshape(-1)

    def solve(self, f):
        g = self._lines(f) * self.free
        y = []
        for k in range(self.lines):
            r = g[k] - (self.w[k - 1].T @ y[k - 1] if k else 0.0)
            y.append(torch.linalg.solve_triangular(self.l[k], r[:, None], upper=False)[:, 0])
        x = [None] * self.lines
        for k in reversed(range(self.lines)):
            r = y[k] - (self.w[k] @ x[k + 1] if k < self.lines - 1 else 0.0)
            x[k] = torch.linalg.solve_triangular(self.l[k].T, r[:, None], upper=True)[:, 0]
        return self._flat(torch.stack(x))


def exact(case, seed):
    lines, width = max(case["nx"], case["ny"]) + 1, 2 * (min(case["nx"], case["ny"]) + 1)
    if 3.4 * lines * width ** 3 > EXACT_FLOPS:
        return None
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    m = _model(case, seed)
    as_t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(device)  # noqa: E731
    nodes = as_t(m.element_nodes - 1)
    xy, n_nodes, young = as_t(m.xy), m.xy.shape[0], as_t(m.young)
    if case["use"] != "whole":
        young = as_t(_moduli(case, seed + 1000003))
    info = {"nu": as_t(m.poisson), "strain": case["plane"] == "strain"}
    d, corners, thick = _elasticity(info, young), xy[nodes], as_t(m.thickness)
    points = [_strain_operators(corners, a * GAUSS, b * GAUSS) for a, b in CORNERS]
    ke = sum(torch.einsum("eri,erc,ecj->eij", b, d, b) * (det * thick)[:, None, None] for b, det in points)
    fixed = torch.zeros(n_nodes, 2, dtype=torch.bool, device=device)
    fixed[as_t(m.bc_node - 1)] = True
    f = torch.zeros(n_nodes, 2, dtype=torch.float64, device=device)
    if m.load_node.size:
        f.index_add_(0, as_t(m.load_node - 1), as_t(np.stack([m.load_fx, m.load_fy], 1)))
    if m.body_element.size:  # gravity: the shape functions' integrals, shared by the element's nodes
        force = as_t(np.stack([m.body_bx, m.body_by], 1))
        for (a, b), (_, det) in zip(CORNERS, points):
            shape = xy.new_tensor([0.25 * (1 + p * a * GAUSS) * (1 + q * b * GAUSS) for p, q in CORNERS])
            share = (det * thick)[:, None, None] * shape[None, :, None] * force[:, None, :]
            f.index_add_(0, nodes.reshape(-1), share.reshape(-1, 2))
    if m.edge_element.size:  # pressure on local edge 3 (third to fourth node)
        e = as_t(m.edge_element - 1)
        t = corners[e, 3] - corners[e, 2]
        p = (as_t(m.edge_first) * thick[e])[:, None] * 0.5
        half = torch.stack([-t[:, 1], t[:, 0]], 1) * p
        for a in (2, 3):
            f.index_add_(0, nodes[e, a], half)
    dofs = torch.stack([2 * nodes, 2 * nodes + 1], -1).reshape(-1, 8)
    k = _Elimination(case["nx"], case["ny"], nodes, ke, fixed.reshape(-1))
    product = lambda v: torch.zeros_like(v).index_add_(  # noqa: E731
        0, dofs.reshape(-1), torch.einsum("eij,ej->ei", ke, v[dofs]).reshape(-1))

    def refined(g):
        x = k.solve(g)
        return x + k.solve(g - product(x))

    u = refined(f.reshape(-1))
    if case["use"] == "solve":
        return {"u": u.cpu()}
    if case["use"] == "gradient":
        lam = refined(as_t(_weights(case, seed)))
        grad = -torch.einsum("ei,eij,ej->e", lam[dofs], ke, u[dofs]) / young
        return {"u": u.cpu(), "gradient": grad.cpu()}
    fields, stresses = [], []
    for a, b in ((0.0, 0.0),) + tuple((a * GAUSS, b * GAUSS) for a, b in CORNERS):
        strain = torch.einsum("eri,ei->er", _strain_operators(corners, a, b)[0], u[dofs])
        stress = torch.einsum("erc,ec->er", d, strain)
        mises = _mises(stress)
        fields.append(torch.cat([strain, stress, mises[:, None]], 1))
        stresses.append(stress)
    # Nodal stress: the Gauss-point values extrapolated bilinearly to the corners, averaged over a node's elements.
    total = torch.zeros(n_nodes, 3, dtype=torch.float64, device=device)
    count = torch.zeros(n_nodes, dtype=torch.float64, device=device)
    for c, (p, q) in enumerate(CORNERS):
        value = sum(0.25 * (1 + p * a / GAUSS) * (1 + q * b / GAUSS) * s
                    for (a, b), s in zip(CORNERS, stresses[1:]))
        total.index_add_(0, nodes[:, c], value)
        count.index_add_(0, nodes[:, c], torch.ones_like(young))
    nodal = total / count[:, None]
    return {"u": u.cpu(), "reaction": (product(u) - f.reshape(-1)).cpu(), "elements": torch.stack(fields, 1).cpu(),
            "nodes": torch.cat([nodal, _mises(nodal)[:, None]], 1).cpu()}


def _mises(s):
    return (s[:, 0] ** 2 - s[:, 0] * s[:, 1] + s[:, 1] ** 2 + 3 * s[:, 2] ** 2).clamp(min=0).sqrt()
