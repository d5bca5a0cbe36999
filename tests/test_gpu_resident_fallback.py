"""The resident PCG where a sum falls far below the last one, so that its total is formed
in FP64 after all: beside an ordinary mesh stands one element with a load 1e5 times as
large, and r.r falls by more than the packed sums take when that element is solved.  In
each way that the CTAs meet: a cluster, tagged z, published z."""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.model import SolverSettings
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu


def two_bodies(nx, ny, load):
    m = mesh.cantilever(nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9),
                        settings=SolverSettings(tolerance=1e-9, max_iterations=50000))
    n, e = m.n_nodes, m.n_elements
    m.node_ids = np.append(m.node_ids, n + 1 + np.arange(4))
    m.xy = np.vstack([m.xy, np.array([[0, 0], [1, 0], [1, 1], [0, 1]]) * 0.01 + 5.0])
    m.element_ids = np.append(m.element_ids, e + 1)
    m.element_nodes = np.vstack([m.element_nodes, n + 1 + np.arange(4)])
    m.element_material = np.append(m.element_material, 1)
    m.bc_node = np.append(m.bc_node, [n + 1, n + 4])
    m.bc_ux, m.bc_uy = np.append(m.bc_ux, [0.0, 0.0]), np.append(m.bc_uy, [0.0, 0.0])
    m.load_node, m.load_fx = np.append(m.load_node, n + 3), np.append(m.load_fx, 0.0)
    m.load_fy = np.append(m.load_fy, load)
    return indexed(m)


def prepared(native, model):
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


def greatest_fall(native, ctx, iterations=12):
    """Of r.r from one iteration to the next in Jacobi PCG, in powers of two."""
    rp, col, _, _ = ctx.download_pattern()
    k, r = ctx.download(native.K_CONSTRAINED), ctx.download(native.F_CONSTRAINED).copy()
    row = np.repeat(np.arange(ctx.n_dofs), np.diff(rp))
    d = k[col == row]
    z = r / d
    p, rho, rr = z.copy(), r @ z, [r @ r]
    for _ in range(iterations):
        q = np.add.reduceat(k * p[col], rp[:-1])
        r -= rho / (p @ q) * q
        z = r / d
        rho, last = r @ z, rho
        p = z + rho / last * p
        rr.append(r @ r)
    return np.log2(np.max(np.array(rr[:-1]) / np.array(rr[1:])))


# nodes: one cluster in both precisions; tagged in both; published in FP64; in both
@pytest.mark.parametrize("nx,ny,precisions", [(41, 37, ("fp64", "mixed")), (99, 101, ("fp64", "mixed")),
                                              (550, 548, ("fp64",)), (640, 630, ("mixed",))])
def test_steep_fall(native, nx, ny, precisions):
    alone = prepared(native, indexed(two_bodies(nx, ny, 0.0)))
    want, _ = alone.solve(alone.options(1e-9, 50000, "csr", "jacobi"))
    fnorm = np.linalg.norm(alone.download(native.F_CONSTRAINED))
    alone.close()
    ctx = prepared(native, two_bodies(nx, ny, -1e5 * fnorm))
    assert greatest_fall(native, ctx) > 12  # the packed sums take ten
    f = ctx.download(native.F_CONSTRAINED)
    for precision in precisions:
        u, rep = ctx.solve(ctx.options(1e-9 * fnorm / np.linalg.norm(f), 50000, "csr", "jacobi", precision))
        assert rep.converged
        assert np.linalg.norm(u[:-8] - want[:-8]) <= 1e-8 * np.linalg.norm(want[:-8])
    ctx.close()
