"""The resident PCG (Jacobi and 2x2 nodal blocks in one kernel) at the sizes where its
shapes change: a few nodes, slices of 32 nodes with a remainder, the largest mesh of
one cluster and the smallest past it, rows of more than eight off-diagonal blocks, and
node numberings whose rows span the whole mesh.

FP64: iterations within 2 of the oracle's PCG on the same system and displacements
within 1e-8, the repository's bar; the tolerance 1e-11 leaves that margin to the stop
rule.  Mixed: the FP64 residual recomputed after the solve at the target (a factor 1.01
for its own rounding), or the FP64 finish.
"""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.model import Model, SolverSettings
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu

# nodes: 4; 40; 65; 3600 (one FP64 cluster at most) and 3660; 8192 (one mixed cluster
# at most) and 8320
GRIDS = [(1, 1), (3, 9), (4, 12), (59, 59), (59, 60), (127, 63), (127, 64)]


def grid(nx, ny):
    return mesh.cantilever(nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9),
                           settings=SolverSettings(tolerance=1e-11, max_iterations=20000))


def star(sectors):
    """Quads around one node that all of them share: its row has 2 x sectors neighbours."""
    a = 2 * np.pi * np.arange(sectors) / sectors
    mid, tip = np.stack([np.cos(a), np.sin(a)], 1), 1.6 * np.stack([np.cos(a + a[1] / 2), np.sin(a + a[1] / 2)], 1)
    i = np.arange(sectors)
    quads = np.stack([np.ones(sectors, int), 2 + i, 2 + sectors + i, 2 + (i + 1) % sectors], 1)
    n = 1 + 2 * sectors
    return Model(node_ids=np.arange(1, n + 1), xy=np.concatenate([np.zeros((1, 2)), mid, tip]),
                 material_ids=np.array([1]), young=np.array([1e6]), poisson=np.array([0.3]), thickness=np.array([1.0]),
                 element_ids=np.arange(1, sectors + 1), element_nodes=quads, element_material=np.ones(sectors, int),
                 bc_node=np.array([2 + sectors, 3 + sectors]), bc_ux=np.zeros(2), bc_uy=np.zeros(2),
                 load_node=np.array([1, 2 + sectors + sectors // 2]), load_fx=np.array([1.0, 0.0]),
                 load_fy=np.array([0.0, -2.0]), settings=SolverSettings(tolerance=1e-11, max_iterations=1000))


def system(native, model):
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


def check(native, oracle, model, storage, precond):
    ctx = system(native, model)
    s = model.settings
    rp, col, _, _ = ctx.download_pattern()
    kc, fc = ctx.download(native.K_CONSTRAINED), ctx.download(native.F_CONSTRAINED)
    u_ref, rep = oracle.pcg(rp, col, kc, fc, s.tolerance, s.max_iterations, storage, precond)
    assert rep["converged"]
    u, r = ctx.solve(ctx.options(s.tolerance, s.max_iterations, storage, precond))
    assert r.converged and abs(r.iterations - rep["iterations"]) <= 2
    assert np.linalg.norm(u - u_ref) <= 1e-8 * np.linalg.norm(u_ref)
    again, _ = ctx.solve(ctx.options(s.tolerance, s.max_iterations, storage, precond))
    np.testing.assert_array_equal(u, again)
    _, m = ctx.solve(ctx.options(1e-9, s.max_iterations, storage, precond, "mixed"))
    assert m.converged
    assert m.true_residual <= 1.01e-9 * max(1.0, np.linalg.norm(fc)) or m.fallback_fp64
    ctx.close()


@pytest.mark.parametrize("storage,precond", [("csr", "jacobi"), ("bsr", "block")])
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_shapes(native, oracle, nx, ny, storage, precond):
    check(native, oracle, indexed(grid(nx, ny)), storage, precond)


@pytest.mark.parametrize("sectors", [5, 9])
def test_rows_of_several_groups(native, oracle, sectors):
    check(native, oracle, indexed(star(sectors)), "csr", "jacobi")


@pytest.mark.parametrize("nx,ny", [(20, 20), (130, 130)])
def test_any_numbering(native, oracle, nx, ny):
    """Random node order: rows span the mesh; at 130x130 the FP64 window no longer fits
    a CTA and the graph of kernels takes the solve."""
    model = indexed(grid(nx, ny))
    model.index_with_node_order(np.random.default_rng(5).permutation(model.node_ids))
    check(native, oracle, model, "bsr", "jacobi")


def test_iteration_cap(native):
    ctx = system(native, indexed(grid(20, 20)))
    for precision in ("fp64", "mixed"):
        _, r = ctx.solve(ctx.options(1e-11, 7, "csr", "jacobi", precision))
        assert r.iterations == 7 and not r.converged
    ctx.close()


@pytest.mark.parametrize("nx,ny", [(99, 101), (550, 540), (640, 630)])
def test_exchanges_of_z(native, nx, ny):
    """Past one cluster: z in tagged words (10,200 nodes), and published behind a release
    (FP64 from 300,000 nodes, mixed from 400,000).  Both precisions agree to the FP64
    stop rule's own accuracy on these meshes (1e-8, measured residuals of 1e-9)."""
    model = indexed(grid(nx, ny))
    ctx = system(native, model)
    u, r = ctx.solve(ctx.options(1e-9, 50000, "csr", "jacobi"))
    v, m = ctx.solve(ctx.options(1e-9, 50000, "bsr", "block", "mixed"))
    assert r.converged and m.converged
    assert np.linalg.norm(u - v) <= 1e-8 * np.linalg.norm(u)
    ctx.close()
