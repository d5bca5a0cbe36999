"""The pipelined IC(0) level sweeps (one CTA, narrow levels) against the polled sweeps:
the same application bit for bit, at meshes whose widest level is one row, a warp and
its neighbours, and the widest the pipeline takes; the mixed loop reaches the FP64
target with them."""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.model import SolverSettings
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu


def check(native, nx, ny, order, fp64_solve):
    model = indexed(mesh.cantilever(nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9),
                                    settings=SolverSettings(tolerance=1e-9, max_iterations=5000)))
    if order == "rcm":
        model.index_with_node_order(native.host_rcm(model.node_ids, model.element_nodes))
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    r = np.random.default_rng(1).standard_normal(ctx.n_dofs)
    z, _ = ctx.apply_preconditioner(r, "ic0")
    ctx.set_option(native.OPTION_IC0_SWEEP, native.IC0_SWEEP["polled"])
    want, _ = ctx.apply_preconditioner(r, "ic0")
    np.testing.assert_array_equal(z, want)
    if fp64_solve:
        u_want, r_want = ctx.solve(ctx.options(1e-9, 5000, "csr", "ic0"))
    ctx.set_option(native.OPTION_IC0_SWEEP, native.IC0_SWEEP["auto"])
    if fp64_solve:
        u, rep = ctx.solve(ctx.options(1e-9, 5000, "csr", "ic0"))
        assert rep.iterations == r_want.iterations
        np.testing.assert_array_equal(u, u_want)
    f = ctx.download(native.F_CONSTRAINED)
    _, m = ctx.solve(ctx.options(1e-8, 20000, "bsr", "ic0", "mixed"))
    assert m.converged and (m.true_residual <= 1.01e-8 * max(1.0, np.linalg.norm(f)) or m.fallback_fp64)
    ctx.close()


@pytest.mark.parametrize("order", ["none", "rcm"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 30), (7, 3), (60, 33), (64, 66), (130, 125), (240, 255)])
def test_same_as_polled(native, nx, ny, order):
    check(native, nx, ny, order, True)


# By rows of nodes the widest levels hold 161, 256 (the widest taken) and 257 rows.
@pytest.mark.parametrize("nx,ny", [(318, 160), (510, 255), (512, 256)])
def test_wide_levels(native, nx, ny):
    check(native, nx, ny, "none", False)
