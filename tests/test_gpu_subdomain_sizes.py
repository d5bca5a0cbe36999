"""The FP64 subdomain application at block sizes around a group of unknowns, a warp of
rows and the largest block, equal blocks and uneven ones in one launch, against the
oracle bit for bit."""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,nodes", [("chunk", 3), ("chunk", 4), ("chunk", 5), ("chunk", 15), ("chunk", 16),
                                         ("chunk", 17), ("chunk", 33), ("chunk", 127), ("chunk", 512), ("rcb", 40)])
def test_application(native, oracle, split, nodes):
    nx, ny = 30, 36
    model = indexed(mesh.cantilever(nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9)))
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    ctx.set_subdomains(nodes, split)
    rp, col, _, _ = ctx.download_pattern()
    r = np.random.default_rng(nodes).standard_normal(ctx.n_dofs)
    z, _ = ctx.apply_preconditioner(r, "subdomain")
    want, _ = oracle.precond_apply(rp, col, ctx.download(native.K_CONSTRAINED), r, "block", split, nodes, model.xy)
    np.testing.assert_array_equal(z, want)
    ctx.close()
