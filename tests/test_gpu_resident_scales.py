"""The resident PCG where a dot product leaves the range of the packed sums: r.z crosses
the smallest normal FP32 total (mixed) or the smallest FP64 scale on its way down, so
that iterations with packed and with FP64 sums alternate on the grid.  The moduli are
scaled by a power of two, which leaves the iteration as it is, and the solve must end
like any other: converged, at its target."""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu

NX, NY = 99, 101  # 10,200 nodes: past one cluster in both precisions


def prepared(native, log2_scale=0):
    model = indexed(mesh.cantilever(NX, NY, per_element_young=mesh.lognormal_moduli(NX * NY, seed=3, scale=70e9)))
    model.young = model.young * 2.0 ** log2_scale
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


# Initial r.z this many powers of two above the limit; at 1e-4 it ends 26 below its start.
@pytest.mark.parametrize("precision,limit,above", [("mixed", -126, 18), ("mixed", -126, 24), ("fp64", -899, 6),
                                                   ("fp64", -899, 12)])
def test_scale_is_lost_and_found(native, precision, limit, above):
    ctx = prepared(native)
    f = ctx.download(native.F_CONSTRAINED)
    z, _ = ctx.apply_preconditioner(f, "jacobi")
    _, plain = ctx.solve(ctx.options(1e-4, 20000, "csr", "jacobi", precision))
    ctx.close()
    ctx = prepared(native, int(np.floor(np.log2(f @ z))) - limit - above)
    _, rep = ctx.solve(ctx.options(1e-4, 20000, "csr", "jacobi", precision))
    assert rep.converged
    assert rep.true_residual <= 1.01e-4 * max(1.0, np.linalg.norm(f))
    if precision == "fp64":
        assert abs(rep.iterations - plain.iterations) <= 2
    ctx.close()
