"""Which kernels a solve runs, told by the launches it counts (a resident solve: its setup
and one kernel; the graph of kernels: two or three an iteration), on both sides of each
line, and the fallback's own paths on a mesh that the resident kernel refuses."""

import numpy as np
import pytest

from cases import by_id_order, indexed
from lightfem_gb300 import mesh
from lightfem_gb300.model import SolverSettings
from lightfem_gb300.solver import upload_model
from test_gpu_waits import SHORT_NS, _expect_timeout, _solves_grid6_after

pytestmark = pytest.mark.gpu


def model_of(nx, ny, order="none", native=None):
    m = indexed(mesh.cantilever(nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9),
                                settings=SolverSettings(tolerance=1e-10, max_iterations=50000)))
    if order == "random":
        m.index_with_node_order(np.random.default_rng(5).permutation(m.node_ids))
    elif order == "rcm":
        m.index_with_node_order(native.host_rcm(m.node_ids, m.element_nodes))
    return m


def prepared(native, model):
    ctx = native.Context(0)
    upload_model(ctx, model)
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


def launches(ctx, call):
    before = ctx.timings()["kernel_launches"]
    result = call()
    return ctx.timings()["kernel_launches"] - before, result


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (59, 59), (59, 60), (127, 63), (127, 64), (300, 200)])
def test_resident(native, nx, ny, precision):
    ctx = prepared(native, model_of(nx, ny))
    options = ctx.options(1e-9, 50000, "csr", "jacobi", precision)
    ctx.solve(options)
    n, (_, rep) = launches(ctx, lambda: ctx.solve(options))
    assert rep.converged and n <= 10
    ctx.close()


# Rows that span more nodes than 16 bits count, and than an FP64 window holds
@pytest.mark.parametrize("nx,ny,precision", [(400, 400, "fp64"), (400, 400, "mixed"), (130, 130, "fp64")])
def test_graph(native, nx, ny, precision):
    ctx = prepared(native, model_of(nx, ny, "random"))
    n, (_, rep) = launches(ctx, lambda: ctx.solve(ctx.options(1e-3, 50000, "csr", "jacobi", precision)))
    assert rep.converged and n > rep.iterations
    ctx.close()


# An application by polls launches two kernels, by levels three; AUTO leaves levels of fewer
# than 192 rows on average to the sweeps of one CTA or to polls.
@pytest.mark.parametrize("nx,ny,order,kernels", [(1, 30, "none", 3), (60, 33, "rcm", 3), (240, 255, "rcm", 3),
                                                 (510, 255, "none", 3)])
def test_ic0_sweeps(native, nx, ny, order, kernels):
    ctx = prepared(native, model_of(nx, ny, order, native))
    r = np.random.default_rng(1).standard_normal(ctx.n_dofs)
    ctx.apply_preconditioner(r, "ic0")
    assert launches(ctx, lambda: ctx.apply_preconditioner(r, "ic0"))[0] == kernels
    _, rep = ctx.solve(ctx.options(1e-9, 3, "csr", "ic0"))
    assert ctx.n_dofs < 192 * rep.ic0_levels
    ctx.set_option(native.OPTION_IC0_SWEEP, native.IC0_SWEEP["polled"])
    assert launches(ctx, lambda: ctx.apply_preconditioner(r, "ic0"))[0] == 2
    ctx.close()


# The mixed loop's direct form: 150,000 nodes and more where the resident kernel does not go.
@pytest.mark.parametrize("storage,precond", [("csr", "jacobi"), ("bsr", "block")])
def test_direct_form_solves(native, storage, precond):
    model = model_of(400, 400, "random")
    ctx = prepared(native, model)
    n, (u, rep) = launches(ctx, lambda: ctx.solve(ctx.options(1e-9, 50000, storage, precond, "mixed")))
    f = ctx.download(native.F_CONSTRAINED)
    assert rep.converged and n > rep.iterations
    assert rep.true_residual <= 1.01e-9 * max(1.0, np.linalg.norm(f)) or rep.fallback_fp64
    ctx.close()
    plain = model_of(400, 400)
    ctx = prepared(native, plain)
    v, _ = ctx.solve(ctx.options(1e-9, 50000, storage, precond))
    ctx.close()
    a, b = by_id_order(model, u), by_id_order(plain, v)
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)


def test_direct_form_wait_expires(native, golden_json):
    ctx = prepared(native, model_of(400, 400, "random"))
    ctx.set_option(native.OPTION_WAIT_LIMIT_NS, SHORT_NS)
    assert _expect_timeout(native, ctx, ctx.options(1e-8, 10000, "bsr", "jacobi", "mixed")) >= 0
    _solves_grid6_after(native, ctx, golden_json)
    ctx.close()


@pytest.mark.parametrize("precond", ["jacobi", "block"])
def test_direct_form_indefinite(native, precond):
    model = model_of(400, 400, "random")
    model.young[80200] *= -10.0  # one element's modulus
    ctx = prepared(native, model)
    with pytest.raises(native.GpuError) as err:
        ctx.solve(ctx.options(1e-8, 200000, "bsr", precond, "mixed"), download=False)
    assert err.value.code in (native.ERR_NOT_SPD, native.ERR_RHO), str(err.value)
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tagged_wait_expires(native, golden_json, precision):
    """The resident kernel past one cluster: its waits for the sums and for the other CTAs'
    tagged z.  (The cluster's waits are not made to run out: a CTA that gave up no longer
    knows which of its peers' stores into its shared memory are on their way.)"""
    ctx = prepared(native, model_of(300, 200))
    ctx.set_option(native.OPTION_WAIT_LIMIT_NS, SHORT_NS)
    assert _expect_timeout(native, ctx, ctx.options(1e-8, 10000, "bsr", "jacobi", precision)) >= 0
    _solves_grid6_after(native, ctx, golden_json)
    ctx.close()
