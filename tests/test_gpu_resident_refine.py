"""Residual replacements of the resident mixed solve: f - K x in FP64 from the x that all
CTAs of a cluster (meshes up to 8,192 nodes) just wrote."""

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def prepared(native, nx, ny):
    ctx = native.Context(0)
    upload_model(ctx, indexed(mesh.cantilever(
        nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9))))
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


def residual_rounding(native, ctx, u):
    """What ||f - K u|| may be off by: a row's terms, each rounded, and their sum."""
    rp, col, _, _ = ctx.download_pattern()
    k, f = ctx.download(native.K_CONSTRAINED), ctx.download(native.F_CONSTRAINED)
    terms = np.add.reduceat(np.abs(k) * np.abs(u[col]), rp[:-1]) + np.abs(f)
    return np.linalg.norm(terms * (np.diff(rp) + 2) * EPS)


# 2, 4, 16 and 16 CTAs in a cluster
@pytest.mark.parametrize("nx,ny", [(15, 12), (25, 17), (41, 37), (126, 63)])
def test_replaced_residual_is_that_of_x(native, nx, ny):
    ctx = prepared(native, nx, ny)
    options = ctx.options(1e-9, 50000, "csr", "jacobi", "mixed", inner_reduction=0.5)
    u, rep = ctx.solve(options)
    assert rep.converged and not rep.fallback_fp64 and rep.refinements >= 20
    # Both sides round, and the norm's own sum adds less than another bound's worth.
    assert abs(rep.final_residual - rep.true_residual) <= 3 * residual_rounding(native, ctx, u)
    for _ in range(20):
        again, r = ctx.solve(options)
        assert (r.iterations, r.refinements) == (rep.iterations, rep.refinements)
        np.testing.assert_array_equal(again, u)
    ctx.close()


def summed(native, ctx, u, sums):
    """||f - K u|| with a row's fused multiply-adds dealt to ``sums`` sums by their place."""
    rp, col, _, _ = ctx.download_pattern()
    k, f = ctx.download(native.K_CONSTRAINED), ctx.download(native.F_CONSTRAINED)
    s = np.zeros((sums, ctx.n_dofs))
    for e in range(np.diff(rp).max()):
        live = np.diff(rp) > e
        at = rp[:-1][live] + e
        s[e % sums, live] = (np.longdouble(k[at]) * u[col[at]] + s[e % sums, live]).astype(np.float64)
    return np.linalg.norm(f - (s[0] if sums == 1 else (s[0] + s[1]) + (s[2] + s[3])))


# A cluster, and a grid whose threads have 64 registers
@pytest.mark.parametrize("nx,ny,replacements", [(41, 37, range(11, 16)), (350, 350, (9, 11))])
def test_residual_is_formed_in_four_sums(native, nx, ny, replacements):
    """A replaced residual is that of the CSR product's four sums a row, and not that of
    one sum, whose rounding is larger by up to a factor of two: it bounds what a mixed solve
    can reach."""
    ctx = native.Context(0)
    upload_model(ctx, indexed(mesh.cantilever(
        nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=1, scale=70e9, sigma=2.0))))
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    # The extended product rounds as an FMA does but for double rounding where long double
    # has fewer than 106 bits.
    tolerance = 1e-9 if np.finfo(np.longdouble).nmant >= 105 else 0.02
    told = []
    for precond in ("jacobi", "block"):
        for count in replacements:
            u, rep = ctx.solve(ctx.options(1e-15, 20000, "csr", precond, "mixed", max_refinements=count))
            four, one = summed(native, ctx, u, 4), summed(native, ctx, u, 1)
            told.append(abs(one - four) / four)
            assert abs(rep.final_residual - four) <= tolerance * four
    assert max(told) > 2 * tolerance  # the two can be told apart here
    ctx.close()
