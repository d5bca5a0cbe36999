"""Distinct handles are independent (include/lfgpu.h): two host threads that solve meshes
of different sizes, whose launches ask for different amounts of shared memory of the same
kernel, get what each gets alone."""

import threading

import numpy as np
import pytest

from cases import indexed
from lightfem_gb300 import mesh
from lightfem_gb300.solver import upload_model

pytestmark = pytest.mark.gpu

# Two sizes each of the resident kernel, one of them past the 48 KB that need no consent,
# and of the sweeps of one CTA; solves a thread.
PAIRS = [("jacobi", "fp64", (99, 101), (300, 300), 1000), ("jacobi", "mixed", (99, 101), (400, 400), 1000),
         ("ic0", "fp64", (20, 20), (90, 90), 400), ("ic0", "mixed", (20, 20), (90, 90), 400)]


def prepared(native, nx, ny):
    ctx = native.Context(0)
    upload_model(ctx, indexed(mesh.cantilever(
        nx, ny, per_element_young=mesh.lognormal_moduli(nx * ny, seed=3, scale=70e9))))
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx


@pytest.mark.parametrize("precond,precision,small,large,solves", PAIRS)
def test_two_threads(native, precond, precision, small, large, solves):
    handles = [prepared(native, *small), prepared(native, *large)]

    def solve(ctx):  # ten iterations: most of the call is its launches
        return ctx.solve(ctx.options(1e-9, 10, "csr", precond, precision))[0]

    alone = [solve(ctx) for ctx in handles]
    failed = []

    def work(ctx, want):
        try:
            for _ in range(solves):
                np.testing.assert_array_equal(solve(ctx), want)
        except Exception as err:
            failed.append(err)

    threads = [threading.Thread(target=work, args=a) for a in zip(handles, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for ctx in handles:
        ctx.close()
