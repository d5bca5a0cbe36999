"""A solve whose second copy of the matrix finds no device memory: it runs as the graph of
kernels, which reads the matrix as it is, and the handle goes back to the resident kernel
once there is room.  Every allocation of a first solve fails in turn, by a cudaMalloc
preloaded in a process of its own (tests/host/failing_malloc.c), which also tells what
the subdomain blocks ask for."""

import glob
import json
import os
import subprocess
import sys

import pytest

from host_cpp import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes, json, sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from cases import indexed
from lightfem_gb300 import _native as native, mesh
from lightfem_gb300.solver import upload_model

fake = ctypes.CDLL(sys.argv[2])
fake.fail_allocation.argtypes, fake.allocations_to_go.restype = [ctypes.c_long], ctypes.c_long
precond, precision = sys.argv[3:5]

def prepared():
    ctx = native.Context(0)
    upload_model(ctx, indexed(mesh.cantilever(99, 101, per_element_young=mesh.lognormal_moduli(9999, seed=3))))
    ctx.assemble("coloring")
    ctx.apply_dirichlet()
    return ctx

ctx = prepared()
options = ctx.options(1e-10, 20000, "csr", precond, precision)
want, _ = ctx.solve(options)
ctx.close()
ends = []
while True:
    ctx = prepared()
    before = ctx.timings()["kernel_launches"]
    fake.fail_allocation(len(ends) + 1)
    try:
        u, rep = ctx.solve(options)
        end = dict(code=0, off=float(np.linalg.norm(u - want) / np.linalg.norm(want)),
                   same_bits=bool(np.array_equal(u, want)), converged=int(rep.converged),
                   launches=ctx.timings()["kernel_launches"] - before, iterations=rep.iterations)
    except native.GpuError as err:
        end = dict(code=err.code)
    done = fake.allocations_to_go() > 0
    fake.fail_allocation(0)
    u, _ = ctx.solve(options)
    end["again"] = bool(np.array_equal(u, want))
    ctx.close()
    if done:
        break
    ends.append(end)
print(json.dumps(ends))
"""


MEMORY = r"""
import ctypes, json, sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from cases import indexed
from lightfem_gb300 import _native as native, mesh
from lightfem_gb300.solver import upload_model

fake = ctypes.CDLL(sys.argv[2])
fake.bytes_asked.restype = ctypes.c_long
model = indexed(mesh.cantilever(99, 101, per_element_young=mesh.lognormal_moduli(9999, seed=3)))
owner, _ = native.host_subdomains(model.xy, 64)
size = 2 * np.bincount(owner)
ctx = native.Context(0)
upload_model(ctx, model)
ctx.assemble("coloring")
ctx.apply_dirichlet()
before = fake.bytes_asked()
ctx.solve(ctx.options(1e-10, 20000, "csr", "subdomain"))
print(json.dumps([fake.bytes_asked() - before, int((size * (size + 1) // 2).sum()) * 8]))
"""


@pytest.fixture(scope="module")
def ends_of(native, tmp_path_factory):
    from lightfem_gb300 import build
    out = str(tmp_path_factory.mktemp("no_room"))
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    objects = [os.path.join(build.OUT_DIR, "obj", s + ".o") for s in build.CUDA_SOURCES + build.HOST_SOURCES]
    lib, fake = os.path.join(out, "liblfgpu.so"), os.path.join(out, "failing_malloc.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-cudart", "shared", "-o", lib, *objects, "-Xcompiler",
                    "-fopenmp", "-lgomp", f"-Xlinker=-rpath,{cuda}/lib64"], check=True, capture_output=True)
    cudart = os.path.basename(glob.glob(os.path.join(cuda, "lib64", "libcudart.so.[0-9][0-9]"))[0])
    subprocess.run([os.environ.get("CC", "gcc"), "-shared", "-fPIC", "-O1", f'-DLIBCUDART="{cudart}"',
                    os.path.join(ROOT, "tests", "host", "failing_malloc.c"), "-o", fake, "-ldl"], check=True)

    def run(*args, script=SCRIPT):
        r = subprocess.run([sys.executable, "-c", script, ROOT, fake, *args], capture_output=True,
                           text=True, timeout=300, env={**os.environ, "LD_PRELOAD": fake, "LFGPU_LIBRARY": lib})
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1])

    return run


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_slices(native, ends_of, precision):
    ends = ends_of("jacobi", precision)
    assert all(e["code"] in (0, native.ERR_NOMEM) and e["again"] for e in ends), ends
    graph = [e for e in ends if e["code"] == 0]
    # window, offsets, values, diagonal and the words of the sums, at the least
    assert len(graph) >= 5 and all(e["launches"] > e["iterations"] for e in graph), ends
    # 1e-10 of the residual at both ends: the repository's bar for displacements
    assert all(e["converged"] and e["off"] <= 1e-8 for e in graph), ends


def test_subdomain_factor_is_kept_once(ends_of):
    asked, factor = ends_of(script=MEMORY)
    # the vectors and the split take a quarter of the factor here, not another factor
    assert factor <= asked < 1.5 * factor
