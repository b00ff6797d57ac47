"""Calls that find the device's memory out give back the kept workspaces and go
on. A shim in front of the CUDA runtime refuses device memory, from a chosen
allocation of a call on, until a kept workspace has been freed."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

# (a growing buffer frees itself first: five frees are a workspace)
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static long skip = -1, frees, refused;
void esf_test_refuse_after(long n) { skip = n; frees = refused = 0; }
long esf_test_refused(void) { skip = -1; return refused; }
int cudaMalloc(void** p, size_t n) {
  static int (*real)(void**, size_t);
  if (!real) *(void**)(&real) = dlsym(RTLD_NEXT, "cudaMalloc");
  if (skip == 0) {
    refused++;
    return 2; /* cudaErrorMemoryAllocation */
  }
  if (skip > 0) skip--;
  return real ? real(p, n) : 999;
}
int cudaFree(void* p) {
  static int (*real)(void*);
  if (!real) *(void**)(&real) = dlsym(RTLD_NEXT, "cudaFree");
  if (skip == 0 && p && ++frees >= 5) skip = -1;
  return real ? real(p) : 999;
}
"""

_CHILD = textwrap.dedent("""
    import ctypes as C, json, sys
    sys.path[:0] = [{root!r}, {tests!r}, {oracle!r}]
    import numpy as np
    import torch
    import eulersf_gb300 as E
    from eulersf_gb300 import abi
    from eulersf_gb300.bake import rasterize_solid
    from eulersf_gb300.scene import SceneDesc, icosphere
    from test_zz_no_alloc import _system, _dev, _ptr
    shim = C.CDLL(None)
    lib = E.load()
    systems = {{X: _system(X, X) for X in (21, 25, 33)}}
    systems = {{X: (s[0], [_dev(a) for a in s[1:]]) for X, s in systems.items()}}
    torch.cuda.synchronize()

    def solve(X, precision):
        g, t = systems[X]
        it, rr = C.c_int(), C.c_double()
        return lib.esf_pressure_solve(C.byref(g), *[_ptr(a) for a in t], C.c_double(1e-30), 5, precision, C.byref(it),
                                      C.byref(rr), None)

    batch_x = [systems[33][1][3].clone() for _ in range(2)]
    torch.cuda.synchronize()

    def batch():
        n, x = 2, batch_x
        g, t = systems[33]
        arr = [(C.c_void_p * n)(*[a.data_ptr() for a in v]) for v in ([t[0]] * n, [t[1]] * n, [t[2]] * n, x)]
        return lib.esf_pressure_solve_batch(n, (abi.Grid * n)(g, g), *arr, C.c_double(1e-30), 5, abi.ESF_MIXED, 1, None,
                                            None, None, None)

    desc = SceneDesc(N=24, mass_sample_dh=1 / 96, eps=1e-2, max_iters=50)

    def scene_of(precision):
        return E.make_scene(desc, precision=precision)

    def bake():
        verts, faces = icosphere(2, 0.1)
        rasterize_solid(verts, faces, 0.1 / 50, 1000.0)

    def case(call, skip, before=None):
        lib.esf_release_workspaces()
        state = before() if before else None
        solve(21, abi.ESF_MIXED)  # kept until memory runs out
        shim.esf_test_refuse_after(skip)
        try:
            status = call(state) if before else call()
        except abi.EsfError as e:
            status = e.status
        return [int(status or 0), shim.esf_test_refused()]

    def step(s):
        try:
            s.stepImplicit()
        finally:
            s.close()

    out = {{}}
    for skip in (0, 4, 9, 10, 11):
        out["solve fp64 " + str(skip)] = case(lambda: solve(33, abi.ESF_FP64), skip)
    out["solve mixed"] = case(lambda: solve(33, abi.ESF_MIXED), 12)
    for skip in (0, 1):  # on a kept workspace of the mixed solve
        out["solve x64 " + str(skip)] = case(lambda _: solve(25, abi.ESF_MIXED_X64), skip, lambda: solve(25, abi.ESF_MIXED))
    for skip in (0, 3):
        out["batch " + str(skip)] = case(batch, skip)
    for precision in (abi.ESF_FP64, abi.ESF_MIXED):
        out["create " + str(precision)] = case(lambda: scene_of(precision).close(), 40)
        for skip in (0, 2, 5, 9, 14, 20):
            out["step " + str(precision) + " " + str(skip)] = case(step, skip, lambda: scene_of(precision))
    for skip in (0, 1, 2):
        out["bake " + str(skip)] = case(bake, skip)
    print(json.dumps(out))
""")


def child(code, tmp_path, **names):
    """The last line that `code` prints, run with the shim."""
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O2", "-o", str(shim), str(src), "-ldl"], check=True)
    code = code.format(root=ROOT, tests=HERE, oracle=os.path.join(ROOT, "oracle"), **names)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_kept_workspaces_are_given_back(gpu_lib, tmp_path):
    out = child(_CHILD, tmp_path)
    bad = {k: v for k, v in out.items() if v[0] not in (0, 6)}  # ESF_OK, or not converged in the iterations given
    assert not bad, bad
    # the refusal was met: in every solve, batch and bake, and in steps' first buffers
    for k, (_, refused) in out.items():
        if k.split()[0] in ("solve", "batch", "bake", "create") or k.endswith(" 0"):
            assert refused > 0, k


_BAKE = textwrap.dedent("""
    import ctypes as C, json, sys
    sys.path[:0] = [{root!r}]
    import numpy as np
    import torch
    import eulersf_gb300 as E
    from eulersf_gb300 import abi
    from eulersf_gb300.bake import rasterize_solid
    from eulersf_gb300.scene import icosphere
    shim = C.CDLL(None)
    lib = E.load()
    verts, faces = icosphere(3, 0.1)
    grid = rasterize_solid(verts, faces, 0.1 / 40, 1000.0)
    assert np.prod(grid[0]) * len(faces) >= 2e8  # by cubes
    lib.esf_release_workspaces()
    shim.esf_test_refuse_after(3)
    try:
        again = rasterize_solid(verts, faces, 0.1 / 40, 1000.0)
        print(json.dumps([shim.esf_test_refused(), bool(np.array_equal(grid[3], again[3]) and grid[4] == again[4])]))
    except abi.EsfError as e:
        print(json.dumps([shim.esf_test_refused(), str(e)]))
""")


def test_baking_without_memory_for_cubes(gpu_lib, tmp_path):
    """The cubes' lists refused, and nothing kept to give back: every node
    against every triangle, the same masses."""
    assert child(_BAKE, tmp_path) == [1, True]
