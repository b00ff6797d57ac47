"""Kernels with more shared memory than a launch has without asking: it is asked
for on the device of each call, not once a process (a counting shim in front of
the CUDA runtime), and a process whose device context is reset goes on with the
same bits."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

_CHILD = textwrap.dedent("""
    import ctypes as C, hashlib, json, sys
    sys.path[:0] = [{root!r}, {tests!r}, {oracle!r}]
    import numpy as np
    import torch  # loads the CUDA runtime for all
    import eulersf_gb300 as E
    from eulersf_gb300 import abi
    from eulersf_gb300.scene import SceneDesc
    from test_zz_no_alloc import _system
    lib = E.load()

    def device(a):
        a = np.ascontiguousarray(a, dtype=np.float64)
        p = C.c_void_p()
        assert lib.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
        assert lib.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
        return p

    def solve(precision):
        g, minv, diag, b, x0 = _system(49, 5)
        p = [device(a) for a in (minv, diag, b, x0)]
        it, rr = C.c_int(), C.c_double()
        st = lib.esf_pressure_solve(C.byref(g), *p, C.c_double(1e-30), 40, precision, C.byref(it), C.byref(rr), None)
        x = np.empty_like(x0)
        lib.cudaMemcpy(x.ctypes.data_as(C.c_void_p), p[3], C.c_size_t(x.nbytes), 2)
        for q in p:
            lib.cudaFree(q)
        return [st, it.value, hashlib.sha256(x.tobytes()).hexdigest()]

    def step():  # (octants of some 2700 columns)
        scene = E.make_scene(SceneDesc(N=128, mass_sample_dh=1 / 256, eps=0.02, max_iters=20, particles_per_cell=2),
                             precision=abi.ESF_MIXED)
        scene.stepImplicit()
        h = [hashlib.sha256(scene.get(n).tobytes()).hexdigest() for n in ("velocity", "solid.velocity")]
        scene.close()
        return h

    def everything():
        out = []
        for call in (lambda: solve(abi.ESF_FP64), lambda: solve(abi.ESF_MIXED), lambda: solve(abi.ESF_MIXED_X64), step):
            try:
                out.append(call())
            except abi.EsfError as e:
                out.append(str(e))
        return out

    first = everything()
    asked = getattr(C.CDLL(None), "esf_test_attribute_calls", None)
    if asked:
        calls = []
        for call in (lambda: solve(abi.ESF_MIXED), lambda: solve(abi.ESF_MIXED_X64), step):
            before = asked()
            call()
            calls.append(asked() - before)
        print(json.dumps(calls))
    else:
        assert lib.cudaDeviceReset() == 0
        print(json.dumps([first, everything()]))
""")

_SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int calls;
int esf_test_attribute_calls(void) { return calls; }
int cudaFuncSetAttribute(const void* f, int what, int value) {
  static int (*real)(const void*, int, int);
  if (!real) *(void**)(&real) = dlsym(RTLD_NEXT, "cudaFuncSetAttribute");
  if (what == 8 && value > 48 * 1024) __atomic_add_fetch(&calls, 1, __ATOMIC_RELAXED);
  return real ? real(f, what, value) : 999;
}
"""


def test_shared_memory_is_asked_for_in_each_call(gpu_lib, tmp_path):
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(_SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O2", "-o", str(shim), str(src), "-ldl"], check=True)
    code = _CHILD.format(root=ROOT, tests=HERE, oracle=os.path.join(ROOT, "oracle"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert r.returncode == 0, r.stderr[-3000:]
    # the loops of a mixed and a double-float solve; the level lists of a step
    assert all(n > 0 for n in json.loads(r.stdout.strip().splitlines()[-1])), r.stdout


def test_calls_after_a_reset(gpu_lib):
    code = _CHILD.format(root=ROOT, tests=HERE, oracle=os.path.join(ROOT, "oracle"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    first, second = json.loads(r.stdout.strip().splitlines()[-1])
    assert all(s[1] == 40 for s in first[:3]) and len(first[3]) == 2, first
    assert second == first
