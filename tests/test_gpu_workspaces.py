"""The solver seam's kept workspaces: a call on a used workspace gives the bits
of a call on a new one, whatever the calls before it were, from several threads
and streams; they are bounded and given back."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
FP64, MIXED, X64 = 0, 1, 2


def _dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


class System:
    def __init__(self, shape, seed, nan=False):
        X, Y, Z = shape
        rng = np.random.default_rng(seed)
        self.g = oracle.grid(X, 0.05)
        self.g.yRes, self.g.zRes = Y, Z
        m = rng.uniform(50.0, 300.0, (Z, Y, X))
        w = np.zeros_like(m)
        w[1:-1, 1:-1, 1:-1] = m[1:-1, 1:-1, 1:-1]
        diag = sum(3 * w[a:a + Z - 1, b:b + Y - 1, c:c + X - 1] for a in (0, 1) for b in (0, 1) for c in (0, 1))
        b = rng.standard_normal(diag.shape)
        if nan:
            b[1, 2, 3] = np.nan
        self.t = [_dev(a) for a in (m, diag, b, 0.1 * rng.standard_normal(diag.shape))]

    def solve(self, lib, precision, stream=None, iters=40):
        import torch
        # (no device-wide synchronisation: another thread may be capturing a graph)
        stream = stream or torch.cuda.current_stream()
        with torch.cuda.stream(stream):
            x = self.t[3].clone()
            it, rr = C.c_int(), C.c_double()
            p = [C.c_void_p(a.data_ptr()) for a in (*self.t[:3], x)]
            s = lib.esf_pressure_solve(C.byref(self.g), *p, C.c_double(1e-30), iters, precision, C.byref(it),
                                       C.byref(rr), C.c_void_p(stream.cuda_stream))
            return s, it.value, repr(rr.value), x.cpu().numpy().tobytes()


SHAPES = [(25, 21, 18), (33, 33, 33), (132, 127, 130)]  # the last: FP64 without a graph


@pytest.mark.parametrize("precision", [FP64, MIXED, X64])
def test_used_workspace_gives_the_same_bits(precision, gpu_lib):
    systems = [System(s, 3 + k) for s in SHAPES for k in (0, 1)]
    bad = [System(s, 9, nan=True) for s in SHAPES]
    new = []
    for s in systems:
        gpu_lib.esf_release_workspaces()
        new.append(s.solve(gpu_lib, precision))
    for _ in range(2):
        for s, ref in zip(systems, new):
            assert s.solve(gpu_lib, precision) == ref
        for s in bad:  # leaves NaN in its workspace
            assert s.solve(gpu_lib, precision)[0] != 0
        for s in reversed(systems):
            s.solve(gpu_lib, MIXED if precision == X64 else X64, iters=7)


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_threads_and_streams(precision, gpu_lib):
    import torch
    systems = [System(SHAPES[k % 2], 20 + k) for k in range(6)]
    ref = [s.solve(gpu_lib, precision) for s in systems]
    torch.cuda.synchronize()
    out = {}

    def work(k):
        stream = torch.cuda.Stream()
        out[k] = [systems[(k + j) % 6].solve(gpu_lib, precision, stream) for j in range(6)]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        assert out[k] == [ref[(k + j) % 6] for j in range(6)]


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_batch_on_used_workspaces(precision, gpu_lib):
    import torch
    systems = [System(SHAPES[0] if k % 3 else SHAPES[1], 40 + k) for k in range(9)]
    ref = [s.solve(gpu_lib, precision)[3] for s in systems]
    n = len(systems)
    grids = (type(systems[0].g) * n)(*[s.g for s in systems])
    for _ in range(3):
        xs = [s.t[3].clone() for s in systems]
        torch.cuda.synchronize()
        arr = [(C.c_void_p * n)(*[a.data_ptr() for a in v])
               for v in ([s.t[0] for s in systems], [s.t[1] for s in systems], [s.t[2] for s in systems], xs)]
        assert gpu_lib.esf_pressure_solve_batch(n, grids, *arr, C.c_double(1e-30), 40, precision, 0, None, None,
                                                None, None) == 0
        torch.cuda.synchronize()
        assert [x.cpu().numpy().tobytes() for x in xs] == ref


def test_bounded_and_given_back(gpu_lib):
    import torch
    gpu_lib.esf_release_workspaces()
    torch.cuda.synchronize()
    free0, total = torch.cuda.mem_get_info()
    # 24 shapes of about 140 MB each, 3.4 GB together
    for k in range(24):
        System((113, 113, 110 + k), 1).solve(gpu_lib, MIXED, iters=1)
    torch.cuda.empty_cache()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= total // 128 + (256 << 20)  # and the allocator's and torch's own few
    gpu_lib.esf_release_workspaces()
    torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20
