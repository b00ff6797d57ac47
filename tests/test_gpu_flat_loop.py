"""Loops of the one-pass iteration with all layers of a block in shared memory
against a launch an iteration of the marching kernel: the same bits, iterations
and residual, on grids of one block to a full wave of blocks, with partly filled
tiles and last chunks of one to four layers."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# cells; x a multiple of 4 as the one-pass iteration wants
CELLS = [(4, 3, 2), (64, 8, 4), (68, 9, 7), (32, 32, 32), (60, 61, 62), (64, 64, 64), (64, 63, 73), (128, 70, 29)]


def _solve(lib, cells, precision, eps, iters):
    import torch
    X, Y, Z = (n + 1 for n in cells)
    rng = np.random.default_rng(X + Y + Z)
    g = oracle.grid(X, 0.05)
    g.yRes, g.zRes = Y, Z
    m = rng.uniform(50.0, 300.0, (Z, Y, X))
    w = np.zeros_like(m)
    w[1:-1, 1:-1, 1:-1] = m[1:-1, 1:-1, 1:-1]
    diag = sum(3 * w[a:a + Z - 1, b:b + Y - 1, c:c + X - 1] for a in (0, 1) for b in (0, 1) for c in (0, 1))
    x0 = 0.1 * rng.standard_normal(diag.shape)
    b = rng.standard_normal(diag.shape)
    t = [torch.tensor(a, dtype=torch.float64, device="cuda") for a in (m, diag, b, x0)]
    it, rr = C.c_int(), C.c_double()
    s = lib.esf_pressure_solve(C.byref(g), *[C.c_void_p(a.data_ptr()) for a in t], C.c_double(eps), iters, precision,
                               C.byref(it), C.byref(rr), None)
    torch.cuda.synchronize()
    return s, it.value, rr.value, t[3].cpu().numpy()


@pytest.mark.parametrize("cells", CELLS)
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("eps,iters", [(1e-30, 75), (1e-6, 2000)])
def test_loop_gives_the_bits_of_single_passes(cells, precision, eps, iters, gpu_lib, monkeypatch):
    loop = _solve(gpu_lib, cells, precision, eps, iters)
    monkeypatch.setenv("ESF_PRESSURE_KERNEL", "pass")
    one = _solve(gpu_lib, cells, precision, eps, iters)
    assert loop[:3] == one[:3]
    assert loop[3].tobytes() == one[3].tobytes()
