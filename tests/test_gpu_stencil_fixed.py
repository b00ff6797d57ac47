"""The FP64 pressure stencil on integers: its arithmetic on the host against
Python's integers, the operator against extended precision, its fall-back to
FP64 where values do not fit a scale, and the solves that use it."""
import ctypes as C
import pathlib
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "eulersf_gb300" / "csrc"

HARNESS = r"""
#include <cstring>
#include "esf_fixed.cuh"
extern "C" {
void h_from(int n, const double* x, int Ev, int* limbs) {
  for (int i = 0; i < n; i++) {
    esf::Fix f = esf::fixed_from(x[i], Ev);
    limbs[3 * i] = f.l0; limbs[3 * i + 1] = f.l1; limbs[3 * i + 2] = f.l2;
  }
}
void h_mul(int n, const int* v, const double* m, int Em, int* limbs) {
  for (int i = 0; i < n; i++) {
    esf::Fix f = esf::fixed_mul(esf::Fix{v[3 * i], v[3 * i + 1], v[3 * i + 2]}, esf::factor_from(m[i], Em));
    limbs[3 * i] = f.l0; limbs[3 * i + 1] = f.l1; limbs[3 * i + 2] = f.l2;
  }
}
void h_to(int n, const int* v, int E, double* x) {
  for (int i = 0; i < n; i++) x[i] = esf::fixed_to(esf::Fix{v[3 * i], v[3 * i + 1], v[3 * i + 2]}, E);
}
}
"""


def _value(l):
    return int(l[0]) + (int(l[1]) << 27) + (int(l[2]) << 54)


def test_limb_arithmetic(tmp_path):
    src, so = tmp_path / "h.cpp", tmp_path / "h.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC),
                    "-I", "/usr/local/cuda/include", "-o", str(so), str(src)], check=True)
    h = C.CDLL(str(so))
    arr = lambda a: a.ctypes.data_as(C.c_void_p)
    rng = np.random.default_rng(3)
    n = 3000
    for Ev, Em in ((0, 0), (37, -20), (-880, 850), (400, 300)):
        # conversion: truncation at 2^(Ev - 77); exact within 24 bits of the top
        x = rng.choice([-1, 1], n) * np.ldexp(rng.uniform(0.5, 1.0, n), Ev - rng.integers(0, 90, n))
        x[:4] = [0.0, -0.0, np.ldexp(1 - 2.0**-53, Ev), 5e-324]
        limbs = np.zeros((n, 3), np.int32)
        h.h_from(n, arr(x), Ev, arr(limbs))
        back = np.zeros(n)
        h.h_to(n, arr(limbs), Ev, arr(back))
        for a, l, y in zip(x, limbs, back):
            exact = Fraction(float(a)) * Fraction(2) ** (77 - Ev)
            assert _value(l) == int(exact)  # int() truncates
            assert all(abs(int(c)) < 1 << 27 for c in l)
            if abs(a) >= np.ldexp(1.0, Ev - 24):
                assert y == a
        # products of sums of eight: what is dropped is below 9 + 2 units
        # (l0 times the factor's low limb, the factor's shift, the floors)
        v = limbs.reshape(-1, 8, 3)[: n // 8].sum(1).astype(np.int32)
        m = np.ldexp(rng.uniform(0.5, 1.0, len(v)), Em - np.where(rng.random(len(v)) < 0.5, 0, rng.integers(0, 120, len(v))))
        m[::17] = 0.0
        p = np.zeros_like(v)
        h.h_mul(len(v), arr(v), arr(m), Em, arr(p))
        for a, f, l in zip(v, m, p):
            exact = _value(a) * Fraction(float(f)) / Fraction(2) ** Em
            assert abs(_value(l) - exact) <= 11
            assert 0 <= l[0] < 1 << 27 and 0 <= l[1] < 1 << 27
    # rounding to the nearest double, ties to even, over all magnitudes
    v = rng.integers(-2**30, 2**30, (20000, 3)).astype(np.int32)
    v[:, 2] >>= rng.integers(0, 31, len(v))
    v[::5, 2] = 0
    v[::10, 1] = 0
    v[1::10, 2] = -1
    v[:4] = [[1 << 26, 0, 1 << 26], [1 << 26, 0, (1 << 26) + 1], [0, 0, 0], [-1, 0, 0]]
    y = np.zeros(len(v))
    h.h_to(len(v), arr(v), 77, arr(y))
    assert all(float(Fraction(_value(l))) == d for l, d in zip(v, y))


def _apply(minv, v, dtype):
    """J diag(1/m) J^T v in the given precision; 1/m of boundary nodes counts as 0."""
    minv, v = minv.astype(dtype), np.pad(v.astype(dtype), 1)
    w = minv.copy()
    w[[0, -1]] = 0
    w[:, [0, -1]] = 0
    w[:, :, [0, -1]] = 0
    lo, hi = slice(None, -1), slice(1, None)
    corner = [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]
    pick = lambda f, k: f[(lo, hi)[k[0]], (lo, hi)[k[1]], (lo, hi)[k[2]]]
    out = 0
    for axis in range(3):
        jt = 0
        for k in corner:
            jt = jt + (1 - 2 * k[axis]) * pick(v, k)
        jt = jt * w
        for k in corner:
            out = out + (2 * k[axis] - 1) * pick(jt, k)
    return out


def _grid(Z, Y, X):
    import oracle
    g = oracle.grid(X, 0.05)
    g.yRes, g.zRes = Y, Z
    return g


def _gpu_apply(lib, minv, v):
    import torch
    Z, Y, X = minv.shape
    g = _grid(Z, Y, X)
    dm = torch.tensor(minv, dtype=torch.float64, device="cuda")
    dv = torch.tensor(v, dtype=torch.float64, device="cuda")
    out = torch.full_like(dv, 7.0)
    assert lib.esf_pressure_apply(C.byref(g), C.c_void_p(dm.data_ptr()), C.c_void_p(dv.data_ptr()),
                                  C.c_void_p(out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


# node counts z, y, x. The integers start at 8192 cells; warps of 30
# columns and 2 rows, products of larger grids 4; two layers, rows and columns
SHAPES = [(17, 17, 33), (18, 17, 32), (33, 33, 33), (34, 35, 31), (41, 34, 32), (33, 36, 62), (3, 132, 128), (128, 3, 132),
          (132, 128, 3), (70, 95, 97), (151, 90, 47)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["even", "wide"])
def test_operator_against_extended_precision(shape, kind, gpu_lib):
    Z, Y, X = shape
    rng = np.random.default_rng(Z * Y + X)
    v = rng.standard_normal((Z - 1, Y - 1, X - 1))
    minv = rng.uniform(0.5, 2.0, shape)
    minv[rng.random(shape) < 0.05] = 0.0
    if kind == "wide":  # 2^+-60 among neighbours; far beyond the limbs' reach
        v = np.ldexp(v, rng.integers(-60, 61, v.shape))
        minv = np.ldexp(minv, rng.integers(-60, 61, shape))
    got = _gpu_apply(gpu_lib, minv, v)
    ref = _apply(minv, v, np.longdouble)
    # eight nodes, three products each, every product off by at most 11 units
    # and its eight values by one each: 24 x 19 units of
    # 2^-77 2^Ev 2^Em < 2^-75 max|v| max(1/m); and the rounding of the result
    bound = 24 * 19 * 2.0**-75 * np.abs(v).max() * minv.max() + 2.0**-53 * np.abs(ref)
    assert (np.abs(got - ref) <= bound).all()
    plain = _apply(minv, v, np.float64)
    assert np.linalg.norm(got - ref) <= np.linalg.norm(plain - ref) + 1e-300


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["nan", "inf", "minus_inf", "nan_mass", "negative_mass", "huge", "tiny", "tiny_mass", "zero"])
def test_operator_outside_the_scales(what, gpu_lib):
    shape = Z, Y, X = 35, 37, 63
    rng = np.random.default_rng(5)
    v = rng.standard_normal((Z - 1, Y - 1, X - 1))
    minv = rng.uniform(0.5, 2.0, shape)
    cells, nodes = ((3, 4, 5), (20, 30, 33), (33, 35, 61)), ((3, 4, 5), (20, 30, 33))
    for c in cells:
        if what in ("nan", "inf", "minus_inf"):
            v[c] = {"nan": np.nan, "inf": np.inf, "minus_inf": -np.inf}[what]
    for c in nodes:
        if what in ("nan_mass", "negative_mass"):
            minv[c] = np.nan if what == "nan_mass" else -minv[c]
    if what == "huge":
        v = np.ldexp(v, 1000)
    if what == "tiny":
        v = np.ldexp(v, -1060)
    if what == "tiny_mass":
        v, minv = np.ldexp(v, 1010), np.ldexp(minv, -1060)
    if what == "zero":
        v[:] = 0.0
    got = _gpu_apply(gpu_lib, minv, v)
    with np.errstate(invalid="ignore"):
        ref = _apply(minv, v, np.float64)
    assert (np.isnan(got) == np.isnan(ref)).all()
    inf = np.isinf(ref)
    assert (got[inf] == ref[inf]).all()
    ok = np.isfinite(ref)
    # 24 terms of at most 16 max|v| max(1/m) in all orders: 2^-53 per addition;
    # denormal values are multiples of 2^-1074, their products are off by 48 of them
    fin = np.abs(v[np.isfinite(v)])
    top = np.nanmax(minv)
    bound = 32 * 2.0**-53 * 24 * 8 * (fin.max() * top) + 48 * 5e-324
    assert (np.abs(got[ok] - ref[ok]) <= bound).all()


def _solve(lib, fn, g, minv, diag, b, x0, eps, max_it):
    import torch
    t = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda") for a in (minv, diag, b, x0)]
    it, rr = C.c_int(), C.c_double()
    p = [C.c_void_p(a.data_ptr()) for a in t]
    if fn == "static":
        s = lib.esf_pressure_solve_static(C.byref(g), *p, C.c_double(eps), max_it, C.byref(it), C.byref(rr),
                                          None)
    else:
        s = lib.esf_pressure_solve(C.byref(g), *p, C.c_double(eps), max_it, 0, C.byref(it), C.byref(rr), None)
    torch.cuda.synchronize()
    return s, it.value, rr.value, t[3].cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0, 400, -400])
def test_solve_matches_fp64(scale, gpu_lib):
    """The same iteration in FP64 (numpy) for 20 iterations, at three scales of
    b and x: relative to max|x| both are off by rounding amplified by the
    iteration; 1e-11 is 1e5 units of it, the measured size of one FP64
    ordering against another being 1e-13."""
    Z, Y, X = 34, 33, 35
    rng = np.random.default_rng(11)
    minv = rng.uniform(50.0, 300.0, (Z, Y, X))
    w = np.zeros_like(minv)
    w[1:-1, 1:-1, 1:-1] = minv[1:-1, 1:-1, 1:-1]
    diag = sum(3 * w[a:a + Z - 1, b:b + Y - 1, c:c + X - 1] for a in (0, 1) for b in (0, 1) for c in (0, 1))
    x0 = 0.1 * rng.standard_normal(diag.shape)
    b = _apply(minv, rng.standard_normal(diag.shape), np.float64)
    x, r = x0.copy(), (b - _apply(minv, x0, np.float64)) / diag
    d, Ap, beta = np.zeros_like(r), np.zeros_like(r), 0.0
    s = _apply(minv, r, np.float64)
    delta = (r * s).sum()
    for _ in range(20):
        d, Ap = r + beta * d, s + beta * Ap
        alpha = delta / (Ap * Ap / diag).sum()
        x, r = x + alpha * d, r - alpha * Ap / diag
        s = _apply(minv, r, np.float64)
        delta, old = (r * s).sum(), delta
        beta = delta / old
    g = _grid(Z, Y, X)
    f = 2.0 ** scale
    st, it, rr, got = _solve(gpu_lib, "solve", g, minv, diag, b * f, x0 * f, 1e-30, 20)
    assert it == 20
    assert np.abs(got / f - x).max() <= 1e-11 * np.abs(x).max()
    if scale == 0:
        st2, it2, rr2, got2 = _solve(gpu_lib, "static", g, minv, diag, b, x0, 1e-30, 20)
        assert (st2, it2, rr2) == (st, it, rr) and (got2 == got).all()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["b", "x", "minv"])
def test_solve_reports_nan(where, gpu_lib):
    Z, Y, X = 33, 33, 33
    rng = np.random.default_rng(2)
    minv, diag = np.full((Z, Y, X), 2.0), np.full((Z - 1, Y - 1, X - 1), 48.0)
    b, x0 = rng.standard_normal(diag.shape), np.zeros(diag.shape)
    {"b": b, "x": x0, "minv": minv}[where][16, 16, 16] = np.nan
    st, *_ = _solve(gpu_lib, "solve", _grid(Z, Y, X), minv, diag, b, x0, 1e-8, 100)
    assert st != 0
