"""The FP64 pressure stencil on integers where the values around one cell lie
far below those around another: each cell as near to the exact value as FP64
brings it, in products and in solves; solves that FP64 takes from the start, and
factors near the exponent range's ends."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_stencil_fixed import _apply, _gpu_apply, _grid, _solve

pytestmark = pytest.mark.gpu
U = 2.0**-53
CORNERS = [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]


def _around(f, k):
    ends = (slice(None, -1), slice(1, None))
    return f[ends[k[0]], ends[k[1]], ends[k[2]]]


def _inner(minv):
    w = minv.copy()
    w[[0, -1]] = 0
    w[:, [0, -1]] = 0
    w[:, :, [0, -1]] = 0
    return w


def _diag(minv):
    return sum(3 * _around(_inner(minv), k) for k in CORNERS)


def _terms(minv, v):
    """A cell's terms without their signs, summed."""
    p = np.abs(np.pad(v, 1))
    n = sum(_around(p, k) for k in CORNERS) * np.abs(_inner(minv))
    return 3 * sum(_around(n, k) for k in CORNERS)


def _fall(shape, axis, per):
    """2^-(per i) along an axis."""
    f = np.ldexp(1.0, -(per * np.arange(shape[axis])).astype(int))
    return f.reshape([-1 if a == axis else 1 for a in range(3)])


def _system(kind, shape):
    """Node factors and values of a kind on `shape` nodes."""
    Z, Y, X = shape
    rng = np.random.default_rng(Z + Y + X)
    cells = (Z - 1, Y - 1, X - 1)
    v, minv = rng.standard_normal(cells), rng.uniform(0.5, 2.0, shape)
    what, *arg = kind.split()
    if what == "fall":  # of the values, along an axis
        v *= _fall(cells, int(arg[0]), float(arg[1]))
    if what == "heavy":  # a ball of small 1/m
        at = np.stack(np.meshgrid(*[np.arange(n) / n - 0.5 for n in shape], indexing="ij"))
        minv = np.where((at ** 2).sum(0) < 0.1, minv / float(arg[0]), minv)
    if what == "light":  # one node
        minv[Z // 2, Y // 2, X // 2] = float(arg[0])
    if what == "source":  # a few cells, tiny values around, zeros elsewhere
        v[:] = 0.0
        v[Z // 2 - 6:Z // 2 + 6, Y // 2 - 6:Y // 2 + 6, X // 2 - 6:X // 2 + 6] = 1e-12
        v[Z // 2, Y // 2, X // 2] = 1.0
    if what == "both":  # values and factors fall along different axes
        v *= _fall(cells, 0, 1.0)
        minv *= _fall(shape, 2, 1.0)
    return minv, v


KINDS = ["fall 0 2", "fall 1 1.5", "fall 2 3", "heavy 1e9", "heavy 1e12", "heavy 1e15", "light 1e15", "source", "both"]
# node counts z, y, x: two rows a warp and four, odd sides
SHAPES = [(33, 33, 33), (41, 34, 63), (132, 128, 30), (97, 95, 92)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_product_in_each_cell(kind, shape, gpu_lib):
    minv, v = _system(kind, shape)
    got = _gpu_apply(gpu_lib, minv, v)
    ref = _apply(minv, v, np.longdouble)
    terms = _terms(minv, v)
    zero = terms == 0
    assert (got[zero] == 0).all()
    err = np.zeros_like(v)
    err[~zero] = (np.abs(got - ref)[~zero] / terms[~zero]).astype(np.float64)
    # FP64: at most nine roundings in a row, each U of its partial sum at most.
    # Integers: 24 x 19 units of 2^-77 2^Ev 2^Em, the terms' sum at least three
    # times a product 2^-(21 + 2) below 2^Ev 2^Em
    assert err.max() <= max(10 * U, 24 * 19 * 2.0**-77 * 2.0**23 / 3 + U)
    # in the mean square nine roundings are 3 U / sqrt(3); by layers, rows and
    # columns of cells, so that the small ones stand for themselves
    for axes in ((1, 2), (0, 2), (0, 1)):
        n = np.maximum((~zero).sum(axes), 1)
        assert np.sqrt((err ** 2).sum(axes) / n).max() <= 2 * U


def _reference(minv, diag, b, x, iters):
    """The conjugate residual iteration in extended precision."""
    L = np.longdouble
    diag, b, x = diag.astype(L), b.astype(L), x.astype(L)
    r = (b - _apply(minv, x, L)) / diag
    d, Ap, beta = np.zeros_like(r), np.zeros_like(r), L(0)
    s = _apply(minv, r, L)
    delta = (r * s).sum()
    for _ in range(iters):
        d, Ap = r + beta * d, s + beta * Ap
        alpha = delta / (Ap * Ap / diag).sum()
        x, r = x + alpha * d, r - alpha * Ap / diag
        s = _apply(minv, r, L)
        delta, old = (r * s).sum(), delta
        beta = delta / old
    return x


@pytest.mark.parametrize("kind", ["fall 0 2", "fall 1 1.5", "fall 2 3", "heavy 1e9", "heavy 1e12", "source"])
def test_solve_in_each_cell(kind, gpu_lib):
    """Three iterations. A cell's correction is off by the roundings of its own
    neighbourhood (its reach is three cells) and by the scalars', sums of 2^15
    FP64 terms: sqrt(2^15) U = 2e-14 in the mean, below 1e-12 of the largest
    value within reach."""
    shape = 34, 33, 35
    minv, b = _system(kind, shape)
    diag = _diag(minv)
    b, iters = b * diag, 3
    x = _reference(minv, diag, b, np.zeros_like(b), iters)
    st, it, rr, got = _solve(gpu_lib, "solve", _grid(*shape), minv, diag, b, np.zeros_like(b), 1e-30, iters)
    assert it == iters
    near = np.pad(np.maximum(np.abs(x), np.abs(b / diag)).astype(np.float64), iters)
    n = 2 * iters + 1
    reach = np.lib.stride_tricks.sliding_window_view(near, (n, n, n)).max((3, 4, 5))
    assert (np.abs(got - x) <= 1e-12 * reach).all()
    got2 = _solve(gpu_lib, "static", _grid(*shape), minv, diag, b, np.zeros_like(b), 1e-30, iters)
    assert got2[1:3] == (it, rr) and (got2[3] == got).all()


@pytest.mark.parametrize("kind", ["negative", "factors far up", "factors far down"])
def test_solve_at_the_bounds(kind, gpu_lib):
    """As above where a negative 1/m has FP64 take the solve from the start, and
    with factors far from 1; the whole grid is one neighbourhood."""
    shape = 34, 33, 35
    minv, b = _system("even", shape)
    if kind == "negative":
        minv[16, 16, 16] *= -0.01
    diag = _diag(minv)
    b, of = b * diag, {"factors far up": 550, "factors far down": -550}.get(kind, 0)
    x0 = 0.1 * b / diag
    x = _reference(minv, diag, b, x0, 3)
    st, it, rr, got = _solve(gpu_lib, "solve", _grid(*shape), np.ldexp(minv, of), np.ldexp(diag, of), b,
                             np.ldexp(x0, -of), 1e-30, 3)
    assert it == 3
    assert np.abs(np.ldexp(got, of) - x).max() <= 1e-12 * np.abs(x).max()
