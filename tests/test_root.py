"""The distance sweeps' square root and division by three, on the host, against
the correctly rounded ones: random numbers, and those next to where a rounding
turns over (squares of numbers and of midpoints, powers of two, multiples of
three), from reciprocal roots off by up to 2^-20."""
import ctypes as C
import pathlib
import subprocess

import numpy as np

CSRC = pathlib.Path(__file__).resolve().parents[1] / "eulersf_gb300" / "csrc"
HARNESS = r"""
#include <cmath>
#include "esf_root.cuh"
extern "C" void h_root(int n, const double* x, const double* off, double* out) {
  for (int i = 0; i < n; i++)
    out[i] = esf::root_from(x[i], (float)((1 + off[i]) / std::sqrt((double)esf::leading_float(x[i]))));
}
extern "C" void h_third(int n, const double* x, double* third, double* half) {
  for (int i = 0; i < n; i++) third[i] = esf::third_of(x[i]), half[i] = esf::half_of(x[i]);
}
"""


def test_root_and_third(tmp_path):
    src, so = tmp_path / "h.cpp", tmp_path / "h.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(CSRC),
                    "-I", "/usr/local/cuda/include", "-o", str(so), str(src)], check=True)
    h = C.CDLL(str(so))
    arr = lambda a: a.ctypes.data_as(C.c_void_p)
    rng = np.random.default_rng(8)
    n = 200000
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-60, 59, n))
    g = rng.uniform(1.0, 2.0, n)
    m = g * g + g * 2.0**-52  # next to the squares of the midpoints g + ulp / 2
    two = np.ldexp(1.0, np.arange(-59, 59))
    edge = np.concatenate([g * g, m, two])
    x = np.concatenate([x, edge, np.nextafter(edge, 0), np.nextafter(edge, np.inf)])
    out = np.zeros_like(x)
    for _ in range(3):
        h.h_root(len(x), arr(x), arr(rng.uniform(-9.5e-7, 9.5e-7, len(x))), arr(out))
        assert (out == np.sqrt(x)).all()
    t = np.concatenate([x, 3.0 * rng.integers(1, 2**51, n), rng.integers(1, 2**53, n).astype(float), 1.5 * two,
                        np.nextafter(1.5 * two, 0)])
    third, half = np.zeros_like(t), np.zeros_like(t)
    h.h_third(len(t), arr(t), arr(third), arr(half))
    assert (third == t / 3.0).all() and (half == t / 2.0).all()
