"""Fixed-point offsets of the float64 fluid (csrc/fixed_offset.cuh), compiled for
the CPU and compared with exact rational arithmetic: streaming o += v h with
the cells moved, conversions, thresholds.

Bounds from the method: the displacement is the exact product of the two
significands truncated twice (the 128-bit product's high half, then the shift
to units of 2^-60, at least two places), so it is within 1.25 units."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import PKG

ONE = 1 << 60
SRC = r"""
#include "fixed_offset.cuh"
using namespace mpcd;
extern "C" {
int stream(unsigned long long* k, int* cells, double v, double h) {
  uint64_t o = *k; int c = 99;
  const bool ok = stream_fixed(o, c, v, fixed_step(h));
  *k = o; *cells = c; return ok;
}
unsigned long long from_double(double o) { return offset_from_double(o); }
double to_double(unsigned long long k) { return offset_to_double(k); }
unsigned long long threshold(double t) { return offset_threshold(t); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = d / "f.cpp", d / "f.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                    str(so)], check=True)
    L = ctypes.CDLL(str(so))
    u, d64 = ctypes.c_ulonglong, ctypes.c_double
    L.stream.argtypes = [ctypes.POINTER(u), ctypes.POINTER(ctypes.c_int), d64, d64]
    L.from_double.argtypes, L.from_double.restype = [d64], u
    L.to_double.argtypes, L.to_double.restype = [u], d64
    L.threshold.argtypes, L.threshold.restype = [d64], u
    return L


def stream(lib, k, v, h):
    o, c = ctypes.c_ulonglong(k), ctypes.c_int(99)
    ok = lib.stream(ctypes.byref(o), ctypes.byref(c), v, h)
    return ok, o.value, c.value


@pytest.mark.parametrize("h", [0.1, 0.01, 1.0, 0.3, 7.5, 2.0 ** -40])
def test_streaming_is_the_exact_sum_within_its_units(lib, h):
    rng = np.random.default_rng(3)
    vs = np.concatenate([rng.normal(size=400), rng.normal(size=100) * 10.0 ** rng.uniform(-300, 2, 100),
                         [0.0, -0.0, 5e-324, -5e-324, 1e-310, 2.0 ** -20, -1.0, 1.0, 30.0, -30.0]])
    edge = [0, 1, ONE - 1, ONE // 2]
    taken = 0
    for i, v in enumerate(vs):
        k = edge[i % 8] if i % 8 < 4 else int(rng.integers(0, ONE))
        ok, o, c = stream(lib, k, float(v), h)
        exact = Fraction(k, ONE) + Fraction(float(v)) * Fraction(h)
        if not ok:
            assert (o, c) == (k, 99) and abs(Fraction(float(v)) * Fraction(h)) >= 1  # unchanged, and far
            continue
        taken += 1
        assert 0 <= o < ONE
        assert abs(Fraction(o, ONE) + c - exact) <= Fraction(5, 4 * ONE), (v, k)
    assert taken > 200 or h > 1


@pytest.mark.parametrize("v", [math.inf, -math.inf, math.nan, 1e300, 41.0])
def test_streaming_declines_what_it_cannot_hold(lib, v):
    assert stream(lib, 12345, v, 0.1) == (0, 12345, 99)


def test_conversions_and_thresholds(lib):
    rng = np.random.default_rng(4)
    os_ = np.concatenate([rng.uniform(0, 1, 500), [0.0, 0.5, 1.0 - 2.0 ** -53, 2.0 ** -7, 2.0 ** -61, 5e-324]])
    for o in map(float, os_):
        k = lib.from_double(o)
        assert 0 <= k < ONE and abs(Fraction(k, ONE) - Fraction(o)) <= Fraction(1, 2 * ONE)
        if o >= 2.0 ** -7 or o == 0.0:
            assert Fraction(k, ONE) == Fraction(o) and lib.to_double(k) == o
    assert lib.to_double(ONE - 1) < 1.0
    for t in map(float, np.concatenate([rng.uniform(0, 1, 300), [1.0, 2.0 ** -53, 0.5]])):
        th = lib.threshold(t)
        for k in (th - 1, th, th + 1):
            if 0 <= k < ONE:
                assert (k >= th) == (Fraction(k, ONE) >= Fraction(t))
    assert lib.threshold(1.0) == ONE  # no offset reaches it
