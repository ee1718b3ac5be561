"""Collision maps in fixed point whose thermostat factor is 2 to 8 (held divided by
four, csrc/fixed_collide.cuh), compiled for the CPU and compared with exact rational
arithmetic.

Bounds, as in test_fixed_collide.py with everything that carries the factor four
times as large and mean velocities below 2 in place of 8, in units of the last
place: a map entry 8 (before the factor); b 24 from the entries, 6 from its
products, 1 for its rounding; the application 4 x 6 for the products of low halves
and 1."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import PKG
from test_fixed_collide import COS, ONE56, ONE58, ONE59, ONE60, SIN, exact_map

SRC = r"""
#include "fixed_collide.cuh"
using namespace mpcd;
typedef long long ll;
extern "C" int map(const ll* r, ll sc, int s, const ll* u, double ca, double sa, ll* A, ll* b, const ll* v, ll* out) {
  int64_t R[3], U[3], V[3], o[3];
  for (int i = 0; i < 3; ++i) { R[i] = r[i]; U[i] = u[i]; V[i] = v[i]; }
  uint64_t w[12];
  map_words(R, sc, U, ca, sa, w, s);
  for (int i = 0; i < 9; ++i) {
    const Limbs l = i ? word_limbs(w[i + i / 3]) : first_limbs(w[0]);
    A[i] = (ll)((uint64_t)(int64_t)l.h << 32) + l.l;
  }
  for (int i = 0; i < 3; ++i) b[i] = (ll)w[4 * i + 3];
  apply_words(w, V, o);
  for (int i = 0; i < 3; ++i) out[i] = o[i];
  return word_scale(w[0]) | (w[0] >> 32 == kMapF64 >> 32) << 4;
}
"""


@pytest.fixture(scope="module")
def fmap(tmp_path_factory):
    d = tmp_path_factory.mktemp("hot")
    src, so = d / "h.cpp", d / "h.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(so)],
                   check=True)
    f = ctypes.CDLL(str(so)).map
    P, ll = ctypes.POINTER(ctypes.c_longlong), ctypes.c_longlong
    f.argtypes = [P, ll, ctypes.c_int, P, ctypes.c_double, ctypes.c_double, P, P, P, P]
    return f


@pytest.mark.parametrize("scale", [0, 2])
@pytest.mark.parametrize("case", ["thermal", "largest"])
def test_scaled_maps(fmap, case, scale):
    rng = np.random.default_rng(8)
    arr = lambda v: (ctypes.c_longlong * len(v))(*[int(q) for q in v])
    worst64 = worst = 0.0
    factor = 1 << scale
    for k in range(400):
        if case == "thermal":  # velocities that the factor brings to a thermal spread
            x = rng.normal(size=3)
            x /= np.linalg.norm(x)
            sc = math.exp(rng.uniform(math.log(2.0), math.log(7.99))) / 4
            u = np.clip(rng.normal(size=3) * 0.7, -1.99, 1.99)
            v = u + rng.normal(size=3) / (sc * factor)
        else:
            x = np.where(rng.integers(0, 2, 3), 1.0, -1.0) / math.sqrt(3)
            if rng.integers(2):
                x = np.roll(np.array([0.0, 0.0, 1.0]), rng.integers(3)) * (1 if rng.integers(2) else -1)
            t = lambda top: math.nextafter(top, 0) * (1 if rng.integers(2) else -1)
            sc, u = abs(t(2.0)), np.array([t(2.0) for _ in range(3)])
            v = u + np.array([t(9.0) for _ in range(3)])  # the result below 128
        r = [int(q * ONE60) for q in x]
        U, V, S = [int(q * ONE58) for q in u], [int(q * ONE58) for q in v], int(sc * ONE60)
        A, b, out = arr([0] * 9), arr([0] * 3), arr([0] * 3)
        assert fmap(arr(r), S, scale, arr(U), COS, SIN, A, b, arr(V), out) == scale
        fr, fu, fv = [Fraction(q, ONE60) for q in r], [Fraction(q, ONE58) for q in U], [Fraction(q, ONE58) for q in V]
        eA, eb = exact_map(fr, Fraction(S, ONE60) * factor, fu)
        for i in range(9):
            assert abs(A[i] - eA[i] / factor * ONE59) <= 8
        for i in range(3):
            assert abs(b[i] - eb[i] * ONE56) <= 31
            own = factor * sum(Fraction(A[3 * i + j], ONE59) * fv[j] for j in range(3)) + Fraction(b[i], ONE56)
            assert abs(out[i] - own * ONE56) <= 6 * factor + 1
            e = sum(eA[3 * i + j] * fv[j] for j in range(3)) + eb[i]
            fA, fb = [float(q) for q in eA], [float(q) for q in eb]
            f64 = fA[3 * i] * v[0] + (fA[3 * i + 1] * v[1] + (fA[3 * i + 2] * v[2] + fb[i]))
            worst = max(worst, abs(float(Fraction(out[i], ONE56) - e)))
            worst64 = max(worst64, abs(float(Fraction(f64) - e)))
    if case == "thermal":
        assert worst <= worst64
