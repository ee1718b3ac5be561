"""Mean velocity and relative kinetic energy of a cell in fixed point
(csrc/fixed_collide.cuh, cell_mean), compiled for the CPU and compared with exact
rational arithmetic over counts, masses and momenta up to and beyond what fits.

Bounds: a momentum is truncated by less than one unit, 1/M is off by one unit, a
product is within one unit of 2^-58, and the energy sums three products of
such a mean (below 8) with such a momentum."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import PKG

SRC = r"""
#include "fixed_collide.cuh"
using namespace mpcd;
extern "C" int mean(const double* p, double K, int num, double mass, long long* u, double* erel) {
  int64_t kin = 0, inv = 0, top, v[3] = {0, 0, 0}, e = 0;
  if (!to_fixed<50, 12>(K, kin)) return 0;
  if (num) {
    inv = (int64_t)(((1ull << 62) + (unsigned)num / 2) / (unsigned)num);
    top = mean_limit(num);
  } else {
    if (!to_fixed<62, 0>(1.0 / mass, inv)) return 0;
    top = mean_limit(mass);
  }
  const bool fit = cell_mean(p, kin, inv, top, v, e);
  for (int i = 0; i < 3; ++i) u[i] = v[i];
  *erel = from_fixed(e, 50);
  return fit;
}
"""


@pytest.fixture(scope="module")
def mean(tmp_path_factory):
    d = tmp_path_factory.mktemp("mean")
    src, so = d / "m.cpp", d / "m.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(so)],
                   check=True)
    f = ctypes.CDLL(str(so)).mean
    dp = ctypes.POINTER(ctypes.c_double)
    f.argtypes = [dp, ctypes.c_double, ctypes.c_int, ctypes.c_double, ctypes.POINTER(ctypes.c_longlong), dp]

    def call(p, K, num, mass=0.0):
        u, e = (ctypes.c_longlong * 3)(), ctypes.c_double()
        fit = f((ctypes.c_double * 3)(*p), K, num, mass, u, ctypes.byref(e))
        return fit, [Fraction(v, 1 << 58) for v in u], e.value

    return call


SPEEDS = [0.0, 1e-3, 0.7, 7.9, 8.0, 8.1, 31.0, 33.0, 55.9, 56.5, 57.0, 60.0, 63.9, 64.0, 65.0, 120.0, 127.0, 500.0]


@pytest.mark.parametrize("num", [1, 2, 3, 7, 10, 31, 63, 64, 65, 200, 255])
@pytest.mark.parametrize("sign", [1, -1])
def test_mean_is_right_or_refused(mean, num, sign):
    for axis in range(3):
        for s in SPEEDS:
            p = [0.3 * num, -0.2 * num, 0.1 * num]
            p[axis] = sign * s * num
            K = min(sum(q * q for q in p) / num + 1.0, 4095.0)
            fit, u, erel = mean(p, K, num)
            exact = [Fraction(q) / num for q in p]
            if max(abs(q) for q in exact) >= 8:
                assert not fit, (num, p)
            elif max(abs(q) for q in p) < 512 and K < 4095:
                assert fit, (num, p)
                for a, b in zip(u, exact):
                    assert abs(a - b) <= Fraction(64, num << 58) + abs(b) * Fraction(num, 1 << 62) + Fraction(1, 1 << 58)
                e = Fraction(K) - sum(a * Fraction(q) for a, q in zip(exact, p))
                assert abs(Fraction(erel) - e) <= Fraction(600, 1 << 50), (num, p)


@pytest.mark.parametrize("mass", [1.5, 5.0, 6.25, 40.0, 1000.0])
def test_mean_with_beads(mean, mass):
    rng = np.random.default_rng(3)
    for s in SPEEDS:
        p = [sign * s * mass for sign in rng.choice([-1.0, 1.0], 3)]
        K = min(sum(q * q for q in p) / mass + 1.0, 4095.0)
        fit, u, _ = mean(p, K, 0, mass)
        assert not (fit and s >= 8)
        if s < 8 and s * mass < 512 and K < 4095:
            assert fit
            for a, q in zip(u, p):
                # 1 / mass in float64, then in units of 2^-62
                assert abs(a - Fraction(q) / Fraction(mass)) <= abs(Fraction(q)) * Fraction(5, 1 << 54) + Fraction(66, 1 << 58)


@pytest.mark.parametrize("mass", [0.25, 1.0, 0.0, -5.0, float("nan")])
def test_masses_that_do_not_fit(mean, mass):
    for s in (0.1, 5.0, 60.0):
        assert not mean([s, -s, 0.0], 3 * s * s + 1, 0, mass)[0]


def test_numbers_that_are_not_finite(mean):
    for bad in (float("inf"), -float("inf"), float("nan"), 1e300, 512.0):
        assert not mean([bad, 0.0, 0.0], 1.0, 10)[0] and not mean([0.0, 0.0, bad], 1.0, 10)[0]


ENERGY = r"""
#include "fixed_collide.cuh"
using namespace mpcd;
extern "C" int energy(const double* p, double K, int num, double* u, double* erel) {
  int64_t kin = 0, v[3] = {0, 0, 0}, e = 0;
  const int bits = kinetic_fixed(K, kin);
  if (!bits) return 0;
  const int64_t inv = (int64_t)(((1ull << 62) + (unsigned)num / 2) / (unsigned)num);
  const bool fit = cell_energy(p, kin, bits, inv, mean_top(bits, num), num == 1, v, e);
  for (int i = 0; i < 3; ++i) u[i] = from_fixed(v[i], kVelBits);
  *erel = from_fixed(e, bits);
  return fit;
}
"""


@pytest.mark.parametrize("num", [2, 3, 10, 40])
@pytest.mark.parametrize("drift", [0.0, 0.3, 5.0])
def test_relative_energy_is_as_close_as_in_float64(tmp_path, num, drift):
    """Cells at thermal speeds from 1 down: what is refused is cold, and what is
    kept has an energy no further from the exact one than float64's in the mean;
    at worst by the roundings of its units beside the half unit of float64 that
    both end with (three products of one unit each, and the mean's rounding)."""
    src, so = tmp_path / "e.cpp", tmp_path / "e.so"
    src.write_text(ENERGY)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                    str(so)], check=True)
    f = ctypes.CDLL(str(so)).energy
    dp = ctypes.POINTER(ctypes.c_double)
    f.argtypes = [dp, ctypes.c_double, ctypes.c_int, dp, dp]
    rng = np.random.default_rng(11)
    ours, theirs = [], []
    for speed in (1.0, 0.5, 0.2, 0.05, 1e-3, 1e-6, 1e-9):
        for _ in range(150):
            v = rng.normal(size=(num, 3)) * speed + drift
            p, K = v.sum(axis=0), float((v * v).sum())
            u, e = (ctypes.c_double * 3)(), ctypes.c_double()
            fit = f((ctypes.c_double * 3)(*p), K, num, u, ctypes.byref(e))
            exact = Fraction(K) - sum(Fraction(q) ** 2 for q in p) / num
            if exact < Fraction(1, 17):
                assert not fit
            if not fit:
                assert exact < Fraction(1, 15) or np.abs(p).max() / num > 7.9 or K > 4000
                continue
            inv = 1.0 / num
            w = p * inv
            e64 = K - (w[0] * p[0] + w[1] * p[1] + w[2] * p[2])
            ours.append(abs(float(Fraction(e.value) - exact)))
            theirs.append(abs(float(Fraction(e64) - exact)))
    assert len(ours) > 100
    assert np.mean(ours) <= np.mean(theirs) and max(ours) <= max(theirs) + 4 * 2.0 ** -50
