"""The fixed-point collision of the float64 fluid (csrc/fixed_collide.cuh),
compiled for the CPU and compared with exact rational arithmetic: conversions,
the map of a cell, its application, the kinetic energy and the streaming.

Bounds from the method, in units of the last place: a rounded or truncated
product (mul_sh) is within 1; a map entry is the sum of at most two products,
each of a factor within one unit, times a factor below two: 8; b adds three
products of such entries with |u| < 8, in units eight times as large, and the
roundings: 28.
"""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import PKG

SRC = r"""
#include "fixed_collide.cuh"
using namespace mpcd;
typedef long long ll;
extern "C" {
int fix50(double x, ll* r) { int64_t v = 77; const bool ok = to_fixed<50, 12>(x, v); *r = v; return ok; }
int fix58(double x, ll* r) { int64_t v = 77; const bool ok = to_fixed<58, 4>(x, v); *r = v; return ok; }
int fix60(double x, ll* r) { int64_t v = 77; const bool ok = to_fixed<60, 1>(x, v); *r = v; return ok; }
double unfix(ll x, int bits) { return from_fixed(x, bits); }
ll mul56(ll a, ll b) { return mul_sh<56>(split_limbs(a), split_limbs(b)); }
ll mul60(ll a, ll b) { return mul_sh<60>(split_limbs(a), split_limbs(b)); }
void axis(const float* f, ll* r) {
  int64_t v[3] = {axis_fixed(f[0]), axis_fixed(f[1]), axis_fixed(f[2])};
  axis_normalise(v);
  for (int i = 0; i < 3; ++i) r[i] = v[i];
}
void map(const ll* r, ll sc, const ll* u, double ca, double sa, ll* A, ll* b, const ll* v, ll* out, ll* K) {
  int64_t R[3], U[3], V[3], o[3];
  for (int i = 0; i < 3; ++i) { R[i] = r[i]; U[i] = u[i]; V[i] = v[i]; }
  uint64_t w[12];
  map_words(R, sc, U, ca, sa, w);
  for (int i = 0; i < 9; ++i) { const Limbs l = word_limbs(w[i + i / 3]); A[i] = (ll)((uint64_t)(int64_t)l.h << 32) + l.l; }
  for (int i = 0; i < 3; ++i) b[i] = (ll)w[4 * i + 3];
  apply_words(w, V, o);
  for (int i = 0; i < 3; ++i) out[i] = o[i];
  if (K) *K = square_words(split_limbs((int64_t)((uint64_t)o[0] << 2)), split_limbs((int64_t)((uint64_t)o[1] << 2)),
                    split_limbs((int64_t)((uint64_t)o[2] << 2)));
}
int stream(unsigned long long* k, int* cells, ll v, double h, double kick, ll* xkick) {
  int64_t x = 0;
  const StreamStep s = stream_step(h, kick, &x);
  uint64_t o = *k;
  int c = 99;
  stream_words(o, c, split_limbs(v), s);
  *k = o; *cells = c; *xkick = x;
  return s.vmax;
}
}
"""
COS, SIN = -0.6427876, 0.76604444
ONE56, ONE58, ONE59, ONE60 = (1 << k for k in (56, 58, 59, 60))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("collide")
    src, so = d / "c.cpp", d / "c.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = ctypes.CDLL(str(so))
    ll, d64, P = ctypes.c_longlong, ctypes.c_double, ctypes.POINTER
    for f in (L.fix50, L.fix58, L.fix60):
        f.argtypes = [d64, P(ll)]
    L.unfix.argtypes, L.unfix.restype = [ll, ctypes.c_int], d64
    for f in (L.mul56, L.mul60):
        f.argtypes, f.restype = [ll, ll], ll
    L.axis.argtypes = [P(ctypes.c_float), P(ll)]
    L.map.argtypes = [P(ll), ll, P(ll), d64, d64, P(ll), P(ll), P(ll), P(ll), P(ll)]
    L.stream.argtypes = [P(ctypes.c_ulonglong), P(ctypes.c_int), ll, d64, d64, P(ll)]
    return L


@pytest.mark.parametrize("name, bits, emax", [("fix50", 50, 12), ("fix58", 58, 4), ("fix60", 60, 1)])
def test_conversion(lib, name, bits, emax):
    f, r = getattr(lib, name), ctypes.c_longlong()
    top = float(2 ** emax)
    xs = np.concatenate([np.random.default_rng(1).normal(size=300), [0.0, -0.0, 5e-324, 1e-300, math.nextafter(top, 0.0)],
                         2.0 ** np.arange(-70, emax)])
    for x in np.concatenate([xs, -xs]):
        if abs(x) >= top:
            continue
        assert f(float(x), ctypes.byref(r))
        exact = Fraction(float(x)) * (1 << bits)
        assert r.value == (math.floor(exact) if exact >= 0 else math.ceil(exact)), x
    for x in (top, -top, 1e300, math.inf, -math.inf, math.nan):
        assert not f(x, ctypes.byref(r)), x
    rng = np.random.default_rng(2)
    vals = [0, 1, -1, (1 << 62) - 1, -(1 << 62), (1 << 53) + 1, (1 << 54) - 1] + [
        int(v) >> int(s) for v, s in zip(rng.integers(-1 << 62, 1 << 62, 300), rng.integers(0, 60, 300))]
    for v in vals:
        got, exact = Fraction(lib.unfix(v, bits)), Fraction(v, 1 << bits)
        assert abs(got - exact) <= abs(exact) / (1 << 53), v


@pytest.mark.parametrize("shift", [56, 60])
def test_product(lib, shift):
    f, rng = getattr(lib, f"mul{shift}"), np.random.default_rng(shift)
    m = 1 << 62
    ends = [0, 1, -1, m, -m, m - 1, (1 << 31), -(1 << 31), (1 << 32) - 1, (1 << 59) + (1 << 31)]
    pairs = [(a, b) for a in ends for b in ends] + [
        (int(a) >> int(s), int(b) >> int(t)) for a, b, s, t in zip(
            rng.integers(-m, m, 2000), rng.integers(-m, m, 2000), rng.integers(0, 40, 2000), rng.integers(0, 40, 2000))]
    for a, b in pairs:
        exact = Fraction(a * b, 1 << shift)
        if abs(exact) < m:
            assert abs(f(a, b) - exact) <= 1, (a, b)


def test_axis(lib):
    rng = np.random.default_rng(3)
    for _ in range(300):
        x = rng.normal(size=3)
        x = (x / np.linalg.norm(x)).astype(np.float32)
        if rng.integers(4) == 0:
            x = np.array([0.0, -1.0, 0.0], np.float32) if rng.integers(2) else np.array([1e-30, 0.0, 1.0], np.float32)
        r = (ctypes.c_longlong * 3)()
        lib.axis(x.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), r)
        # |r|^2 - 1 = -5/8 e^3 (|e| < 2^-20) and the roundings, 2 per component
        assert abs(sum(Fraction(v, ONE60) ** 2 for v in r) - 1) < Fraction(16, ONE60)
        n = math.sqrt(float((x.astype(float) ** 2).sum()))
        assert max(abs(v / ONE60 - float(c) / n) for v, c in zip(r, x)) < 4e-16


def exact_map(r, sc, u):
    ca, sa = Fraction(COS), Fraction(SIN)
    oc = Fraction(1.0 - COS)
    x, y, z = r
    R = [x * x * oc + ca, x * y * oc - z * sa, x * z * oc + y * sa, x * y * oc + z * sa, y * y * oc + ca,
         y * z * oc - x * sa, x * z * oc - y * sa, y * z * oc + x * sa, z * z * oc + ca]
    A = [sc * q for q in R]
    return A, [u[i] - sum(A[3 * i + j] * u[j] for j in range(3)) for i in range(3)]


@pytest.mark.parametrize("case", ["thermal", "largest"])
def test_map_and_application(lib, case):
    rng = np.random.default_rng(5)
    arr = lambda v: (ctypes.c_longlong * len(v))(*[int(q) for q in v])
    worst64 = worst = 0.0
    for k in range(400):
        if case == "thermal":
            x = rng.normal(size=3)
            x /= np.linalg.norm(x)
            sc, u, v = abs(rng.normal(1, 0.2)), rng.normal(size=3) * 0.4, rng.normal(size=3)
            sc = min(sc, 1.9)
        else:  # the ends of every range, all signs
            x = np.where(rng.integers(0, 2, 3), 1.0, -1.0) / math.sqrt(3)
            if rng.integers(2):
                x = np.array([0.0, 0.0, 1.0]) * (1 if rng.integers(2) else -1)
            t = lambda top: math.nextafter(top, 0) * (1 if rng.integers(2) else -1)
            sc, u, v = abs(t(2.0)), np.array([t(8.0) for _ in range(3)]), np.array([t(16.0) for _ in range(3)])
        r = [int(q * ONE60) for q in x]
        U, V, S = [int(q * ONE58) for q in u], [int(q * ONE58) for q in v], int(sc * ONE60)
        A, b, out, K = arr([0] * 9), arr([0] * 3), arr([0] * 3), ctypes.c_longlong()
        lib.map(arr(r), S, arr(U), COS, SIN, A, b, arr(V), out, None)
        fr, fu, fv = [Fraction(q, ONE60) for q in r], [Fraction(q, ONE58) for q in U], [Fraction(q, ONE58) for q in V]
        eA, eb = exact_map(fr, Fraction(S, ONE60), fu)
        for i in range(9):
            assert abs(A[i] - eA[i] * ONE59) <= 8
        for i in range(3):
            assert abs(b[i] - eb[i] * ONE56) <= 28
            own = sum(Fraction(A[3 * i + j], ONE59) * fv[j] for j in range(3)) + Fraction(b[i], ONE56)
            assert abs(out[i] - own * ONE56) <= 7  # three products of low halves, one rounding
            # against the same map in float64 throughout
            e = sum(eA[3 * i + j] * fv[j] for j in range(3)) + eb[i]
            fA, fb = [float(q) for q in eA], [float(q) for q in eb]
            f64 = fA[3 * i] * v[0] + (fA[3 * i + 1] * v[1] + (fA[3 * i + 2] * v[2] + fb[i]))
            worst = max(worst, abs(float(Fraction(out[i], ONE56) - e)))
            worst64 = max(worst64, abs(float(Fraction(f64) - e)))
        if max(abs(o) for o in out) < 16 * ONE56:
            lib.map(arr(r), S, arr(U), COS, SIN, A, b, arr(V), out, ctypes.byref(K))
            assert abs(K.value - sum(Fraction(o, ONE56) ** 2 for o in out) * (1 << 52)) <= 8
    if case == "thermal":
        assert worst <= worst64  # no further off than float64 applied to the rounded exact map


@pytest.mark.parametrize("h", [0.1, 0.005, 1.0, 1.999, 2.0 ** -20])
def test_streaming(lib, h):
    rng = np.random.default_rng(7)
    x = ctypes.c_longlong()
    for k in range(500):
        k0, c = ctypes.c_ulonglong(int(rng.integers(0, ONE60))), ctypes.c_int()
        if k < 2:
            k0 = ctypes.c_ulonglong((0, ONE60 - 1)[k])
        o = k0.value
        v = rng.normal() * min(1.0, 1.0 / h)
        V = int(v * ONE58)
        vmax = lib.stream(ctypes.byref(k0), ctypes.byref(c), V, h, 0.25, ctypes.byref(x))
        assert 0 <= k0.value < ONE60
        d = c.value * ONE60 + k0.value - o
        assert abs(d - Fraction(V, ONE58) * Fraction(h) * ONE60) <= 1 + abs(v) / 2  # h in units of 2^-61
    top = Fraction(vmax << 32, ONE56)
    assert top + Fraction(1, 4) <= 16 and top * Fraction(h) <= 4 and x.value == ONE56 // 4
    for bad in (2.0, 100.0, math.nan, -1.0):
        assert lib.stream(ctypes.byref(k0), ctypes.byref(c), V, bad, 0.0, ctypes.byref(x)) == 0
    assert lib.stream(ctypes.byref(k0), ctypes.byref(c), V, h, 9.0, ctypes.byref(x)) == 0 and x.value == 0
