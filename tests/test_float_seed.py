"""The float nearest to a float64 number by integer arithmetic
(csrc/fixed_offset.cuh, the seed of the reciprocal square root), compiled for the
CPU: the bits of the conversion, ties to even included."""
import ctypes
import os
import subprocess

import numpy as np

from conftest import PKG

SRC = r"""
#include "fixed_offset.cuh"
extern "C" void bits(const double* x, unsigned* r, int n) {
  for (int i = 0; i < n; ++i) r[i] = mpcd::nearest_float_bits(x[i]);
}
"""


def test_nearest_float(tmp_path):
    src, so = tmp_path / "s.cpp", tmp_path / "s.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                    str(so)], check=True)
    rng = np.random.default_rng(4)
    x = np.exp2(rng.uniform(-100, 99.9, 200000))
    f = x.astype(np.float32)
    tie = (f.astype(np.float64) + np.nextafter(f, np.float32(np.inf)).astype(np.float64)) / 2
    x = np.concatenate([x, f.astype(np.float64), tie, np.nextafter(tie, 0), np.nextafter(tie, np.inf),
                        2.0 ** np.arange(-100, 100), np.nextafter(2.0 ** np.arange(-99, 100), 0)])
    got = np.zeros(len(x), dtype=np.uint32)
    ctypes.CDLL(str(so)).bits(x.ctypes.data_as(ctypes.c_void_p), got.ctypes.data_as(ctypes.c_void_p), len(x))
    assert np.array_equal(got, x.astype(np.float32).view(np.uint32))
