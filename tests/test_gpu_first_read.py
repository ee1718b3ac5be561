"""The first read-back of a prepared engine or ensemble makes nothing that a later
one does not: no buffer, stream or event (they cost a first measured call up
to milliseconds).  A preloaded library counts the CUDA runtime calls that make them."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
extern "C" {
int made = 0;
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }
int cudaMalloc(void** p, unsigned long n) { ++made; return ((int (*)(void**, unsigned long))real("cudaMalloc"))(p, n); }
int cudaHostAlloc(void** p, unsigned long n, unsigned f) {
  ++made;
  return ((int (*)(void**, unsigned long, unsigned))real("cudaHostAlloc"))(p, n, f);
}
int cudaStreamCreateWithFlags(void** p, unsigned f) {
  ++made;
  return ((int (*)(void**, unsigned))real("cudaStreamCreateWithFlags"))(p, f);
}
int cudaEventCreateWithFlags(void** p, unsigned f) {
  ++made;
  return ((int (*)(void**, unsigned))real("cudaEventCreateWithFlags"))(p, f);
}
}
"""
CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
import cilia_gpu as cg, simcfg
made = ctypes.c_int.in_dll(ctypes.CDLL(%r), "made")
rng = np.random.default_rng(1)
for prec in (cg.MPCD_FP64, cg.MPCD_FP32):
    for edge in (6, 48):  # read at once, and in parts
        for nb in (100, 4000):  # through pinned memory, and by copies
            n = 10 * edge ** 3
            e = cg.Engine(edge, precision=prec)
            e.set_fluid(rng.uniform(0, edge, (n, 3)), rng.normal(size=(n, 3)))
            e.set_beads(rng.uniform(0, edge, (nb, 3)), np.zeros((nb, 3)))
            e.prepare()
            before = made.value
            assert before > 0
            e.fluid()
            e.beads(nb)
            assert made.value == before, ("engine", prec, edge, nb, made.value - before)
            e.close()
specs = [dict(L=16, radius=4.0, n_cilia=3, rodlength=10, seed=1), dict(L=32, radius=8.0, n_cilia=60, rodlength=15, seed=2)]
b = cg.Batch.for_specs(specs)
ids = []
for sp in specs:
    r = b.add_cfg(simcfg.dumps(simcfg.swimmer_config(sp["L"], radius=sp["radius"], n_cilia=sp["n_cilia"],
                                                     rodlength=sp["rodlength"], seed=sp["seed"])), ststep=0.002)
    b.admit(r)
    ids.append((r, 643 + 3 * sp["n_cilia"] * sp["rodlength"]))
before = made.value
for r, nb in ids:
    b.beads(r, nb)
assert made.value == before, ("batch", made.value - before)
print("nothing made")
"""


def test_first_reads_make_nothing(tmp_path):
    src, so = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD % (PKG, str(so))], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0 and "nothing made" in r.stdout, r.stdout + r.stderr
