"""A read-back whose kernel the CUDA runtime refuses to launch returns an error,
not what an earlier call left in the buffers.  The refusal is a stand-in's: a
preloaded library answers the launch with an error code, and nothing of it
reaches the GPU."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
extern "C" {
int refuse = 0;  // launches to let through before one is refused, counted from 1; 0: none
struct dim { unsigned x, y, z; };
static bool due() { return refuse > 0 && --refuse == 0; }
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }
int __cudaLaunchKernel(void* k, dim g, dim b, void** a, unsigned long m, void* s) {
  typedef int (*F)(void*, dim, dim, void**, unsigned long, void*);
  return due() ? 701 : ((F)real("__cudaLaunchKernel"))(k, g, b, a, m, s);
}
int cudaLaunchKernelExC(const void* c, const void* f, void** a) {
  typedef int (*F)(const void*, const void*, void**);
  return due() ? 701 : ((F)real("cudaLaunchKernelExC"))(c, f, a);
}
}
"""
CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
import cilia_gpu as cg, simcfg
refuse = ctypes.c_int.in_dll(ctypes.CDLL(%r), "refuse")

def refused(call, launches):
    for k in range(1, launches + 1):
        refuse.value = k
        try:
            call()
        except cg.MpcdError:
            assert refuse.value == 0
        else:
            raise SystemExit("launch %%d of %%r was refused, and the call returned" %% (k, call))
    call()  # and the next one is served

rng = np.random.default_rng(1)
for prec in (cg.MPCD_FP64, cg.MPCD_FP32):
    for edge, launches in ((6, 1), (48, 4)):  # in one launch, and in parts
        n = 10 * edge ** 3
        e = cg.Engine(edge, precision=prec)
        e.set_fluid(rng.uniform(0, edge, (n, 3)), rng.normal(size=(n, 3)))
        e.run(1)
        e.fluid()
        refused(e.fluid, launches)
        e.close()
for nb in (100, 4000):  # through pinned memory, and by copies
    e = cg.Engine(24)
    e.set_fluid(rng.uniform(0, 24, (1000, 3)), rng.normal(size=(1000, 3)))
    e.set_beads(rng.uniform(2, 22, (nb, 3)), np.zeros((nb, 3)))
    e.run(1)
    e.beads(nb)
    refused(lambda: e.beads(nb), 1)
    e.close()
text = simcfg.dumps(simcfg.swimmer_config(16, radius=4.0, n_cilia=3, rodlength=10, seed=1))
b = cg.Batch.for_specs([dict(L=16, radius=4.0, n_cilia=3, rodlength=10, seed=1)])
r = b.add_cfg(text, ststep=0.002)
b.admit(r)
b.set_steps(r, 10)
b.run(1)
b.sync()
b.beads(r, 643 + 90)
refused(lambda: b.beads(r, 643 + 90), 1)
print("all refusals reported")
"""


def test_refused_launches_are_reported(tmp_path):
    src, so = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD % (PKG, str(so))], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0 and "all refusals reported" in r.stdout, r.stdout + r.stderr
