"""mpcd_fluid_step_noalloc decides on the device whether a step happens: a
refused step leaves every particle as it was, and the next step is not touched
by what the refused one had binned.  Two good steps of the same input differ by
the order of float additions into the cell sums: 10 of them, 2^-24 each and of
order one, give 1e-5 with room."""
import ctypes

import numpy as np
import pytest

import cilia_gpu as cg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, n", [((2, 2, 2), 1), ((5, 7, 3), 1051), ((33, 20, 41), 270601)])
def test_refused_step_leaves_no_trace(sizes, n):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3)) * sizes
    cell = np.minimum(np.floor(pos).astype(np.int64), np.array(sizes) - 1)
    P = np.empty((n, 4), np.float32)
    P[:, :3] = np.clip(pos - cell, 0, 1 - 2.0 ** -24)
    P[:, 3] = (cell[:, 0] | cell[:, 1] << 10 | cell[:, 2] << 20).astype(np.uint32).view(np.float32)
    V = np.zeros((n, 4), np.float32)
    V[:, :3] = rng.normal(size=(n, 3))
    dp = ctypes.POINTER(ctypes.c_double)
    a, b, diss = np.array([0.2, 0.7, 0.4]), np.array([0.9, 0.1, 0.5]), ctypes.c_double(-7.0)

    def step(p, v):
        q, w = torch.from_numpy(p).cuda(), torch.from_numpy(v).cuda()
        torch.cuda.synchronize()
        rc = cg.lib().mpcd_fluid_step_noalloc((ctypes.c_int * 3)(*sizes), n, ctypes.c_void_p(q.data_ptr()),
                                              ctypes.c_void_p(w.data_ptr()), 0.1, a.ctypes.data_as(dp), b.ctypes.data_as(dp),
                                              5, 9, ctypes.byref(diss), None)
        return rc, q.cpu().numpy(), w.cpu().numpy(), diss.value

    rc, p0, v0, d0 = step(P, V)
    assert rc == 0
    bad = P.copy()
    bad[n // 2, 1] = np.float32(np.nan)  # not inside [0, 1)
    diss.value = -7.0
    rc, p1, v1, d1 = step(bad, V)
    assert rc == 4 and d1 == -7.0  # MPCD_EDEVICE
    assert np.array_equal(p1.view(np.uint32), bad.view(np.uint32)) and np.array_equal(v1, V)
    rc, p2, v2, d2 = step(P, V)
    assert rc == 0
    assert np.abs(v2 - v0).max() < 1e-5
    at = lambda p: (p[:, 3].copy().view(np.uint32)[:, None] >> np.array([0, 10, 20]) & 1023) + p[:, :3].astype(float)
    d = at(p2) - at(p0)
    assert np.abs(d - np.round(d / sizes) * sizes).max() < 1e-5
    assert abs(d2 - d0) < 1e-5 * n
