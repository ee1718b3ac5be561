"""The float64 step at and beyond the ends of its fixed-point form: velocities
around 16, mean velocities around 8, thermostat factors around 2, full
cells, a long time step, and fast particles among thermal ones.  Reference: one collision and streaming step in numpy float64 with
injected Gamma variates and axes (src/libcilia/mpcd.cpp:140-247, 285-293, with
its constants).  Tolerance: 1e-12 of the largest velocity, about a hundred
float64 roundings of the sums over a cell."""
import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu
COS, SIN = -0.6427876, 0.76604444


def numpy_step(pos, vel, sizes, h, a, gamma, axis):
    L = np.array(sizes)
    c = np.floor(pos + a).astype(int) % L
    cid = c[:, 0] + L[0] * (c[:, 1] + L[1] * c[:, 2])
    out = vel.copy()
    for k in np.unique(cid):
        m = cid == k
        v, n = vel[m], m.sum()
        u = v.mean(axis=0)
        e = (v * v).sum() - n * (u * u).sum()
        sc = np.sqrt(2 * gamma[k] / e) if n > 1 and e > 0 else 1.0
        r = axis[k]
        x = np.array([[0, -r[2], r[1]], [r[2], 0, -r[0]], [-r[1], r[0], 0]])
        R = np.outer(r, r) * (1 - COS) + COS * np.eye(3) + SIN * x
        out[m] = u + sc * (v - u) @ R.T
    return pos + h * out, out


@pytest.mark.parametrize("h", [0.1, 2.5])
@pytest.mark.parametrize("case", ["thermal", "fast", "drift", "cold", "crowded", "mixed"])
def test_ends_of_the_fixed_point_form(case, h):
    sizes = (4, 5, 3)
    nc = 60
    rng = np.random.default_rng(12)
    n = {"crowded": 40000}.get(case, 600)
    pos = rng.uniform(0, 1, (n, 3)) * sizes
    vel = rng.normal(size=(n, 3))
    gamma = rng.gamma(1.5 * (n / nc - 1), size=nc)
    if case == "fast":  # on both sides of 16
        vel *= 7.0
    if case == "drift":  # mean velocities on both sides of 8
        vel += [7.9, -0.5, 0.2]
    if case == "cold":  # factors on both sides of 2
        vel *= rng.choice([0.3, 0.5, 0.7, 0.9], size=(n, 1))
    if case == "mixed":
        vel[::50] *= 1000.0
        vel[7] = [15.9999, -15.9999, 16.0]
        vel[8] = 0.0
    axis = rng.normal(size=(nc, 3))
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    a = np.array([0.3, 0.6, 0.8])
    e = cg.Engine(sizes, tstep=h, ststep=h / 50, seed=1)
    e.set_fluid(pos, vel)
    e.shift = a
    e.prepare()
    e.step(shift_next=np.array([0.1, 0.2, 0.7]), gamma=gamma, axis=axis)
    x, v = e.fluid()
    wx, wv = numpy_step(pos, vel, sizes, h, a, gamma, axis)
    top = max(1.0, np.abs(wv).max())
    assert np.abs(v - wv).max() < 1e-12 * top
    d = x - wx
    d -= np.round(d / np.array(sizes)) * np.array(sizes)
    assert np.abs(d).max() < 1e-12 * top * max(1.0, h)
    assert x.min() >= 0 and (x <= sizes).all()
