"""Cold fluids in the float64 step: the thermostat brings a cell to its
temperature however little its particles differ, down to speeds whose squares
vanish in fixed point.  Reference and tolerance: test_gpu_fixed_limits.py."""
import numpy as np
import pytest

import cilia_gpu as cg
from test_gpu_fixed_limits import numpy_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(4, 5, 3), (40, 36, 38)])  # both forms of the cell maps
@pytest.mark.parametrize("speed", [1.0, 0.2, 0.1, 1e-2, 1e-4, 1e-7, 1e-9, 1e-12])
@pytest.mark.parametrize("density", [2, 10])
def test_a_cold_fluid_is_thermostatted(box, speed, density):
    rng = np.random.default_rng(4)
    nc = box[0] * box[1] * box[2]
    corner = np.array((4, 5, 3))  # the particles fill a corner of the larger box
    n = density * 60
    pos = rng.uniform(0, 1, (n, 3)) * corner
    vel = rng.normal(size=(n, 3)) * speed
    gamma = rng.gamma(1.5 * max(1, density - 1), size=nc)
    axis = rng.normal(size=(nc, 3))
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    a = np.array([0.3, 0.6, 0.8])
    e = cg.Engine(box, tstep=0.1, ststep=0.002, seed=1)
    e.set_fluid(pos, vel)
    e.shift = a
    e.prepare()
    e.step(shift_next=np.array([0.1, 0.2, 0.7]), gamma=gamma, axis=axis)
    x, v = e.fluid()
    wx, wv = numpy_step(pos, vel, box, 0.1, a, gamma, axis)
    top = max(1.0, np.abs(wv).max())
    assert np.abs(v - wv).max() < 1e-12 * top
    d = x - wx
    d -= np.round(d / np.array(box)) * np.array(box)
    assert np.abs(d).max() < 1e-12 * top
    # particles alone in their cells keep their speed to float64's own precision of it
    c = np.floor(pos + a).astype(int) % box
    cid = c[:, 0] + box[0] * (c[:, 1] + box[1] * c[:, 2])
    alone = np.bincount(cid, minlength=nc)[cid] == 1
    assert (np.abs(v - vel)[alone] <= 1e-14 * np.abs(vel[alone]).max(axis=1, keepdims=True)).all()
