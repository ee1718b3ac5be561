"""The exported collision draws are those of the float64 step: the axis is a unit
vector to the rounding of its components, and one free-running step is the step
that the exported draws make."""
from fractions import Fraction

import numpy as np
import pytest

import cilia_gpu as cg
from test_gpu_fixed_limits import numpy_step

pytestmark = pytest.mark.gpu


def test_the_axis_has_unit_length_to_its_components_rounding():
    """Each component is the nearest float64 number of a unit vector's (known to
    2^-59): |r|^2 differs from 1 by at most twice the sum of |r_i| times half a
    unit of r_i, and 2^-57."""
    _, ax = cg.collision_draws(10, 4000, seed=99, step=2, gamma=False)
    for r in ax:
        n2 = sum(Fraction(c) ** 2 for c in r)
        bound = sum(2 * abs(Fraction(c)) * Fraction(np.spacing(abs(c))) / 2 for c in r) + Fraction(1, 1 << 57)
        assert abs(n2 - 1) <= bound, r


@pytest.mark.parametrize("box", [(6, 7, 5), (40, 36, 38)])  # both forms of the cell maps
def test_one_step_uses_the_exported_draws(box):
    """Tolerance as test_gpu_fixed_limits.py."""
    rng = np.random.default_rng(6)
    nc = box[0] * box[1] * box[2]
    n = 2000
    pos = rng.uniform(0, 1, (n, 3)) * (6, 7, 5)
    vel = rng.normal(size=(n, 3))
    a = np.array([0.3, 0.6, 0.8])
    e = cg.Engine(box, tstep=0.1, ststep=0.002, seed=17)
    e.set_fluid(pos, vel)
    e.shift = a
    e.run(1)
    x, v = e.fluid()
    c = np.floor(pos + a).astype(int) % box
    count = np.bincount(c[:, 0] + box[0] * (c[:, 1] + box[1] * c[:, 2]), minlength=nc)
    gamma = np.zeros(nc)
    for k in np.unique(count[count > 1]):
        g, _ = cg.collision_draws(int(k), nc, seed=17, step=1, axis=False)
        gamma[count == k] = g[count == k]
    _, axis = cg.collision_draws(10, nc, seed=17, step=1, gamma=False)
    _, wv = numpy_step(pos, vel, box, 0.1, a, gamma, axis)
    assert np.abs(v - wv).max() < 1e-12 * np.abs(wv).max()
