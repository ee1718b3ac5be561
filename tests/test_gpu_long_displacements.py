"""Displacements of four cells and more in one float64 step, across the edge of a
long box.  Reference: exact rational arithmetic.  Bound: the velocity's rounding
in the collision (2 units of 2^-46, times the time step: 3e-15), the offset's (12: 9e-16) and
the position's (2e-15 at 12); a coordinate near 1000 would round to 6e-14."""
from fractions import Fraction

import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu


def test_fast_particles_across_the_edge_of_a_long_box():
    box = (1000, 12, 12)
    rng = np.random.default_rng(2)
    pos = np.array([[991.0 + 2 * i, 1.5 + 2 * j, 1.5 + 2 * k] for i in range(5) for j in range(5) for k in range(5)])
    pos[:, 0] += rng.uniform(0.2, 0.8, len(pos))
    vel = np.zeros_like(pos)
    vel[:, 0] = rng.uniform(100.0, 120.0, len(pos))  # 10 to 12 cells, past the edge
    e = cg.Engine(box, tstep=0.1, ststep=0.002, seed=3)
    e.set_fluid(pos, vel)
    e.run(1)
    x, _ = e.fluid()
    worst = 0.0
    for a, v, b in zip(pos[:, 0], vel[:, 0], x[:, 0]):
        exact = Fraction(a) + Fraction(v) * Fraction(0.1)
        d = Fraction(b) - (exact - 1000 if exact >= 1000 else exact)
        assert exact >= 1000 and b < 12
        worst = max(worst, abs(float(d)))
    assert worst < 1e-14
