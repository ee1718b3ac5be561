"""Cells of one particle, which a collision leaves as it is whatever its speed
(u = v, nothing to rotate or scale): components below, at and beyond the ends of
the fixed-point form of the float64 step, with and without a body force.
Tolerance: 1e-14 of the particle's speed, some tens of float64 roundings."""
import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu

SPEEDS = [0.0, 0.7, 7.9, 8.0, 8.1, 15.99, 16.0, 31.0, 33.0, 55.9, 56.1, 57.0, 60.0, 63.9, 64.0, 65.0, 300.0, 1e5]


@pytest.mark.parametrize("gravity", [0.0, 0.5])
@pytest.mark.parametrize("box", [6, 80])  # both forms of the cell maps
def test_a_lone_particle_keeps_its_velocity(box, gravity):
    combos = [(a * s, b * t, 0.3) for s in SPEEDS for t in SPEEDS[::3] for a in (1, -1) for b in (1, -1)]
    combos += [(c[2], c[0], c[1]) for c in combos] + [(c[1], c[2], c[0]) for c in combos]
    for k in range(0, len(combos), 27):
        vel = np.array(combos[k:k + 27], dtype=float)
        n = len(vel)
        i = np.arange(n)
        # no two of them share a cell for any grid shift
        pos = np.stack([1.5 + 2 * (i % 3) * (box // 6), 1.5 + 2 * (i // 3 % 3) * (box // 6), 1.5 + 2 * (i // 9) * (box // 6)],
                       axis=1)
        e = cg.Engine(box, tstep=0.1, ststep=0.002, gravity=gravity)
        e.set_fluid(pos % box, vel)
        e.run(1)
        x, v = e.fluid()
        e.close()
        want = vel + [gravity * 0.1, 0.0, 0.0]
        top = np.maximum(1.0, np.abs(vel).max(axis=1, keepdims=True))
        assert (np.abs(v - want) <= 1e-14 * top).all()
        d = x - (pos + 0.1 * vel)
        d -= np.round(d / box) * box
        assert (np.abs(d) <= 1e-14 * np.maximum(box, top)).all()
