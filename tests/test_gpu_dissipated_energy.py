"""The float64 step's account of dissipated energy: sum of v^2 before a collision
less the sum after it, to float64's precision.  Reference: the exactly rounded
sums of the velocities put in and read back.

Bound, rms over the seeds: the cells' sums (64 of about ten addends near 32:
1e-13), about a dozen additions of warps' and blocks' sums to a total near 2000 (half a
unit each, 1.1e-13: 4e-13), the velocities' own rounding (640 of 2 v 2^-54:
3e-15); 1.5e-12 leaves a factor of three."""
import math

import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu


def test_dissipated_energy_of_one_collision():
    off = []
    for seed in range(24):
        rng = np.random.default_rng(seed)
        pos, vel = rng.uniform(0, 4, (640, 3)), rng.normal(size=(640, 3))
        e = cg.Engine(4, tstep=0.1, ststep=0.002, seed=seed + 1)
        e.set_fluid(pos, vel)
        e.run(1)
        _, after = e.fluid()
        exact = math.fsum((vel * vel).ravel()) - math.fsum((after * after).ravel())
        off.append(e.observables()["diss_energy"] - exact)
        e.close()
    assert np.sqrt(np.mean(np.square(off))) < 1.5e-12, off
