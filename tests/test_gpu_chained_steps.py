"""Steps of a plain fluid launched one into the other (each kernel placed while
its predecessor drains) against the same steps with a wait after each: the same
trajectory up to the order of the atomic additions into the cell sums.  Float64
to 1e-9 after 6 steps; split precision for 99.9 % of the particles to 1e-4 after
3 (a particle on a cell's edge may collide with another cell)."""
import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cg.MPCD_FP64, cg.MPCD_FP32])
@pytest.mark.parametrize("sizes, walls", [((2, 2, 2), 0), ((9, 7, 5), 0), ((9, 7, 6), 1), ((40, 33, 41), 0)])
def test_chain_of_steps(sizes, walls, precision):
    rng = np.random.default_rng(11)
    n = 10 * int(np.prod(sizes))
    top = np.array(sizes, float) - [0, 0, 1 if walls else 0]
    pos, vel = rng.uniform(0, 1, (n, 3)) * top, rng.normal(size=(n, 3))
    steps = 6 if precision == cg.MPCD_FP64 else 3
    runs = []
    for wait in (False, True):
        e = cg.Engine(sizes, precision=precision, seed=4, walls=walls, gravity=0.02 if walls else 0.0)
        e.set_fluid(pos, vel)
        e.prepare()
        if wait:
            for _ in range(steps):
                e.run(1)
                e.sync()
        else:
            e.run(steps)
        runs.append(e.fluid())
    d = runs[0][0] - runs[1][0]
    d -= np.round(d / np.array(sizes)) * np.array(sizes)
    d, w = np.abs(d).max(axis=1), np.abs(runs[0][1] - runs[1][1]).max(axis=1)
    if precision == cg.MPCD_FP64:
        assert d.max() < 1e-9 and w.max() < 1e-9
    else:
        assert (d < 1e-4).mean() > 0.999 and (w < 1e-3).mean() > 0.99
