"""The fluid's read-back: one scatter launch below 2^20 particles, gathered and
copied in parts from there on.  After an upload and the first sort by cell the
read-back gives the input in the input's order: velocities bit for bit (split
precision: their float32 values), positions to the rounding of the in-cell
offsets (2^-60 and the addition of the cell; 2^-24)."""
import ctypes

import numpy as np
import pytest

import cilia_gpu as cg
import simcfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cg.MPCD_FP64, cg.MPCD_FP32])
@pytest.mark.parametrize("n", [1, 33, 5000, (1 << 20) - 1, 1 << 20, (1 << 20) + 77])
def test_read_back_order(n, precision):
    rng = np.random.default_rng(n)
    sizes = (3, 4, 5) if n < 1000 else ((8, 9, 10) if n < 10000 else (47, 48, 49))
    pos = rng.uniform(0, 1, (n, 3)) * np.array(sizes)
    vel = rng.normal(size=(n, 3))
    e = cg.Engine(sizes, precision=precision, seed=1)
    e.set_fluid(pos, vel)
    e.prepare()
    got, gotv = e.fluid()
    if precision == cg.MPCD_FP64:
        assert np.array_equal(gotv, vel)
        assert np.abs(got - pos).max() <= 2.0 ** -47  # one rounding of a position below 64
    else:
        assert np.array_equal(gotv, vel.astype(np.float32).astype(np.float64))
        d = got - pos  # an offset that rounds to 1 is kept just below
        assert np.abs(d - np.round(d / np.array(sizes)) * np.array(sizes)).max() <= 2.0 ** -23
    # either array alone
    dp = ctypes.POINTER(ctypes.c_double)
    for q, want in enumerate((got, gotv)):
        buf = np.full((n, 3), np.nan)
        args = [None, None]
        args[q] = buf.ctypes.data_as(dp)
        assert cg.lib().mpcd_get_fluid(e._h, n, *args) == 0
        assert np.array_equal(buf, want)


@pytest.mark.parametrize("precision, arith", [(cg.MPCD_FP64, cg.MD_AUTO), (cg.MPCD_FP64, cg.MD_PAIR), (cg.MPCD_FP32, cg.MD_AUTO)])
@pytest.mark.parametrize("cilia", [0, 1, 10])
def test_beads_come_back_in_their_order(cilia, precision, arith):
    """Right after the upload the beads are those of the configuration, bit for bit."""
    s = cg.Sim(simcfg.dumps(simcfg.swimmer_config(16, radius=4.0, n_cilia=cilia, rodlength=8, seed=3, ststep=0.002)),
               precision=precision, seed=3, ststep=0.002, create_fluid=False, md_arith=arith)
    before = s.beads()  # the host's description: not uploaded yet
    s.engine.prepare()
    after = s.beads()
    again = s.beads()
    for a, b, c in zip(before, after, again):
        assert a.shape == (s.nbeads, 3)
        assert np.array_equal(a, b) and np.array_equal(b, c)
    dp = ctypes.POINTER(ctypes.c_double)
    for q, want in enumerate(after):
        buf = np.full((s.nbeads, 3), np.nan)
        args = [None, None]
        args[q] = buf.ctypes.data_as(dp)
        assert cg.lib().mpcd_get_beads(s.engine._h, s.nbeads, *args) == 0
        assert np.array_equal(buf, want)
