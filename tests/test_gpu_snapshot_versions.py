"""Float64 snapshots of version 1 (in-cell offsets as float64) are still read;
version 2 holds them as integers in units of 2^-60.  A version 2 snapshot
rewritten as version 1 restores the same fluid: velocities bit for bit,
positions to the rounding of an offset to float64 (2^-54) and the addition of
the cell."""
import struct

import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu


def test_version_1_offsets_are_converted():
    sizes = (6, 5, 7)
    n = 2100
    rng = np.random.default_rng(2)
    e = cg.Engine(sizes, seed=3)
    e.set_fluid(rng.uniform(0, 1, (n, 3)) * sizes, rng.normal(size=(n, 3)))
    e.run(3)
    pos, vel = e.fluid()
    snap = bytearray(e.snapshot())
    assert struct.unpack_from("<i", snap, 8) == (2,)
    head = len(snap) - 56 * n  # a plain fluid: ids, cells, offsets, velocities end the snapshot
    at = head + 8 * n
    off = np.frombuffer(snap, np.uint64, 3 * n, at)
    assert off.max() < 1 << 60
    old = bytearray(snap)
    struct.pack_into("<i", old, 8, 1)
    old[at:at + 24 * n] = (off.astype(np.float64) / 2.0 ** 60).clip(0, 1 - 2.0 ** -53).tobytes()
    for data, tol in ((snap, 0.0), (old, 2.0 ** -50)):
        f = cg.Engine(sizes, seed=3)
        f.restore(bytes(data))
        p, v = f.fluid()
        assert np.array_equal(v, vel)
        assert np.abs(p - pos).max() <= tol
    a, b = cg.Engine(sizes, seed=3), cg.Engine(sizes, seed=3)
    a.restore(bytes(snap))
    b.restore(bytes(old))
    a.run(2)
    b.run(2)
    d = a.fluid()[0] - b.fluid()[0]
    assert np.abs(d - np.round(d / sizes) * sizes).max() < 1e-9
