"""The two double-float MD kernels give the same results bit for bit: a thread
per spring pair (md_entries.cu) adds every bead's forces in the order in which
the lanes and helper slots of the slot kernel (md_df.cu) add them.  Equality is
the bound: the springs are stiff, so a rounding done differently grows by orders
of magnitude over a run."""
import ctypes

import numpy as np
import pytest

import cilia_gpu as cg
import simcfg

pytestmark = pytest.mark.gpu


def one_step(precision, size, min_tile, slots, monkeypatch):
    """Beads after one MPC step (50 substeps) from rest."""
    box, radius, cilia, rod = size
    monkeypatch.setenv("MPCD_MD_SLOTS", str(int(slots)))
    monkeypatch.setenv("MPCD_MD_MIN_TILE", str(min_tile))
    text = simcfg.dumps(simcfg.swimmer_config(box, radius=radius, n_cilia=cilia, rodlength=rod, seed=7, ststep=0.002))
    s = cg.Sim(text, precision=precision, seed=11, ststep=0.002, create_fluid=False)
    s.engine.set_fluid(np.array([[0.5, 0.5, 0.5]]), np.zeros((1, 3)))
    s.engine.run(1)
    layout = s.engine.md_layout()
    return s.beads(), layout


# tiles of 8, 4 and 2 lanes per slot; a sphere alone (its centre in a tile of
# its own, beads with helper slots), with few and with many cilia
@pytest.mark.parametrize("min_tile", [0, 128, 256])
@pytest.mark.parametrize("size", [(24, 6.0, 0, 10), (10, 2.5, 4, 10), (24, 6.0, 33, 15)])
@pytest.mark.parametrize("precision", [cg.MPCD_FP64, cg.MPCD_FP32])
def test_pairs_and_slots_agree_bit_for_bit(precision, size, min_tile, monkeypatch):
    (pos, vel), pairs = one_step(precision, size, min_tile, False, monkeypatch)
    (spos, svel), slots = one_step(precision, size, min_tile, True, monkeypatch)
    assert pairs["ntiles"] != slots["ntiles"]  # two layouts
    assert np.abs(vel).max() > 0
    assert np.array_equal(pos, spos) and np.array_equal(vel, svel)


# a bead with a list of its own tile: slots in order (up to 8 of 15 springs), by a
# warp's tree, and with more slots than the warp has lanes
@pytest.mark.parametrize("springs", [65, 70, 120, 121, 480, 481, 1000])
@pytest.mark.parametrize("precision", [cg.MPCD_FP64, cg.MPCD_FP32])
@pytest.mark.parametrize("min_tile", [0, 128])
def test_long_lists_agree_bit_for_bit(springs, precision, min_tile, monkeypatch):
    rng = np.random.default_rng(springs)
    nb = springs + 40
    pos = rng.uniform(4, 28, (nb, 3))
    hub = 17
    other = np.setdiff1d(rng.permutation(nb), [hub])[:springs]
    t = np.concatenate([np.full(springs, hub), other]).astype(np.int32)
    o = np.concatenate([other, np.full(springs, hub)]).astype(np.int32)
    order = rng.permutation(2 * springs)
    rest = np.tile(np.sqrt(((pos[hub] - pos[other]) ** 2).sum(axis=1)) * rng.uniform(0.9, 1.1, springs), 2)
    k = np.tile(rng.uniform(0.5, 3.0, springs), 2)
    t, o, rest, k = t[order], o[order], rest[order], k[order]
    ip, dp = ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double)
    z = np.zeros(len(t), dtype=np.int32)
    got = []
    for slots in ("0", "1"):
        monkeypatch.setenv("MPCD_MD_SLOTS", slots)
        monkeypatch.setenv("MPCD_MD_MIN_TILE", str(min_tile))
        e = cg.Engine(32, tstep=0.1, ststep=0.002, precision=precision)
        e.set_fluid(np.array([[0.5, 0.5, 0.5]]), np.zeros((1, 3)))
        e.set_beads(pos, np.zeros((nb, 3)))
        assert cg.lib().mpcd_set_springs(e.handle, len(t), t.ctypes.data_as(ip), o.ctypes.data_as(ip), z.ctypes.data_as(ip),
                                         z.ctypes.data_as(ip), rest.ctypes.data_as(dp), k.ctypes.data_as(dp)) == 0
        e.run(1)
        got.append(e.beads(nb))
        e.close()
    assert np.abs(got[0][1][hub]).max() > 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


def test_a_bead_set_beyond_the_pair_layout_runs_on_the_slot_kernel(monkeypatch):
    """Six beads with 200 springs each: four get a tile of their own, the others'
    slots are more than the pair kernel adds in order."""
    rng = np.random.default_rng(9)
    nb, hubs, springs = 1300, 6, 200
    pos = rng.uniform(4, 28, (nb, 3))
    t, o = [], []
    for h in range(hubs):
        other = hubs + h * springs + np.arange(springs)
        t += [np.full(springs, h), other]
        o += [other, np.full(springs, h)]
    t, o = np.concatenate(t).astype(np.int32), np.concatenate(o).astype(np.int32)
    rest = np.sqrt(((pos[t] - pos[o]) ** 2).sum(axis=1)) * 1.02
    k = np.full(len(t), 1.5)
    ip, dp = ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double)
    z = np.zeros(len(t), dtype=np.int32)
    got = []
    for slots in ("0", "1"):
        monkeypatch.setenv("MPCD_MD_SLOTS", slots)
        e = cg.Engine(32, tstep=0.1, ststep=0.002)
        e.set_fluid(np.array([[0.5, 0.5, 0.5]]), np.zeros((1, 3)))
        e.set_beads(pos, np.zeros((nb, 3)))
        assert cg.lib().mpcd_set_springs(e.handle, len(t), t.ctypes.data_as(ip), o.ctypes.data_as(ip), z.ctypes.data_as(ip),
                                         z.ctypes.data_as(ip), rest.ctypes.data_as(dp), k.ctypes.data_as(dp)) == 0
        e.run(1)
        got.append((e.beads(nb), e.md_layout()))
        e.close()
    assert got[0][1] == got[1][1]  # one layout
    assert np.abs(got[0][0][1]).max() > 0
    assert np.array_equal(got[0][0][0], got[1][0][0]) and np.array_equal(got[0][0][1], got[1][0][1])
