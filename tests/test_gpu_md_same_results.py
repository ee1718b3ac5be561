"""The two double-float MD kernels give the same results bit for bit: a thread
per spring pair (md_entries.cu) adds every bead's forces in the order in which
the lanes and helper slots of the slot kernel (md_df.cu) add them.  Equality is
the bound: the springs are stiff, so a rounding done differently grows by orders
of magnitude over a run."""
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
