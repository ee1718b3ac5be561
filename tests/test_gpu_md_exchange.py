"""The grid MD kernels (double-float: a thread per spring pair, lanes per bead
slot; the pair kernels) and their exchange of positions between tiles (tagged packets, no grid
barrier) on spring networks that the shipped objects do not make: one-sided
lists (a tile that reads another without being read), long lists (a tile of
their own; helper slots in short and long runs), and all tile widths.

Reference: the same velocity Verlet (src/libcilia/mdobject.cpp:36-72) in numpy
float64.  Every bead is alone in its collision cell, so the collision leaves
its velocity as it is.  Tolerance: the double-float arithmetic's 1e-10 of the
parity tests (positions of order 10, about 48 significand bits)."""
import ctypes

import numpy as np
import pytest

import cilia_gpu as cg

pytestmark = pytest.mark.gpu

L, TSTEP, SUB = 48, 0.1, 0.002


def lattice():
    g = 5.0 + 6.0 * np.arange(7)
    x, y, z = np.meshgrid(g, g, g, indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)


def network(kind, rng):
    """(target, other) lists of one-sided springs over 343 beads."""
    n = 343
    if kind == "oneway":  # bead i pulled by i + 60: every reader is unread
        t = np.arange(n - 60)
        return t, t + 60
    if kind == "random":  # sparse random reads, few of them answered
        return rng.integers(0, n, 600), rng.integers(0, n, 600)
    # "hub": bead 100 reads 250 others (a long run), bead 7 reads 40 (a short run)
    t = np.concatenate([np.full(250, 100), np.full(40, 7), np.arange(200, 300)])
    o = np.concatenate([rng.choice(n, 250, replace=False), rng.choice(n, 40, replace=False), np.full(100, 100)])
    return t, o


def verlet(pos, vel, t, o, rest, k, nsub, dt):
    def force(x):
        d = x[t] - x[o]
        r = np.sqrt((d * d).sum(axis=1))
        f = (-2.0 * k * (1.0 - rest / r))[:, None] * d
        out = np.zeros_like(x)
        np.add.at(out, t, f)
        return out

    x, v = pos.copy(), vel.copy()
    f = force(x)
    v += f * dt / 2
    x += v * dt
    f = force(x)
    for _ in range(1, nsub):
        v += f * dt
        x += v * dt
        f = force(x)
    return x, v + f * dt / 2


def run_network(kind, arith, min_tile):
    rng = np.random.default_rng(5)
    pos = lattice() + rng.uniform(-0.3, 0.3, (343, 3))
    vel = rng.normal(0, 0.2, (343, 3))
    t, o = network(kind, rng)
    keep = t != o
    t, o = t[keep].astype(np.int32), o[keep].astype(np.int32)
    d = np.sqrt(((pos[t] - pos[o]) ** 2).sum(axis=1))
    rest, k = d * rng.uniform(0.97, 1.03, len(t)), rng.uniform(0.5, 3.0, len(t))
    e = cg.Engine(L, tstep=TSTEP, ststep=SUB, precision=cg.MPCD_FP64, md_split=arith)
    e.set_fluid(np.array([[1.5, 1.5, 1.5]]), np.zeros((1, 3)))
    e.set_beads(pos, vel)
    ip, dp = ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double)
    z = np.zeros(len(t), dtype=np.int32)
    rc = cg.lib().mpcd_set_springs(e.handle, len(t), t.ctypes.data_as(ip), o.ctypes.data_as(ip), z.ctypes.data_as(ip),
                                   z.ctypes.data_as(ip), rest.ctypes.data_as(dp), k.ctypes.data_as(dp))
    assert rc == 0
    lay = e.md_layout()
    assert lay["arith"] == arith and lay["ntiles"] > 1 and lay["tile"] >= min_tile
    for _ in range(2):
        e.run(1)
        pos, vel = verlet(pos, vel, t, o, rest, k, 50, SUB)
    x, v = e.beads(343)
    assert np.abs(x - pos).max() < 1e-10
    assert np.abs(v - vel).max() < 1e-8


@pytest.mark.parametrize("min_tile", [0, 128, 256])
@pytest.mark.parametrize("kind", ["oneway", "random", "hub"])
@pytest.mark.parametrize("slots", [False, True])
def test_one_sided_networks_match_float64(kind, min_tile, slots, monkeypatch):
    if slots:
        monkeypatch.setenv("MPCD_MD_SLOTS", "1")
    if min_tile:
        monkeypatch.setenv("MPCD_MD_MIN_TILE", str(min_tile))
    run_network(kind, cg.MD_DF, min_tile)


@pytest.mark.parametrize("min_tile", [0, 128, 256])
@pytest.mark.parametrize("kind", ["oneway", "random", "hub"])
@pytest.mark.parametrize("arith", [cg.MD_PAIR, cg.MD_PAIR_DF])
def test_pair_kernel_on_one_sided_networks(kind, min_tile, arith, monkeypatch):
    """One warp waits for the other tiles while the rest evaluate: tiles that
    reach no other tile, many, or a hub."""
    if min_tile:
        monkeypatch.setenv("MPCD_MD_MIN_TILE", str(min_tile))
    run_network(kind, arith, min_tile)
