"""The workloads whose time is followed, through the package's public entry
points: `listed()` names them, `draw(rng)` gives more of the same ranges,
`prepare` makes what a program has in hand before the call, `run` is one pass,
`work` the bytes and operations it cannot do without, `exact` its result in
64 bits without this repository's code.

Families (sizes from the tests, the benchmark and the shipped configurations):
  fluid    a plain float64 box (Engine): `steps` MPC steps, then the fluid read
           back as positions and velocities; with walls, a body-force channel
  split    one split-precision step on the caller's own device arrays
           (mpcd_fluid_step_noalloc)
  swimmer  a ciliated sphere in a fluid (Sim): `steps` MPC steps of 50 MD
           substeps, then what a measuring interval reads: the beads, and in
           float64 also the fluid
  batch    an ensemble of uneven swimmer boxes (Batch): `steps` steps of all of
           them, then every replica's beads
The float32 passes are short: the order of float additions differs from run to
run, and over many steps single particles end up in other cells.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-ciliated-microswimmers_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cilia_gpu as cg  # noqa: E402
import simcfg  # noqa: E402

H = 0.1         # MPC time step of every shipped configuration
SUBSTEP = 0.002  # MD step: 50 substeps
DENSITY = 10    # fluid particles per cell
NOALLOC_CELLS = 65536  # the largest box of the allocation-free step
GRAVITY = 0.02  # body force of the channel


def listed():
    return [
        # one step of the smallest box and a look at it: launch and call latency
        dict(name="box8_f64", family="fluid", lx=8, ly=8, lz=8, walls=0, steps=1),
        # the plain 32^3 fluid of the benchmark over a measuring interval
        dict(name="plain32_f64", family="fluid", lx=32, ly=32, lz=32, walls=0, steps=10),
        # Poiseuille channel between no-slip walls, ragged edges
        dict(name="channel_f64", family="fluid", lx=24, ly=21, lz=37, walls=1, steps=8),
        # a box of several million particles, uneven edges
        dict(name="fluid5m_f64", family="fluid", lx=80, ly=71, lz=89, walls=0, steps=6),
        # the allocation-free step: a small ragged box, and the largest it takes
        dict(name="split_small_f32", family="split", lx=11, ly=9, lz=13),
        dict(name="split_large_f32", family="split", lx=39, ly=40, lz=42),
        # a small swimmer as in the parity tests: MD latency
        dict(name="swimmer10_f64", family="swimmer", l=10, radius=2.5, cilia=4, rod=10, f32=0, ieee=0, steps=5),
        # the benchmark's headline: 64^3, 100 cilia; and with IEEE float64 MD
        dict(name="swimmer64_f64", family="swimmer", l=64, radius=8.0, cilia=100, rod=15, f32=0, ieee=0, steps=20),
        dict(name="swimmer64_ieee", family="swimmer", l=64, radius=8.0, cilia=100, rod=15, f32=0, ieee=1, steps=10),
        # the same swimmer and the large one in split precision
        dict(name="swimmer64_f32", family="swimmer", l=64, radius=8.0, cilia=100, rod=15, f32=1, ieee=0, steps=2),
        dict(name="swimmer128_f32", family="swimmer", l=128, radius=16.0, cilia=400, rod=20, f32=1, ieee=0, steps=1),
        # uneven swimmer boxes advanced together
        dict(name="ensemble12_f32", family="batch", replicas=12, specs=11, steps=2),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["fluid", "fluid", "split", "swimmer", "swimmer", "batch"])
    if family == "fluid":
        walls = int(rng.random() < 0.3)
        lx, ly, lz = (_edge(rng, 6, 80) for _ in range(3))
        return dict(family="fluid", lx=lx, ly=ly, lz=lz, walls=walls, steps=rng.randint(1, 8))
    if family == "split":
        top = NOALLOC_CELLS
        lx, ly = _edge(rng, 5, 48), _edge(rng, 5, 48)
        return dict(family="split", lx=lx, ly=ly, lz=_edge(rng, 5, min(48, top // (lx * ly))))
    if family == "swimmer":
        f32 = int(rng.random() < 0.5)
        l = _edge(rng, 10, 72)
        radius = round(min(8.0, l / 4.0), 2)
        return dict(family="swimmer", l=l, radius=radius, cilia=rng.randint(2, max(3, int(10 * radius))),
                    rod=rng.randint(8, 15), f32=f32, ieee=0 if f32 else int(rng.random() < 0.3),
                    steps=2 if f32 else rng.randint(2, 15))
    return dict(family="batch", replicas=rng.randint(3, 12), specs=rng.randint(20, 10 ** 6), steps=2)


# ------------------------------------------------------------------ inputs --

def _fluid(sizes, seed, top=None):
    """Uniform positions and Maxwell velocities (kT = 1, no drift), float64 on
    the GPU; `top`: the highest z (a channel's upper wall)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n = DENSITY * sizes[0] * sizes[1] * sizes[2]
    span = torch.tensor([sizes[0], sizes[1], sizes[2] if top is None else top], dtype=torch.float64, device="cuda")
    pos = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) * span
    vel = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel - vel.mean(dim=0)


def _sizes(case):
    return case["lx"], case["ly"], case["lz"]


def _run_seed(seed):
    return int(seed) % 1000003 + 1


def _shifts(seed, n):
    return np.random.default_rng(int(seed) + 7).uniform(0.01, 0.99, (n, 3))


def _split_inputs(case, seed):
    """Particles in the split layout: {offset x, y, z, cell bits}, {v, 0}."""
    pos, vel = _fluid(_sizes(case), seed)
    cell = pos.floor()
    off = (pos - cell).float().clamp(max=1.0 - 2.0 ** -24)
    c = cell.to(torch.int32)
    bits = c[:, 0] | (c[:, 1] << 10) | (c[:, 2] << 20)
    p = torch.cat([off, bits.view(torch.float32)[:, None]], dim=1).contiguous()
    v = torch.cat([vel.float(), torch.zeros_like(off[:, :1])], dim=1).contiguous()
    return p, v


def _specs(case):
    """Uneven boxes as a server holds them: edges of the ensemble workload,
    sphere radius min(8, L / 4), up to ten cilia per unit of radius."""
    rng = np.random.default_rng(case["specs"])
    specs = []
    for k in range(case["replicas"]):
        l = int(rng.choice((16, 24, 32, 40, 48)))
        radius = min(8.0, l / 4.0)
        specs.append(dict(L=l, radius=radius, n_cilia=int(rng.integers(0, int(10 * radius) + 1)),
                          rodlength=int(rng.integers(10, 16)), seed=1000 * case["specs"] % 999983 + k + 1))
    return specs


def prepare(case, seed):
    family = case["family"]
    if family == "fluid":
        sizes = _sizes(case)
        top = sizes[2] - 1 if case["walls"] else None
        pos, vel = (a.cpu().numpy() for a in _fluid(sizes, seed, top))
        e = cg.Engine(sizes, tstep=H, ststep=SUBSTEP, seed=_run_seed(seed), walls=case["walls"],
                      gravity=GRAVITY if case["walls"] else 0.0)
        e.set_fluid(pos, vel)
        e.prepare()
        e.sync()
        return dict(case=case, engine=e, out=(pos, vel))  # the arrays are reused for the read-back
    if family == "split":
        p, v = _split_inputs(case, seed)
        return dict(case=case, p=p, v=v, n=len(p), sizes=(ctypes.c_int * 3)(*_sizes(case)), shifts=_shifts(seed, 64),
                    step=0, seed=_run_seed(seed), diss=ctypes.c_double(0.0))
    if family == "swimmer":
        l = case["l"]
        text = simcfg.dumps(simcfg.swimmer_config(l, radius=case["radius"], n_cilia=case["cilia"],
                                                  rodlength=case["rod"], seed=int(seed) % 1000003, ststep=SUBSTEP))
        s = cg.Sim(text, precision=cg.MPCD_FP32 if case["f32"] else cg.MPCD_FP64, seed=_run_seed(seed),
                   ststep=SUBSTEP, create_fluid=False, md_arith=cg.MD_PAIR if case["ieee"] else cg.MD_AUTO)
        pos, vel = (a.cpu().numpy() for a in _fluid((l, l, l), seed))
        s.engine.set_fluid(pos, vel)
        s.engine.prepare()
        s.engine.sync()
        return dict(case=case, sim=s, out=None if case["f32"] else (pos, vel))
    specs = _specs(case)
    b = cg.Batch.for_specs(specs)
    b.set_md_layout(1, 512)
    ids = []
    for k, sp in enumerate(specs):
        text = simcfg.dumps(simcfg.swimmer_config(sp["L"], radius=sp["radius"], n_cilia=sp["n_cilia"],
                                                  rodlength=sp["rodlength"], seed=sp["seed"]))
        r = b.add_cfg(text, seed=_run_seed(seed) + k, ststep=SUBSTEP, create_fluid=False)
        pos, vel = _fluid((sp["L"],) * 3, int(seed) + 1000 * (k + 1))
        b.set_fluid(r, pos.cpu().numpy(), vel.cpu().numpy())
        b.admit(r)
        b.set_steps(r, 10 ** 9)
        ids.append((r, 643 + 3 * sp["n_cilia"] * sp["rodlength"]))
    b.sync()
    return dict(case=case, batch=b, ids=ids)


# -------------------------------------------------------------------- pass --

def run(state):
    case = state["case"]
    family = case["family"]
    if family == "fluid":
        e = state["engine"]
        e.run(case["steps"])
        pos, vel = e.fluid(out=state["out"])
        return dict(pos=pos, vel=vel)
    if family == "split":
        k = state["step"]
        a = state["shifts"]
        dp = ctypes.POINTER(ctypes.c_double)
        cur, nxt = a[k % len(a)], a[(k + 1) % len(a)]
        rc = cg.lib().mpcd_fluid_step_noalloc(
            state["sizes"], state["n"], ctypes.c_void_p(state["p"].data_ptr()), ctypes.c_void_p(state["v"].data_ptr()),
            H, cur.ctypes.data_as(dp), nxt.ctypes.data_as(dp), state["seed"], k + 1, ctypes.byref(state["diss"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("mpcd_fluid_step_noalloc: %d" % rc)
        state["step"] = k + 1
        return dict(pos=state["p"], vel=state["v"])
    if family == "swimmer":
        s = state["sim"]
        s.engine.run(case["steps"])
        bp, bv = s.beads()
        if case["f32"]:  # float32 split: the state's own precision
            return dict(bead_pos=bp.astype(np.float32), bead_vel=bv.astype(np.float32))
        pos, vel = s.engine.fluid(out=state["out"])
        return dict(bead_pos=bp, bead_vel=bv, pos=pos, vel=vel)
    b = state["batch"]
    b.run(case["steps"])
    out = []
    for r, nb in state["ids"]:
        out.append(np.stack(b.beads(r, nb)).astype(np.float32))  # the swimmer's state: positions, velocities
    return out


# -------------------------------------------------------------------- work --

def _fluid_work(n, steps, f32):
    """Every step has to read and write the particles' positions and
    velocities (the state does not fit into on-chip memory); per particle the
    3 x 3 collision map, the streaming and the cell sums."""
    return 2 * 6 * (4 if f32 else 8) * n * steps, 50.0 * n * steps


def _md_work(nb, nspring, steps):
    """Per substep every spring's difference, distance and force (about 30
    operations) and every bead's update; the beads stay on the chip."""
    sub = int((H + 1e-8) / SUBSTEP)
    return 2 * 48 * nb * steps, (30.0 * nspring + 20.0 * nb) * (sub + 1) * steps


def _swimmer_size(radius_cilia, rod):
    """Beads and one-sided springs of a 643-bead sphere with its cilia (about
    eight springs a bead)."""
    nb = 643 + 3 * radius_cilia * rod
    return nb, 8 * nb


def work(case):
    family = case["family"]
    if family == "split":
        n = DENSITY * case["lx"] * case["ly"] * case["lz"]
        by, fl = _fluid_work(n, 1, True)
        return dict(bytes=by, flops=fl)
    if family == "fluid":
        n = DENSITY * case["lx"] * case["ly"] * case["lz"]
        by, fl = _fluid_work(n, case["steps"], False)
        return dict(bytes=by + 48 * n, flops=fl)
    if family == "swimmer":
        n = DENSITY * case["l"] ** 3
        by, fl = _fluid_work(n, case["steps"], case["f32"])
        nb, ns = _swimmer_size(case["cilia"], case["rod"])
        mb, mf = _md_work(nb, ns, case["steps"])
        return dict(bytes=by + mb + (0 if case["f32"] else 48 * n), flops=fl + mf)
    by = fl = 0.0
    for sp in _specs(case):
        b1, f1 = _fluid_work(DENSITY * sp["L"] ** 3, case["steps"], True)
        nb, ns = _swimmer_size(sp["n_cilia"], sp["rodlength"])
        b2, f2 = _md_work(nb, ns, case["steps"])
        by, fl = by + b1 + b2, fl + f1 + f2
    return dict(bytes=by, flops=fl)


# ------------------------------------------------------------------- exact --
# The fluid step in 64 bits: SRD collision with the Maxwell-Boltzmann-scaling
# thermostat, random shift, streaming, walls.  The draws are those of the
# documented generator (Philox4x32-10 of Salmon et al., SC'11; Marsaglia and
# Tsang's Gamma sampler), whose uniforms have 24 bits.

_M32 = 0xFFFFFFFF
COS_A, SIN_A = -0.6427876, 0.76604444  # the rotation constants of the method


def _philox(index, step, stream, rnd, seed):
    c0 = index.to(torch.int64)
    full = lambda v: torch.full_like(c0, v & _M32)  # noqa: E731
    c1, c2, c3 = full(step), full((step >> 32) ^ (stream << 24)), full(rnd)
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        h0, l0, h1, l1 = (p0 >> 32) & _M32, p0 & _M32, (p1 >> 32) & _M32, p1 & _M32
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


def _u24(u):
    return (((u >> 8).float() + 0.5) * (1.0 / 16777216.0)).double()


def _u32(u):
    return (u.double() + 0.5) / 4294967296.0


def _gamma(num, cells, step, seed):
    """Gamma(3 (num - 1) / 2) of the given cells."""
    d = 1.5 * num.double() - 11.0 / 6.0
    c = 1.0 / (3.0 * d.sqrt())
    out = torch.zeros_like(d)
    todo = torch.arange(len(d), device=d.device)
    for rnd in range(64):
        if len(todo) == 0:
            break
        r = _philox(cells[todo], step, 2, 16 + rnd, seed)
        u1, u2, u = _u24(r[0]), _u24(r[1]), _u24(r[2])
        x = (-2.0 * u1.log()).sqrt() * torch.cos(2.0 * math.pi * u2)
        dd = d[todo]
        v = (1.0 + c[todo] * x) ** 3
        vs = v.clamp(min=1e-300)
        ok = (v > 0) & ((u < 1.0 - 0.0331 * x ** 4) | (u.log() < 0.5 * x * x + dd * (1.0 - vs + vs.log())))
        out[todo[ok]] = (dd * v)[ok]
        todo = todo[~ok]
    return out


def _virtual(cells, dm, step, seed):
    r = _philox(cells, step, 3, 0, seed)
    r1, r3 = (-2.0 * _u32(r[0]).log()).sqrt(), (-2.0 * _u32(r[2]).log()).sqrt()
    t, w = 2.0 * math.pi * _u32(r[1]), 2.0 * math.pi * _u32(r[3])
    return dm.double().sqrt()[:, None] * torch.stack([r1 * torch.cos(t), r1 * torch.sin(t), r3 * torch.cos(w)], dim=1)


def _collide(v, cid, sizes, step, seed, walls):
    nc = sizes[0] * sizes[1] * sizes[2]
    count = torch.bincount(cid, minlength=nc)
    mom = torch.zeros(nc, 3, dtype=torch.float64, device=v.device).index_add_(0, cid, v)
    kin = torch.zeros(nc, dtype=torch.float64, device=v.device).index_add_(0, cid, (v * v).sum(dim=1))
    cells = torch.arange(nc, device=v.device)
    num = count.clone()
    used = count > 0
    if walls:  # wall layers are filled up to the mean density with particles at rest on average
        layer = sizes[0] * sizes[1]
        low = ((cells < layer) | (cells > layer * (sizes[2] - 1))) & (num < DENSITY) & used
        dm = (DENSITY - num)[low]
        p = _virtual(cells[low], dm, step, seed)
        mom[low] += p
        kin[low] += (p * p).sum(dim=1) / dm
        num[low] += dm
    u = mom / num.clamp(min=1).double()[:, None]
    erel = kin - (u * mom).sum(dim=1)
    sc = torch.ones_like(erel)
    hot = used & (erel > 0) & (num > 1)
    sc[hot] = (2.0 * _gamma(num[hot], cells[hot], step, seed) / erel[hot]).sqrt()
    r = _philox(cells, step, 2, 0, seed)
    ct, phi = 2.0 * _u24(r[1]) - 1.0, 2.0 * math.pi * _u24(r[0])
    st = (1.0 - ct * ct).clamp(min=0.0).sqrt()
    ax = torch.stack([st * torch.cos(phi), st * torch.sin(phi), ct], dim=1)[cid]
    w = v - u[cid]
    rot = COS_A * w + SIN_A * torch.linalg.cross(ax, w) + (1.0 - COS_A) * (ax * w).sum(dim=1, keepdim=True) * ax
    return u[cid] + sc[cid][:, None] * rot


def _cells(ijk, sizes):
    return ijk[:, 0] + sizes[0] * (ijk[:, 1] + sizes[1] * ijk[:, 2])


def exact(case, seed):
    if case["family"] == "split":
        # the offset and cell of a particle on a cell's face are not unique: velocities only
        p, v = _split_inputs(case, seed)
        bits = p[:, 3].contiguous().view(torch.int32).long()
        ijk = torch.stack([bits & 1023, (bits >> 10) & 1023, (bits >> 20) & 1023], dim=1)
        sizes = _sizes(case)
        ta = torch.tensor(1.0 - _shifts(seed, 64)[0], device="cuda").float()
        span = torch.tensor(sizes, device="cuda")
        cid = _cells((ijk + (p[:, :3] >= ta)) % span, sizes)
        w = _collide(v[:, :3].double(), cid, sizes, 1, _run_seed(seed), False)
        return dict(pos=None, vel=torch.cat([w, torch.zeros_like(w[:, :1])], dim=1))
    if case["family"] != "fluid":
        # a swimmer's beads and springs come from the object model (mesh,
        # attachment, beat), which is this repository's own
        return None
    sizes, walls, rs = _sizes(case), bool(case["walls"]), _run_seed(seed)
    top = sizes[2] - 1.0
    x, v = _fluid(sizes, seed, top if walls else None)
    span = torch.tensor(sizes, dtype=torch.float64, device="cuda")
    zero = torch.zeros(1, dtype=torch.int64, device="cuda")

    def shift(step):
        return torch.stack([_u32(c)[0] for c in _philox(zero, step, 1, 0, rs)[:3]])

    a = shift(0)
    for step in range(1, case["steps"] + 1):
        cid = _cells((x + a).floor().long() % span.long(), sizes)
        v = _collide(v, cid, sizes, step, rs, walls)
        x = x + v * H
        if walls:
            for hit, plane in ((x[:, 2] > top, top), (x[:, 2] < 0, 0.0)):
                t = ((x[:, 2] - plane) / v[:, 2])[:, None]
                v = torch.where(hit[:, None], -v, v)
                x = torch.where(hit[:, None], x + 2.0 * t * v, x)
            v = v + torch.tensor([GRAVITY * H, 0.0, 0.0], dtype=torch.float64, device="cuda")
        x = x - (x / span).floor() * span
        a = shift(step)
    return dict(pos=x, vel=v)
