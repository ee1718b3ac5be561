// MD substeps of one MPC step for the float64 path, in double-float
// arithmetic on the FP32 pipes.
//
// The general form of the double-float MD: every bead set whose layout fits the
// device runs here; those that fit the layout of md_entries.cu (a thread per
// spring pair, less than half the time on large swimmers) run there.
//
// Same integrator and forces as md_kernels.cu (velocity Verlet of
// src/libcilia/mdobject.cpp:36-72 inside the loop of src/simulation.cpp:217-265;
// springs of src/cilia.cpp:127-239, src/sphere.cpp:87-119, src/clami.cpp:188-198)
// on the same cooperative-grid tile layout (md_plan.cu: a CTA per tile, helper
// slots for long spring lists, halos), with eight lanes per slot (four for
// tiles over 64 slots).  The difference
// is the arithmetic: GB300 issues float64 at a small fraction of its float32
// rate, and the float64 MD kernel spent most of its time on the FP64 pipe.
// Here every bead's position and velocity live in registers as double-float
// pairs (about 48 significand bits) for the whole MPC step; spring forces,
// their sums and the Verlet updates are double-float operations built from
// float adds, multiplies and fused multiply-adds.  The state is read from and
// written back to the float64 arrays once per MPC step.  Rest lengths and
// spring constants come as float pairs prepared on the host.
//
// Each CTA keeps its tile's spring and bond tables in shared memory for the
// whole launch.  Positions are exchanged between tiles as tagged packets: a
// coordinate of a bead is one 16-byte packet {offset high, offset low, cell,
// tag} written by one 128-bit store into one of two global buffers, the tag
// naming the force evaluation it belongs to; a tile that needs the bead polls
// the packet itself until the tag is the one it waits for.  No barrier and no
// second read: data and flag arrive together, one way through L2.  The chain
// of a substep is what bounds the launch (a few thousand beads, 51 dependent
// evaluations; every pipe and DRAM are idle), so it is kept short: the lanes
// that sum a bead's force own its state (lane k its coordinate k), the lanes'
// partial forces are combined by a transposing exchange that leaves each
// coordinate with its owner, and a tile without helper slots needs two CTA
// barriers per substep.  Measured alone on swimmer64 (116 tiles, 51
// evaluations), against a grid barrier followed by copies of the halo: 168
// against 217 us in double-float, 148 against 203 with float springs; the
// 19 tiles of a 700-bead swimmer 158 against 192.
// The partial forces of a bead's helper slots are added in a fixed order: by
// one warp (lane-strided, then by a transposing tree) for long runs, in slot
// order for short ones.
//
// The cilia's rest lengths: the beat's target length of every bond is fixed
// during one MPC step's substeps (the midpoint moves after them), so it is
// computed once per launch in float64; the bending-rate limit that uses the
// current bond length runs in pairs at every refresh (every 0.01 time units).
#include <cstdlib>

#include "../../include/mpcd_gpu.h"
#include "df32.cuh"
#include "md_common.cuh"
#include "md_df_coord.cuh"
#include "md_packets.cuh"

namespace mpcd {

namespace {

// Tile-resident spring and bond tables in shared memory.
struct Tables {
  const uint32_t* code;  // other bead | kind << 16 | bond << 18
  const float2* rest;    // static rest length (kinds CONST, GUARDED)
  const float2* m2k;     // -2k
  const float2* nl;      // bonds: current rest length (newlength)
  const float2* dg;      // bonds: diagonal rest length sqrt(0.5^2 + 0.5 newlength)
};

// Force on staged bead `me` from springs [a, b) step LANES (indices local
// to the tile's table).  Per spring, with d = x_me - x_o and rest length b:
// fac = -2k (1 - b / |d|), F += fac d, all in pairs; components accumulate as
// compensated sums (h, l).  kFloat: the difference d is formed exactly as a
// pair and rounded to float, the rest of the spring in float (the split
// arithmetic of the float32 path); the sums stay compensated.
template <int LANES, bool kFloat>
__device__ __forceinline__ void springs_df(const Tables& tb, const float4* st, const float4 m0, const float4 m1, int a,
                                           int b, float& fxh, float& fxl, float& fyh, float& fyl, float& fzh,
                                           float& fzl) {
  for (int s = a; s < b; s += LANES) {
    const uint32_t code = tb.code[s];
    const int o = (int)(code & 0xffffu);
    const int kind = (int)((code >> 16) & 3u);
    const int lref = (int)(code >> 18);
    const float2 b2 = kind <= MPCD_SPRING_GUARDED ? tb.rest[s] : (kind == MPCD_SPRING_BOND ? tb.nl[lref] : tb.dg[lref]);
    const float2 k2 = tb.m2k[s];
    if constexpr (kFloat) {
      const float4 o0 = st[2 * o], o1 = st[2 * o + 1];
      const dfloat ex = coord_diff((float)(cell_x(m1) - cell_x(o1)), m0.x, o0.x, m0.w, o0.w);
      const dfloat ey = coord_diff((float)(cell_y(m1) - cell_y(o1)), m0.y, o0.y, m1.x, o1.x);
      const dfloat ez = coord_diff(__fsub_rn(m1.w, o1.w), m0.z, o0.z, m1.y, o1.y);
      const float dx = ex.h + ex.l, dy = ey.h + ey.l, dz = ez.h + ez.l;
      const float d2 = dx * dx + dy * dy + dz * dz;
      if (kind == MPCD_SPRING_GUARDED && d2 == 0.0f) continue;
      const float fac = k2.x * (1.0f - b2.x * rsqrtf(d2));
      fxh += fac * dx;
      fyh += fac * dy;
      fzh += fac * dz;
      continue;
    }
    const DfDiff d = df_diff(m0, m1, st[2 * o], st[2 * o + 1]);
    if (kind == MPCD_SPRING_GUARDED && d.d2.h == 0.0f) continue;  // vector-form spring: no force at zero distance
    const dfloat r = df_rsqrt(d.d2);
    // w = 1 - b r
    const dfloat u = df_two_prod(b2.x, r.h);
    const dfloat w = df_two_sum(1.0f, -u.h);
    const float wl = ((w.l - u.l) - b2.x * r.l) - b2.y * r.h;
    // fac = -2k w
    const dfloat f = df_two_prod(k2.x, w.h);
    const float fl = (f.l + k2.x * wl) + k2.y * w.h;
    const dfloat gx = df_two_prod(f.h, d.dx.h), gy = df_two_prod(f.h, d.dy.h), gz = df_two_prod(f.h, d.dz.h);
    df_acc(fxh, fxl, gx.h, (gx.l + f.h * d.dx.l) + fl * d.dx.h);
    df_acc(fyh, fyl, gy.h, (gy.l + f.h * d.dy.l) + fl * d.dy.h);
    df_acc(fzh, fzl, gz.h, (gz.l + f.h * d.dz.l) + fl * d.dz.h);
  }
}


// Coordinate k of a staged entry (two float4, md_df_coord.cuh): its words are
// the offset's high part k, low part 3 + k, and the cell (x and y as 16-bit
// halves of word 6, z as a float in word 7).
__device__ __forceinline__ void stage_coord(float4* e, int k, float h, float l, int c) {
  float* w = reinterpret_cast<float*>(e);
  w[k] = h;
  w[3 + k] = l;
  if (k < 2)
    reinterpret_cast<unsigned short*>(w + 6)[k] = (unsigned short)c;
  else
    w[7] = (float)c;
}

// shared-memory layout of one tile: two buffers of its own beads, its halo,
// the halo's slots and the tables
struct DfSmem {
  size_t st, halo, hslot, flag, code, rest, m2k, nl, ol, dg, tg, bd, part, total;
  __host__ __device__ DfSmem(int T, int hmax, int nsp, int nb) {
    size_t o = 0;
    auto take = [&](size_t bytes, size_t align) {
      o = (o + align - 1) / align * align;
      const size_t r = o;
      o += bytes;
      return r;
    };
    st = take(64 * (size_t)T, 16);
    halo = take(32 * (size_t)hmax, 16);
    hslot = take(4 * (size_t)hmax, 4);
    flag = take(4, 4);
    rest = take(8 * (size_t)nsp, 8);
    m2k = take(8 * (size_t)nsp, 8);
    nl = take(8 * (size_t)nb, 8);
    ol = take(8 * (size_t)nb, 8);
    dg = take(8 * (size_t)nb, 8);
    tg = take(8 * (size_t)nb, 8);
    bd = take(8 * (size_t)nb, 8);
    code = take(4 * (size_t)nsp, 4);
    part = take(24 * (size_t)T, 8);
    total = o;
  }
};

template <int LANES, bool kFloat, typename Bin>
__device__ void md_df_body(const MDState& m, const MDStepArgs& a, Bin bin) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int T = m.tile;
  const DfSmem L(T, m.hmax, m.df_nsp_max, m.df_nb_max);
  float4* own0 = reinterpret_cast<float4*>(smem + L.st);  // buffer b at own0 + 2 T b
  float4* halo = reinterpret_cast<float4*>(smem + L.halo);
  int* s_hslot = reinterpret_cast<int*>(smem + L.hslot);
  int* s_fail = reinterpret_cast<int*>(smem + L.flag);  // 1: a packet never came
  uint32_t* s_code = reinterpret_cast<uint32_t*>(smem + L.code);
  float2* s_rest = reinterpret_cast<float2*>(smem + L.rest);
  float2* s_m2k = reinterpret_cast<float2*>(smem + L.m2k);
  float2* s_nl = reinterpret_cast<float2*>(smem + L.nl);
  float2* s_ol = reinterpret_cast<float2*>(smem + L.ol);
  float2* s_dg = reinterpret_cast<float2*>(smem + L.dg);
  float2* s_tg = reinterpret_cast<float2*>(smem + L.tg);
  float2* s_bd = reinterpret_cast<float2*>(smem + L.bd);
  float2* part = reinterpret_cast<float2*>(smem + L.part);  // per slot: its lanes' force (three pairs)
  const Tables tb{s_code, s_rest, s_m2k, s_nl, s_dg};

  const int tile = blockIdx.x;
  const int base = tile * T;
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  // spring lanes: LANES per slot; springs [s0, sm) reach in-tile beads, [sm, s1) the halo
  const int q = tid / LANES, lane = tid % LANES;
  const int slot = base + q;
  const int S0 = m.sp_start[base];
  const int mv = m.moves[slot];
  const int me = mv >= 0 ? m.prim[slot] - base : 0;
  const int s0 = m.sp_start[slot] - S0, sm = m.sp_split[slot] - S0, s1 = m.sp_start[slot + 1] - S0;
  // the lanes of a primary slot own its bead: coordinate k belongs to lane
  // k mod LANES (with two lanes, x and z to lane 0)
  constexpr int NC = (3 + LANES - 1) / LANES;
  const bool prim = mv == 0 || mv == 1, moves = mv == 1;
  const bool helpers = m.tile_help[tile] != 0;
  // a primary with helpers and its helper slots form a run of 1 + nh slots;
  // runs longer than kTreeRun are summed by the primary's warp, shorter ones
  // by the owners
  constexpr int kTreeRun = 8;
  const int nh = prim ? m.nhelp[slot] : 0;
  const int h0 = m.halo_start[tile], hn0 = m.halo_start[tile + 1] - h0;
  const int c0 = m.tile_cil[tile], c1 = m.tile_cil[tile + 1];
  const int b0 = m.tile_b0[tile], nb = m.tile_nb[tile];
  const int nsp = m.sp_start[base + T] - S0;
  const dfloat dt{a.dt_pair.x, a.dt_pair.y}, dt2{a.dt2_pair.x, a.dt2_pair.y};

  // the halo's slots; every one must lie in the packet buffers
  if (tid == 0) *s_fail = hn0 > m.hmax;
  __syncthreads();
  for (int i = tid; i < hn0 && hn0 <= m.hmax; i += nthr) {
    const int g = m.halo[h0 + i];
    s_hslot[i] = g;
    if (g < 0 || g >= m.nslots) *s_fail = 1;
  }
  __syncthreads();
  const int hn = *s_fail ? 0 : hn0;  // no halo (and an error) for an inconsistent plan
  if (*s_fail && tid == 0) atomicOr(a.err, kErrLayout);
  __syncthreads();
  if (tid == 0) *s_fail = 0;
  // tile-resident tables
  for (int i = tid; i < nsp; i += nthr) {
    s_code[i] = __ldg(m.sp_code + S0 + i);
    s_rest[i] = __ldg(m.sp_rest2 + S0 + i);
    s_m2k[i] = __ldg(m.sp_m2k2 + S0 + i);
  }
  for (int i = tid; i < nb; i += nthr) {
    const dfloat n = df_from_double(m.newlen[b0 + i]), o = df_from_double(m.oldlen[b0 + i]);
    const dfloat g = df_from_double(m.diag[b0 + i]);
    s_nl[i] = make_float2(n.h, n.l);
    s_ol[i] = make_float2(o.h, o.l);
    s_dg[i] = make_float2(g.h, g.l);
  }
  // the beat's rest length of every refreshed bond for this step, and the bending limit
  {
    int off = 0;
    for (int c = c0; c < c1; ++c) {
      const CiliumDev cl = m.cil[c];
      const int nbnd = cl.len - cl.num_anker;
      const int w = tid - off;
      if (w >= 0 && w < nbnd) {
        const int i = cl.num_anker - 1 + w;
        const int k = cl.bond_base + i - b0;
        const dfloat t = df_from_double(cilium_target(cl, i, m.midpnt[c]));
        const dfloat bd = df_from_double(cl.bending);
        s_tg[k] = make_float2(t.h, t.l);
        s_bd[k] = make_float2(bd.h, bd.l);
      }
      off += nbnd;
    }
  }
  // the owned coordinates
  BeadCoord x[NC];
  dfloat v[NC], f[NC];
  double ke_coll = 0.0;
  {
    double X[3] = {0.0, 0.0, 0.0}, V[3] = {0.0, 0.0, 0.0};
    if (prim) {
      X[0] = m.x[0][slot];
      X[1] = m.y[0][slot];
      X[2] = m.z[0][slot];
      V[0] = m.vx[slot];
      V[1] = m.vy[slot];
      V[2] = m.vz[slot];
      if (a.collide && moves) {  // the beads' collision, folded in (every lane of the slot the same)
        const double ke = bin.collide(X[0], X[1], X[2], V[0], V[1], V[2]);
        if (lane == 0) ke_coll = ke;
      }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const int k = lane + j * LANES;
      x[j] = coord_from_double(k == 0 ? X[0] : (k == 1 ? X[1] : X[2]));
      v[j] = df_from_double(k == 0 ? V[0] : (k == 1 ? V[1] : V[2]));
      f[j] = {0.f, 0.f};
    }
  }
  if (a.collide) {  // the dissipated-energy bookkeeping of the collided beads
    const double tot = block_sum_f64(ke_coll);
    if (tid == 0 && tot != 0.0) atomicAdd(a.diss, -tot);
  }
  bool refreshed = false;

  // own beads of evaluation e: into shared memory (buffer e & 1) and, as
  // packets, into global buffer e & 1
  auto publish = [&](int e) {
    if (prim) {
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int k = lane + j * LANES;
        if (k < 3) {
          const Packet pk{__float_as_uint(x[j].o.h), __float_as_uint(x[j].o.l), (uint32_t)x[j].c, a.tag0 + (uint32_t)e};
          packet_store(m.qp[e & 1] + (size_t)k * m.nslots + slot, pk);
          stage_coord(own0 + 2 * ((size_t)T * (e & 1) + q), k, x[j].o.h, x[j].o.l, x[j].c);
        }
      }
    }
  };
  // the halo of evaluation e into shared memory.  A tile writes a buffer again
  // two evaluations later, for which it has to have received the next
  // evaluation's packets of every tile that reads it (the planner makes the
  // halo relation symmetric), and those are published after this read.
  auto receive = [&](int e) {
    receive_packets(m.qp[e & 1], m.nslots, a.tag0 + (uint32_t)e, hn, s_hslot, tid, nthr, a.err, s_fail,
                    [&](int p, int k, const Packet& d) {
                      stage_coord(halo + 2 * p, k, __uint_as_float(d.h), __uint_as_float(d.l), (int)d.c);
                    });
  };
  // forces on the owned beads at evaluation e; false when a packet never came
  auto evaluate = [&](int e) -> bool {
    const float4* own = own0 + 2 * (size_t)T * (e & 1);
    __syncthreads();  // the tile's own positions are staged
    if (*s_fail) return false;
    if (c1 > c0 && refresh_due(a, e)) {
      // Cilia::length (src/cilia.cpp:79-121) for every refreshed bond, in pairs
      refreshed = true;
      int off = 0;
      for (int c = c0; c < c1; ++c) {
        const CiliumDev cl = m.cil[c];
        const int nbnd = cl.len - cl.num_anker;
        const int w = tid - off;
        if (w >= 0 && w < nbnd) {
          const int i = cl.num_anker - 1 + w;
          const int k = cl.bond_base + i - b0;
          const int l0 = cl.slot0 - base;
          const int ia = l0 + cl.stride * i, ib = l0 + cl.stride * (i + 1);
          const DfDiff d = df_diff(own[2 * ia], own[2 * ia + 1], own[2 * ib], own[2 * ib + 1]);
          const dfloat tl = df_mul(d.d2, df_rsqrt(d.d2));
          const dfloat tg{s_tg[k].x, s_tg[k].y}, bd{s_bd[k].x, s_bd[k].y}, ol{s_ol[k].x, s_ol[k].y};
          dfloat l = tg;
          if (df_lt(bd, df_abs(df_sub(tg, tl)))) {
            const dfloat t2 = df_lt(tg, tl) ? df_sub(tl, bd) : df_add(tl, bd);
            l = df_sign(df_sub(tg, ol)) * df_sign(df_sub(t2, ol)) > 0 ? t2 : ol;
          }
          const dfloat g = df_sqrt(df_add(dfloat{0.25f, 0.f}, df_mul(dfloat{0.5f, 0.f}, l)));
          s_nl[k] = make_float2(l.h, l.l);
          s_ol[k] = make_float2(l.h, l.l);
          s_dg[k] = make_float2(g.h, g.l);
        }
        off += nbnd;
      }
      __syncthreads();
    }
    float axh = 0.f, axl = 0.f, ayh = 0.f, ayl = 0.f, azh = 0.f, azl = 0.f;
    float4 m0 = make_float4(0.f, 0.f, 0.f, 0.f), m1 = m0;
    if (mv >= 0) {
      m0 = own[2 * me];
      m1 = own[2 * me + 1];
      springs_df<LANES, kFloat>(tb, own, m0, m1, s0 + lane, sm, axh, axl, ayh, ayl, azh, azl);
    }
    if (hn > 0) {
      receive(e);
      __syncthreads();
      if (mv >= 0)
        springs_df<LANES, kFloat>(tb, halo - 2 * T, m0, m1, sm + lane, s1, axh, axl, ayh, ayl, azh, azl);
    }
    // the lanes' partial forces, each coordinate to its owner
    float fh[NC], fl[NC];
    if constexpr (LANES == 2) {
      fh[0] = lane ? ayh : axh;
      fl[0] = lane ? ayl : axl;
      exchange_add(fh[0], fl[0], lane ? axh : ayh, lane ? axl : ayl, 1);
      fh[1] = azh;
      fl[1] = azl;
      exchange_add(fh[1], fl[1], azh, azl, 1);
    } else {
      // quarters of the group: with eight lanes, lanes 2k and 2k + 1 hold
      // component k; lane k of the slot takes it from there
      group_sum_xyz<LANES>(lane, axh, axl, ayh, ayl, azh, azl, fh[0], fl[0]);
      if constexpr (LANES == 8) {
        const int src = (tid & 31 & ~7) | (2 * lane & 7);
        fh[0] = __shfl_sync(0xffffffffu, fh[0], src);
        fl[0] = __shfl_sync(0xffffffffu, fl[0], src);
      }
    }
    if (helpers) {
#pragma unroll
      for (int j = 0; j < NC; ++j)
        if (lane + j * LANES < 3) part[3 * q + lane + j * LANES] = make_float2(fh[j], fl[j]);
      __syncthreads();
      // long runs: the warp holding the primary's lanes adds the run's slot
      // sums, lane-strided and then by a tree -- a fixed order
      const int lane32 = tid & 31;
      unsigned runs = __ballot_sync(0xffffffffu, lane == 0 && nh + 1 > kTreeRun);
      while (runs) {
        const int src = __ffs(runs) - 1;  // the primary's lane 0
        runs &= runs - 1;
        const int p = ((tid & ~31) + src) / LANES;
        const int len = 1 + __shfl_sync(0xffffffffu, nh, src);
        float gxh = 0.f, gxl = 0.f, gyh = 0.f, gyl = 0.f, gzh = 0.f, gzl = 0.f;
        for (int k = lane32; k < len; k += 32) {
          const float2* ph = part + 3 * (p + k);
          df_acc(gxh, gxl, ph[0].x, ph[0].y);
          df_acc(gyh, gyl, ph[1].x, ph[1].y);
          df_acc(gzh, gzl, ph[2].x, ph[2].y);
        }
        float h, l;
        group_sum_xyz<32>(lane32, gxh, gxl, gyh, gyl, gzh, gzl, h, l);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const int k = lane + j * LANES;  // component k lies in lanes 8 k ..
          const float oh = __shfl_sync(0xffffffffu, h, 8 * k & 31), ol = __shfl_sync(0xffffffffu, l, 8 * k & 31);
          if ((lane32 & ~(LANES - 1)) == src) {
            fh[j] = oh;
            fl[j] = ol;
          }
        }
      }
      if (nh > 0 && nh + 1 <= kTreeRun) {  // short runs, in slot order
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const int k = lane + j * LANES;
          if (k < 3)
            for (int r = 1; r <= nh; ++r) {
              const float2 ph = part[3 * (q + r) + k];
              df_acc(fh[j], fl[j], ph.x, ph.y);
            }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) f[j] = df_norm(fh[j], fl[j]);
    return true;
  };
  auto kick_all = [&](dfloat c) {
#pragma unroll
    for (int j = 0; j < NC; ++j) kick(v[j], f[j], c);
  };
  auto drift_all = [&]() {
#pragma unroll
    for (int j = 0; j < NC; ++j) coord_kick(x[j], v[j], dt);
  };

  // md_loop_start: forces at t0, v += F dt/2, x += v dt
  publish(0);
  if (!evaluate(0)) return;
  if (moves) {
    kick_all(dt2);
    drift_all();
  }
  publish(1);
  if (!evaluate(1)) return;
  // md_loop: v += F dt, x += v dt, forces
  for (int k = 1; k < a.n; ++k) {
    if (moves) {
      kick_all(dt);
      drift_all();
    }
    publish(k + 1);
    if (!evaluate(k + 1)) return;
  }
  __syncthreads();
  if (*s_fail) return;  // the last evaluation's packets never came
  // md_loop_stop: v += F dt/2, then bin with the next shift
  if (moves) kick_all(dt2);
  {
    double X[3], V[3];
    const int g0 = (tid & 31) - lane;  // the slot's lane 0 within the warp
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      constexpr int kL = LANES;
      const int j = k / kL;
      X[k] = __shfl_sync(0xffffffffu, coord_to_double(x[j < NC ? j : 0]), g0 + k % kL);
      V[k] = __shfl_sync(0xffffffffu, df_to_double(v[j < NC ? j : 0]), g0 + k % kL);
    }
    if (prim && lane == 0) {
      m.x[0][slot] = X[0];
      m.y[0][slot] = X[1];
      m.z[0][slot] = X[2];
      m.vx[slot] = V[0];
      m.vy[slot] = V[1];
      m.vz[slot] = V[2];
      if (moves) {
        if (a.deferred)
          bin.defer(slot, X[0], X[1], X[2], V[0], V[1], V[2]);
        else
          bin(X[0], X[1], X[2], V[0], V[1], V[2]);
      }
    }
  }
  // refreshed bonds back to float64
  if (refreshed) {
    int off = 0;
    for (int c = c0; c < c1; ++c) {
      const CiliumDev cl = m.cil[c];
      const int nbnd = cl.len - cl.num_anker;
      const int w = tid - off;
      if (w >= 0 && w < nbnd) {
        const int k = cl.bond_base + cl.num_anker - 1 + w;
        const double l = df_to_double(dfloat{s_nl[k - b0].x, s_nl[k - b0].y});
        m.newlen[k] = l;
        m.oldlen[k] = l;
        m.diag[k] = df_to_double(dfloat{s_dg[k - b0].x, s_dg[k - b0].y});
      }
      off += nbnd;
    }
  }
  // switch_logic for the cilia of this tile (the staged positions are the final ones)
  const StageDF sv{own0 + 2 * (size_t)T * (a.n & 1)};
  for (int c = c0 + tid; c < c1; c += nthr) cilium_switch(m, a, c, a.t_end, base, sv);
}

template <int LANES, bool kFloat, typename Bin>
__global__ void __launch_bounds__(512) k_md_df(MDState m, typename Bin::Cells c, MDStepArgs a) {
  md_df_body<LANES, kFloat>(m, a, Bin{c, &a});
}

// the kernel for a layout: lanes per slot, double-float (m.df == 1) or float springs (2)
template <typename Bin>
const void* df_kernel(const MDState& m, int lanes) {
  const bool fl = m.df == 2;
  if (lanes == 8) return fl ? (const void*)k_md_df<8, true, Bin> : (const void*)k_md_df<8, false, Bin>;
  if (lanes == 2) return fl ? (const void*)k_md_df<2, true, Bin> : (const void*)k_md_df<2, false, Bin>;
  return fl ? (const void*)k_md_df<4, true, Bin> : (const void*)k_md_df<4, false, Bin>;
}

}  // namespace

// eight lanes per slot when the tile allows it (more warps in flight), else
// four, and two for the widest tiles (at most 512 threads per CTA)
int md_df_lanes(int tile) {
  static const int forced = [] {
    const char* env = std::getenv("MPCD_MD_DF_LANES");  // 4 or 8
    return env ? std::atoi(env) : 0;
  }();
  if (tile > 128) return 2;
  if (forced == 4 || (forced == 8 && tile <= 64)) return forced;
  return tile <= 64 ? 8 : 4;
}

namespace {

size_t md_df_smem(const MDState& m) {
  return DfSmem(m.tile, m.hmax, m.df_nsp_max, m.df_nb_max).total;
}

template <typename Bin>
int launch_df(const MDState& m, const typename Bin::Cells& c, const MDStepArgs& a, cudaStream_t s, cudaError_t* st) {
  if (m.nslots == 0 || m.ntiles == 0) return 0;
  MDState mm = m;
  typename Bin::Cells cc = c;
  MDStepArgs aa = a;
  md_set_dt_pairs(aa);
  void* args[] = {&mm, &cc, &aa};
  const size_t smem = md_df_smem(m);
  const int lanes = md_df_lanes(m.tile);
  const void* k = df_kernel<Bin>(m, lanes);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  *st = cudaLaunchCooperativeKernel(k, dim3(m.ntiles), dim3(lanes * m.tile), args, smem, s);
  return 1;
}

}  // namespace

int launch_md_df_f64cells(const MDState& m, const CellsF64& c, const MDStepArgs& a, cudaStream_t s, cudaError_t* st) {
  return launch_df<BinF64>(m, c, a, s, st);
}

int launch_md_df_f32cells(const MDState& m, const CellsF32& c, const MDStepArgs& a, cudaStream_t s, cudaError_t* st) {
  return launch_df<BinF32>(m, c, a, s, st);
}

int md_df_max_coresident_blocks(const MDState& m, int f32cells) {
  int dev = 0, sms = 0, per_sm = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t smem = md_df_smem(m);
  if (smem > (size_t)optin) return 0;
  const int lanes = md_df_lanes(m.tile);
  const void* k = f32cells ? df_kernel<BinF32>(m, lanes) : df_kernel<BinF64>(m, lanes);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, lanes * m.tile, smem);
  return per_sm * sms;
}

}  // namespace mpcd
