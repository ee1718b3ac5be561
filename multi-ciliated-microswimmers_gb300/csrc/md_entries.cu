// MD substeps of one MPC step on the double-float coordinates of md_df.cu,
// every spring pair evaluated once, a thread per pair.
//
// Same integrator, forces and arithmetic as md_df.cu (velocity Verlet of
// src/libcilia/mdobject.cpp:36-72 inside the loop of src/simulation.cpp:217-265;
// springs of src/cilia.cpp:127-239, src/sphere.cpp:87-119, src/clami.cpp:188-198;
// positions as integer cell + offset pair, forces and sums in float pairs) and
// the same exchange of positions by tagged packets (md_packets.cuh).  What
// differs is how a tile's work is cut.  There the lanes of a slot walk the
// slot's own springs: a substep is two or more spring evaluations deep, one
// behind the other, although every CTA has threads to spare.  Here a spring
// and its exact reverse inside the tile form one entry (the reference makes
// cilium and sphere springs from both ends; the two forces are negations of
// each other bit for bit), the threads take one entry each, and every bead's
// forces are then added in the order in which md_df.cu's lanes and slots add
// them: the two kernels give the same results bit for bit (a sum in another
// order grows, in stiff springs, to 1e-9 of a small swimmer's velocities within
// five steps).  The planner cuts the beads into many
// small tiles, up to the number of SMs: cilia as they are, the other beads in
// compact patches, and a bead with a very long list (a sphere's centre) in a
// tile of its own.
//
// The chain of one substep: packets arrive -> one entry -> a bead's sum ->
// Verlet -> packets leave.  The entries between the tile's own beads are
// evaluated by the first warps while the last warps poll.  The launch is
// latency bound (51 dependent evaluations of about 2.6 us; issue slots, pipes
// and DRAM mostly idle): a packet takes 250-600 ns from one SM to another,
// an entry about 0.4 us, a bead's sum and Verlet step 0.4 us, and the round of
// the sphere centre's tile (its 642 beads' packets, written elsewhere since the
// last read, take about 0.9 us to fetch) alternates
// with the patches' rounds.
//
// MD per launch timed alone, this kernel / md_df.cu: swimmer64 135 / 217 us in
// double-float, 124 / 196 with float springs; a 700-bead swimmer 131 / 187;
// swimmer128 with float springs 223 / 431 (there a tile of 256 slots has two
// lanes per slot, and its springs follow one another; here 152 tiles of three
// cilia or 151 sphere beads).  Running sums of the entries in any order took
// 122, 114, 117 and 213 us.
#include <algorithm>

#include "../../include/mpcd_gpu.h"
#include "df32.cuh"
#include "md_common.cuh"
#include "md_df_coord.cuh"
#include "md_packets.cuh"

namespace mpcd {

namespace {

// A staged position: {h of x, y, z, the cell of x}, {l of x, y, z, the cell of
// y}, the cell of z (exact as floats below 2^24).
struct Staged {
  float4* a;
  float4* b;
  float* c;
  __device__ void put(int i, int k, float h, float l, int cell) const {
    reinterpret_cast<float*>(a + i)[k] = h;
    reinterpret_cast<float*>(b + i)[k] = l;
    const float f = (float)cell;
    if (k == 0)
      reinterpret_cast<float*>(a + i)[3] = f;
    else if (k == 1)
      reinterpret_cast<float*>(b + i)[3] = f;
    else
      c[i] = f;
  }
  // float64 distance (switch_logic's bend measure)
  __device__ double dist(int i, int j) const {
    const float4 ai = a[i], bi = b[i], aj = a[j], bj = b[j];
    const double dx = ((double)ai.w - (double)aj.w) + (df_to_double({ai.x, bi.x}) - df_to_double({aj.x, bj.x}));
    const double dy = ((double)bi.w - (double)bj.w) + (df_to_double({ai.y, bi.y}) - df_to_double({aj.y, bj.y}));
    const double dz = ((double)c[i] - (double)c[j]) + (df_to_double({ai.z, bi.z}) - df_to_double({aj.z, bj.z}));
    return sqrt(dx * dx + dy * dy + dz * dz);
  }
};

// a b + c d + e f with the roundings that the compiler gives df_diff's sums (it
// may fuse either product of the first two): both kernels' springs are the same
// bit for bit
__device__ __forceinline__ float dot3(float a, float b, float c, float d, float e, float f) {
  return fmaf(e, f, fmaf(c, d, __fmul_rn(a, b)));
}
// x_i - x_j of two staged positions as pairs, and its squared length as a
// normalised pair (as df_diff)
__device__ __forceinline__ DfDiff staged_diff(const float4 a0, const float4 a1, float az, const float4 b0,
                                              const float4 b1, float bz) {
  DfDiff r;
  r.dx = coord_diff(__fsub_rn(a0.w, b0.w), a0.x, b0.x, a1.x, b1.x);
  r.dy = coord_diff(__fsub_rn(a1.w, b1.w), a0.y, b0.y, a1.y, b1.y);
  r.dz = coord_diff(__fsub_rn(az, bz), a0.z, b0.z, a1.z, b1.z);
  const dfloat px = df_two_prod(r.dx.h, r.dx.h), py = df_two_prod(r.dy.h, r.dy.h), pz = df_two_prod(r.dz.h, r.dz.h);
  const dfloat q1 = df_two_sum(px.h, py.h);
  const dfloat q2 = df_two_sum(q1.h, pz.h);
  float low = __fadd_rn(__fadd_rn(q1.l, q2.l), __fadd_rn(__fadd_rn(px.l, py.l), pz.l));
  low = fmaf(2.0f, dot3(r.dx.h, r.dx.l, r.dy.h, r.dy.l, r.dz.h, r.dz.l), low);
  low = __fadd_rn(low, dot3(r.dx.l, r.dx.l, r.dy.l, r.dy.l, r.dz.l, r.dz.l));
  r.d2 = df_fast_two_sum(q2.h, low);
  return r;
}

// The three components of a force: pairs (high part, unnormalised low part)
// or, with float springs, the factors {fac, d} of a product that the sum rounds
// once (fused multiply-add).
struct Force {
  float2 x, y, z;
};
template <bool kFloat>
__device__ __forceinline__ float2 opposite(float2 p) {
  return kFloat ? make_float2(p.x, -p.y) : make_float2(-p.x, -p.y);
}
template <bool kFloat>
__device__ __forceinline__ void force_acc(float& h, float& l, float2 p) {
  if constexpr (kFloat)
    h = fmaf(p.x, p.y, h);
  else
    df_acc(h, l, p.x, p.y);
}
// F = -2k (1 - b / |d|) d on the first bead, d its position less the other's,
// rk = {b, -2k} as pairs; guarded: no force at zero distance (the vector-form
// spring).  kFloat: d formed exactly as pairs and rounded to float, the rest in
// float (the split arithmetic of the float32 path).
template <bool kFloat>
__device__ __forceinline__ Force spring_force(const float4 a0, const float4 a1, float az, const float4 b0,
                                              const float4 b1, float bz, const float4 rk, bool guarded) {
  Force F;
  if constexpr (kFloat) {
    const dfloat ex = coord_diff(__fsub_rn(a0.w, b0.w), a0.x, b0.x, a1.x, b1.x);
    const dfloat ey = coord_diff(__fsub_rn(a1.w, b1.w), a0.y, b0.y, a1.y, b1.y);
    const dfloat ez = coord_diff(__fsub_rn(az, bz), a0.z, b0.z, a1.z, b1.z);
    const float dx = ex.h + ex.l, dy = ey.h + ey.l, dz = ez.h + ez.l;
    const float d2 = dot3(dx, dx, dy, dy, dz, dz);
    float fac = rk.z * (1.0f - rk.x * rsqrtf(d2));
    if (guarded && d2 == 0.0f) fac = 0.0f;
    F.x = make_float2(fac, dx);
    F.y = make_float2(fac, dy);
    F.z = make_float2(fac, dz);
  } else {
    const DfDiff d = staged_diff(a0, a1, az, b0, b1, bz);
    const dfloat r = df_rsqrt(d.d2);
    // w = 1 - b r
    const dfloat u = df_two_prod(rk.x, r.h);
    const dfloat w = df_two_sum(1.0f, -u.h);
    const float wl = ((w.l - u.l) - rk.x * r.l) - rk.y * r.h;
    // fac = -2k w
    dfloat f = df_two_prod(rk.z, w.h);
    float fl = (f.l + rk.z * wl) + rk.w * w.h;
    if (guarded && d.d2.h == 0.0f) f.h = fl = 0.0f;
    const dfloat px = df_two_prod(f.h, d.dx.h), py = df_two_prod(f.h, d.dy.h), pz = df_two_prod(f.h, d.dz.h);
    F.x = make_float2(px.h, (px.l + f.h * d.dx.l) + fl * d.dx.h);
    F.y = make_float2(py.h, (py.l + f.h * d.dy.l) + fl * d.dy.h);
    F.z = make_float2(pz.h, (pz.l + f.h * d.dz.l) + fl * d.dz.h);
  }
  return F;
}

// the same with the other bead's three packets
template <bool kFloat>
__device__ __forceinline__ Force packet_force(const float4 a0, const float4 a1, float az, const Packet* d,
                                              const float4 rk, bool guarded) {
  const float4 b0 = make_float4(__uint_as_float(d[0].h), __uint_as_float(d[1].h), __uint_as_float(d[2].h),
                                (float)(int)d[0].c);
  const float4 b1 = make_float4(__uint_as_float(d[0].l), __uint_as_float(d[1].l), __uint_as_float(d[2].l),
                                (float)(int)d[1].c);
  return spring_force<kFloat>(a0, a1, az, b0, b1, (float)(int)d[2].c, rk, guarded);
}

// A slot's sum as md_df.cu's lanes make it: LN running sums over the rows of
// the slot's words (a row: one word per lane, `step` apart), combined by the
// lanes' tree as its lane 0 sees it.  A lane without a spring in a row holds zero,
// which changes nothing.
template <int LN, bool kFloat>
__device__ __forceinline__ void lane_sums(const float2* F, int step, int row, int rows, float& h, float& l) {
  float sh[LN], sl[LN];
#pragma unroll
  for (int q = 0; q < LN; ++q) {
    const float2 p = F[q * step];
    sh[q] = kFloat ? __fmul_rn(p.x, p.y) : p.x;
    sl[q] = kFloat ? 0.f : p.y;
  }
  constexpr int kAhead = LN >= 4 ? 1 : 4;  // rows whose loads go out together; past the last one zero
#pragma unroll 1
  for (int r = 1; r < rows; r += kAhead) {
    float2 p[kAhead][LN];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      F += row;
#pragma unroll
      for (int q = 0; q < LN; ++q) p[u][q] = r + u < rows ? F[q * step] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
#pragma unroll
      for (int q = 0; q < LN; ++q) force_acc<kFloat>(sh[q], sl[q], p[u][q]);
  }
#pragma unroll
  for (int o = 1; o < LN; o <<= 1)
#pragma unroll
    for (int q = 0; q + o < LN; q += 2 * o) df_acc(sh[q], sl[q], sh[q + o], sl[q + o]);
  h = sh[0];
  l = sl[0];
}
template <int HALVES, bool kFloat>
__device__ __forceinline__ void slot_sum(int lanes, const float2* F, int step, int rows, float& h, float& l) {
  if (lanes == 8)
    lane_sums<8 / HALVES, kFloat>(F, step, lanes * step, rows, h, l);
  else if (lanes == 4)
    lane_sums<4 / HALVES, kFloat>(F, step, lanes * step, rows, h, l);
  else
    lane_sums<2 / HALVES, kFloat>(F, step, lanes * step, rows, h, l);
}
// The sum of n slots' sums w[0 .. n) as a warp of md_df.cu makes it (lane l adds l,
// l + 32, ... and the lanes are combined by a xor tree, 16 first, each adding its
// partner's value to its own), as its lane `src` ends with it.  By the eight lanes
// of a group: t stands for the four of that warp's lanes whose low bits are src's xor t.
// The sum is in the group's lane 0.
__device__ __forceinline__ void slots_tree(const float2* w, int n, int src, int t, float& h, float& l) {
  const int c = src ^ t;
  auto strided = [&](int k, float& sh, float& sl) {
    sh = sl = 0.f;
    if (k < n) {
      sh = w[k].x;
      sl = w[k].y;
    }
#pragma unroll 1
    for (k += 32; k < n; k += 32) df_acc(sh, sl, w[k].x, w[k].y);
  };
  float ah, al, bh, bl, ch, cl, dh, dl;
  strided(c, ah, al);
  strided(c ^ 16, bh, bl);
  strided(c ^ 8, ch, cl);
  strided(c ^ 24, dh, dl);
  df_acc(ah, al, bh, bl);
  df_acc(ch, cl, dh, dl);
  df_acc(ah, al, ch, cl);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, ah, o), ol = __shfl_xor_sync(0xffffffffu, al, o);
    df_acc(ah, al, oh, ol);
  }
  h = ah;
  l = al;
}

// md_df.cu adds the slots of a bead with more than this many by a warp's tree,
// fewer in order
constexpr int kTreeRun = 8;

// Makes x opaque to the compiler from here on: what a substep uses stays in
// its register instead of being computed again (integer divisions, float64
// conversions) in every turn of the substep loop.
__device__ __forceinline__ void keep(int& x) { asm volatile("" : "+r"(x)); }

// shared-memory layout of one tile
struct EntSmem {
  size_t oa, ob, oc, ha, hb, hc, hslot, flag, code, rk, meta, f, nl, ol, dg, tg, bd, fin, total;
  __host__ __device__ EntSmem(int T, int hmax, int nent, int ninc, int nb) {
    size_t o = 0;
    auto take = [&](size_t bytes, size_t align) {
      o = (o + align - 1) / align * align;
      const size_t r = o;
      o += bytes;
      return r;
    };
    oa = take(32 * (size_t)T, 16);
    ob = take(32 * (size_t)T, 16);
    ha = take(16 * (size_t)hmax, 16);
    hb = take(16 * (size_t)hmax, 16);
    rk = take(16 * (size_t)nent, 16);
    code = take(8 * (size_t)nent, 8);
    f = take(24 * (size_t)ninc, 8);
    nl = take(8 * (size_t)nb, 8);
    ol = take(8 * (size_t)nb, 8);
    dg = take(8 * (size_t)nb, 8);
    tg = take(8 * (size_t)nb, 8);
    bd = take(8 * (size_t)nb, 8);
    fin = take(48 * (size_t)T, 8);
    oc = take(8 * (size_t)T, 4);
    hc = take(4 * (size_t)hmax, 4);
    hslot = take(4 * (size_t)hmax, 4);
    meta = take(4 * (size_t)nent, 4);
    flag = take(4, 4);
    total = o;
  }
};

template <int NC, int HALVES, bool kFloat, typename Bin>
__device__ void md_entries_body(const MDState& m, const MDStepArgs& a, Bin bin) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int T = m.tile;
  const EntSmem L(T, m.hmax, m.de_nent_max, m.de_ninc_max, m.df_nb_max);
  float4* const oa = reinterpret_cast<float4*>(smem + L.oa);
  float4* const ob = reinterpret_cast<float4*>(smem + L.ob);
  float* const oc = reinterpret_cast<float*>(smem + L.oc);
  const Staged halo{reinterpret_cast<float4*>(smem + L.ha), reinterpret_cast<float4*>(smem + L.hb),
                    reinterpret_cast<float*>(smem + L.hc)};
  int* s_hslot = reinterpret_cast<int*>(smem + L.hslot);
  int* s_fail = reinterpret_cast<int*>(smem + L.flag);  // 1: a packet never came
  // entries: {bead a | guarded << 15 | bead b << 16, incidence of a | of b << 16 (0xffff: none)},
  // {rest length, -2k} as pairs, {kind | bond << 2} (a solo tile: the rows of its i-th slot)
  uint2* s_code = reinterpret_cast<uint2*>(smem + L.code);
  float4* s_rk = reinterpret_cast<float4*>(smem + L.rk);
  uint32_t* s_meta = reinterpret_cast<uint32_t*>(smem + L.meta);
  // the force each incidence (a bead's spring, in its spring order) puts on its bead
  float2* const s_fx = reinterpret_cast<float2*>(smem + L.f);
  const int fw = m.de_ninc_max;  // y at s_fx + fw, z at s_fx + 2 fw
  float2* s_nl = reinterpret_cast<float2*>(smem + L.nl);
  float2* s_ol = reinterpret_cast<float2*>(smem + L.ol);
  float2* s_dg = reinterpret_cast<float2*>(smem + L.dg);
  float2* s_tg = reinterpret_cast<float2*>(smem + L.tg);
  float2* s_bd = reinterpret_cast<float2*>(smem + L.bd);

  const int tile = blockIdx.x;
  const int base = tile * T;
  const int tid = threadIdx.x, nthr = blockDim.x, back = nthr - 1 - tid;
  const int lane32 = tid & 31, warp = tid >> 5;
  const bool solo = m.de_solo[tile] != 0;
  // narrow tiles go with slots of eight lanes: known here, the sums' code is one
  // straight line (64^3 swimmer 138 to 135 us per launch, with float springs 127 to 123)
  const int lanes = HALVES == 2 ? 8 : m.de_lanes;
  // owned coordinates: number c = tid / HALVES + j nthr below 3 T is coordinate
  // c / T of bead c mod T, so that few warps run the sums and the Verlet step
  // (a warp's instructions count once, however many lanes take part); with
  // two halves two neighbouring threads share a sum, the even one owns it
  const int half = HALVES == 2 ? tid & 1 : 0;
  int cq[NC], ck[NC], cmv[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int c = tid / HALVES + j * nthr;
    ck[j] = solo ? ((tid & 7) || j ? 3 : tid >> 3) : c / T;  // a solo tile's bead: lanes 0, 8, 16
    cq[j] = solo ? 0 : c - ck[j] * T;
    cmv[j] = ck[j] < 3 ? m.moves[base + cq[j]] : -1;  // 1 moves, 0 fixed, -1 none
  }
  const int h0 = m.halo_start[tile], hn0 = m.halo_start[tile + 1] - h0;
  const int c0 = m.tile_cil[tile], c1 = m.tile_cil[tile + 1];
  const int b0 = m.tile_b0[tile], nb = m.tile_nb[tile];
  const int e0 = m.de_start[tile], nent0 = m.de_start[tile + 1] - e0, nloc0 = m.de_local_end[tile] - e0;
  // a bead's force words: from f0 on, fstep apart, a nibble of fshape per slot:
  // its rows of one word per lane
  const int ninc = m.de_nslot[tile];
  const int fstep = m.de_step;
  int f0[NC];
  uint32_t fshape[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int s = base + cq[j];
    f0[j] = cmv[j] >= 0 && !solo ? m.de_at[s] : 0;
    fshape[j] = cmv[j] == 1 && !solo ? m.de_shape[s] : 0u;  // a fixed bead needs no force
  }
  const int wmax = m.de_slots[tile];  // most slots of one of its beads
  // a solo tile's words: as many rows for every slot, then the slots' sums
  const int solo_src = solo ? m.de_at[base] : 0, solo_slots0 = solo ? (int)m.de_shape[base] : 0;
  const dfloat dt{a.dt_pair.x, a.dt_pair.y}, dt2{a.dt2_pair.x, a.dt2_pair.y};

  // the plan must fit the tables and the halo's slots the packet buffers
  if (tid == 0)
    *s_fail = hn0 < 0 || hn0 > m.hmax || nent0 < 0 || nent0 > m.de_nent_max || nloc0 < 0 || nloc0 > nent0 || ninc < 0 ||
              ninc > m.de_ninc_max || nb > m.df_nb_max ||
              (solo && (solo_slots0 < 1 || solo_slots0 > nent0 || wmax < 0 || solo_slots0 * (wmax * lanes + 1) > ninc));
  __syncthreads();
  const bool fits = *s_fail == 0;
  __syncthreads();
  for (int i = tid; i < hn0 && fits; i += nthr) {
    const int g = m.halo[h0 + i];
    s_hslot[i] = g;
    if (g < 0 || g >= m.nslots) *s_fail = 1;
  }
  for (int i = tid; i < nent0 && fits; i += nthr) {
    const uint4 c = __ldg(m.de_code + e0 + i);
    const int ea = (int)(c.x & 0x7fffu), eb = (int)(c.x >> 16), ka = (int)(c.y & 0xffffu), kb = (int)(c.y >> 16);
    const int kind = (int)(c.z & 3u), lref = (int)(c.z >> 2);
    if (ea >= T || eb >= T + hn0 || (eb >= T) != (i >= nloc0) || ka >= ninc || (kb != 0xffff && kb >= ninc) ||
        (kind >= MPCD_SPRING_BOND && lref >= nb) || (solo && (int)c.w > wmax))
      *s_fail = 1;
    s_code[i] = make_uint2(c.x, c.y);
    s_meta[i] = solo ? c.w : c.z;
    float4 rk = __ldg(m.de_rk + e0 + i);
    if (kind >= MPCD_SPRING_BOND && lref < nb) {
      const dfloat r = df_from_double((kind == MPCD_SPRING_BOND ? m.newlen : m.diag)[b0 + lref]);
      rk.x = r.h;
      rk.y = r.l;
    }
    s_rk[i] = rk;
  }
  for (int i = tid; i < 3 * fw && fits; i += nthr) s_fx[i] = make_float2(0.f, 0.f);  // words without a spring stay zero
#pragma unroll
  for (int j = 0; j < NC && fits; ++j) {  // every owned bead's words lie in the table
    int words = 0;
    for (uint32_t t = fshape[j]; t; t >>= 4) words += (int)(t & 15u) * lanes;
    if (f0[j] < 0 || (words > 0 && f0[j] + (words - 1) * fstep >= ninc)) *s_fail = 1;
  }
  __syncthreads();
  const bool plan_ok = *s_fail == 0;  // an inconsistent plan: no halo, no entries (and an error)
  __syncthreads();
  if (!plan_ok && tid == 0) {
    atomicOr(a.err, kErrLayout);
    *s_fail = 0;
  }
  const int hn = plan_ok ? hn0 : 0, nent = plan_ok ? nent0 : 0, nloc = plan_ok ? nloc0 : 0;
  const int nbt = plan_ok ? nb : 0, solo_slots = plan_ok ? solo_slots0 : 0;
  for (int i = tid; i < nbt; i += nthr) {
    const dfloat n = df_from_double(m.newlen[b0 + i]), o = df_from_double(m.oldlen[b0 + i]);
    const dfloat g = df_from_double(m.diag[b0 + i]);
    s_nl[i] = make_float2(n.h, n.l);
    s_ol[i] = make_float2(o.h, o.l);
    s_dg[i] = make_float2(g.h, g.l);
  }
  // calls f(cilium, bond i, table index) for every refreshed bond, a thread each
  auto each_bond = [&](auto&& f) {
    int off = 0;
    for (int c = c0; c < c1; ++c) {
      const CiliumDev cl = m.cil[c];
      const int nbnd = cl.len - cl.num_anker;
      const int w = tid - off;
      if (w >= 0 && w < nbnd) {
        const int i = cl.num_anker - 1 + w, k = cl.bond_base + i - b0;
        if (k >= 0 && k < nbt) f(c, cl, i, k);
      }
      off += nbnd;
    }
  };
  // the beat's rest length of every refreshed bond for this step, and the bending limit
  each_bond([&](int c, const CiliumDev& cl, int i, int k) {
    const dfloat t = df_from_double(cilium_target(cl, i, m.midpnt[c]));
    const dfloat bd = df_from_double(cl.bending);
    s_tg[k] = make_float2(t.h, t.l);
    s_bd[k] = make_float2(bd.h, bd.l);
  });
  // the owned coordinates
  BeadCoord x[NC];
  dfloat v[NC];
  double ke_coll = 0.0;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    double X[3] = {0.0, 0.0, 0.0}, V[3] = {0.0, 0.0, 0.0};
    if (cmv[j] >= 0) {
      const int s = base + cq[j];
      X[0] = m.x[0][s];
      X[1] = m.y[0][s];
      X[2] = m.z[0][s];
      V[0] = m.vx[s];
      V[1] = m.vy[s];
      V[2] = m.vz[s];
      if (a.collide && cmv[j] == 1) {  // the beads' collision, folded in (the same for a bead's three owners)
        const double ke = bin.collide(X[0], X[1], X[2], V[0], V[1], V[2]);
        if (ck[j] == 0 && half == 0) ke_coll += ke;
      }
      if (!plan_ok) fshape[j] = 0u;
    }
    x[j] = coord_from_double(ck[j] == 0 ? X[0] : (ck[j] == 1 ? X[1] : X[2]));
    v[j] = df_from_double(ck[j] == 0 ? V[0] : (ck[j] == 1 ? V[1] : V[2]));
  }
  if (a.collide) {  // the dissipated-energy bookkeeping of the collided beads
    const double tot = block_sum_f64(ke_coll);
    if (tid == 0 && tot != 0.0) atomicAdd(a.diss, -tot);
  }
  int my_k = (back >= hn) + (back >= 2 * hn), my_p = back - my_k * hn;  // this thread's halo packet
  int my_src = back < 3 * hn ? my_k * m.nslots + s_hslot[my_p] : 0;
  int si = tid - 32, si2 = si + nthr - 32 < nent ? si + nthr - 32 : si;  // a solo tile's first two entries
  // the place of number p of a solo tile's sums: slot (-1: none), first word
  // (word j of slot k at j solo_slots + k), and where the sum goes
  auto solo_place = [&](int p, int& k, int& at, int& to) {
    const int ax = (p >> 1) / max(1, solo_slots);
    k = ax < 3 && solo ? (p >> 1) - ax * solo_slots : -1;
    at = ax * fw + (p & 1) * (lanes / 2) * solo_slots + k;
    to = ax * fw + lanes * wmax * solo_slots + k;
  };
  int sk, sat, sout;
  solo_place(tid, sk, sat, sout);
  int pub[NC], fat[NC];  // packet of each owned coordinate (-1: not this thread's), and its first incidence
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    pub[j] = cmv[j] < 0 || half ? -1 : ck[j] * m.nslots + base + cq[j];
    fat[j] = ck[j] * fw + f0[j] + half * (lanes / HALVES) * fstep;
    keep(pub[j]);
    keep(fat[j]);
    keep(cq[j]);
    keep(ck[j]);
    keep(cmv[j]);
  }
  keep(my_k);
  keep(my_p);
  keep(my_src);
  keep(si);
  keep(si2);
  keep(sk);
  keep(sat);
  keep(sout);
  int wslots[NC];  // most slots of a bead of this warp
#pragma unroll
  for (int j = 0; j < NC; ++j) wslots[j] = (int)__reduce_max_sync(0xffffffffu, (35u - __clz((int)fshape[j])) >> 2);
  bool refreshed = false;

  // md_loop_start, n x md_loop, md_loop_stop: evaluation e of the forces at
  // the positions of substep e, then v += F dt (dt / 2 at both ends), x += v dt
  for (int e = 0;; ++e) {
    const Staged own{oa + (size_t)T * (e & 1), ob + (size_t)T * (e & 1), oc + (size_t)T * (e & 1)};
    // own beads into shared memory and, as packets, into global buffer e & 1
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (pub[j] >= 0) {
        packet_store(m.qp[e & 1] + pub[j],
                     Packet{__float_as_uint(x[j].o.h), __float_as_uint(x[j].o.l), (uint32_t)x[j].c, a.tag0 + (uint32_t)e});
        own.put(cq[j], ck[j], x[j].o.h, x[j].o.l, x[j].c);
      }
    // a solo tile's other warps ask for the next positions of their entries'
    // beads while the first one sums and moves the tile's bead
    Packet d[6];
    uint2 sc1 = make_uint2(0, 0), sc2 = sc1;
    if (solo && tid >= 32 && si < nent) {
      // not at once: the polls' loads stand in the way of the first warp's shared
      // memory and shuffles (64^3 swimmer 143 to 138 us per launch, with float springs 133
      // to 127; 130 ns and more 142, 127)
      __nanosleep(80);
      sc1 = s_code[si];
      sc2 = s_code[si2];
      receive_two(m.qp[e & 1], m.nslots, a.tag0 + (uint32_t)e, s_hslot[(int)(sc1.x >> 16) - T],
                  s_hslot[(int)(sc2.x >> 16) - T], d, a.err, s_fail);
    }
    // the tile's own positions are staged, the last evaluation's forces read;
    // now and then the CTA looks, as one, whether a packet never came
    if ((e & 7) == 7) {
      if (__syncthreads_or(*(volatile int*)s_fail)) return;
    } else {
      __syncthreads();
    }
    const bool due = c1 > c0 && refresh_due(a, e);
    if (due) {
      // Cilia::length (src/cilia.cpp:79-121) for every refreshed bond, in pairs
      refreshed = true;
      each_bond([&](int, const CiliumDev& cl, int i, int k) {
        const int l0 = cl.slot0 - base;
        const int p = l0 + i;
        const DfDiff d = staged_diff(own.a[p], own.b[p], own.c[p], own.a[p + 1], own.b[p + 1], own.c[p + 1]);
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
      });
      __syncthreads();
    }
    if (solo) {
      // one bead with a long list: a thread takes its entries' other beads
      // straight from their packets, two at a time; the lanes of the bead's slots
      // then add their words
      const float4 ca = own.a[0], cb = own.b[0];
      const float cc = own.c[0];
      if (tid >= 32) {
        auto put = [&](uint32_t k, const Force& g) {
          s_fx[k] = g.x;
          s_fx[k + fw] = g.y;
          s_fx[k + 2 * fw] = g.z;
        };
#pragma unroll 1
        for (int i = si, i2 = si2; i < nent;) {
          put(sc1.y & 0xffffu, packet_force<kFloat>(ca, cb, cc, d, s_rk[i], (sc1.x & 0x8000u) != 0));
          if (i2 != i) put(sc2.y & 0xffffu, packet_force<kFloat>(ca, cb, cc, d + 3, s_rk[i2], (sc2.x & 0x8000u) != 0));
          i += 2 * (nthr - 32);
          if (i >= nent) break;
          i2 = i + nthr - 32 < nent ? i + nthr - 32 : i;
          sc1 = s_code[i];
          sc2 = s_code[i2];
          receive_two(m.qp[e & 1], m.nslots, a.tag0 + (uint32_t)e, s_hslot[(int)(sc1.x >> 16) - T],
                      s_hslot[(int)(sc2.x >> 16) - T], d, a.err, s_fail);
        }
      }
      __syncthreads();
      // a thread per slot, half of its lanes and coordinate (sk, its words at
      // sat, its sum to sout): the first round's place is kept
#pragma unroll 1
      for (int p = tid, k = sk, at = sat, to = sout; p - lane32 < 6 * solo_slots;) {  // whole warps
        float h = 0.f, l = 0.f;
        if (k >= 0) slot_sum<2, kFloat>(lanes, s_fx + at, solo_slots, (int)s_meta[k], h, l);
        const float oh = __shfl_xor_sync(0xffffffffu, h, 1), ol = __shfl_xor_sync(0xffffffffu, l, 1);
        df_acc(h, l, oh, ol);
        if (k >= 0 && !(tid & 1)) s_fx[to] = make_float2(h, l);
        p += nthr;
        if (p - lane32 < 6 * solo_slots) solo_place(p, k, at, to);
      }
    } else {
      // phase 0: the entries between own beads, from the first thread up;
      // phase 1: the halo arrives and its entries, from the last thread down
      // (one copy of the code for both: it is fetched again at every substep)
#pragma unroll 1
      for (int ph = 0; ph < 2; ++ph) {
        int i = tid, iend = nloc;
        Staged other = own;
        if (ph) {
          if (hn > 0) {
            const uint4* src = m.qp[e & 1];
            const uint32_t tag = a.tag0 + (uint32_t)e;
            if (3 * hn <= nthr) {  // at most one packet a thread, always the same
              if (back < 3 * hn) {
                Packet d = packet_load(src + my_src);
                for (uint32_t spins = 0; d.tag != tag && !poll_given_up(spins, a.err, s_fail); ++spins)
                  d = packet_load(src + my_src);
                halo.put(my_p, my_k, __uint_as_float(d.h), __uint_as_float(d.l), (int)d.c);
              }
            } else {
              receive_packets(src, m.nslots, tag, hn, s_hslot, back, nthr, a.err, s_fail,
                              [&](int p, int k, const Packet& d) {
                                halo.put(p, k, __uint_as_float(d.h), __uint_as_float(d.l), (int)d.c);
                              });
            }
            __syncthreads();
          }
          i = nloc + back;
          iend = nent;
          other = Staged{halo.a - T, halo.b - T, halo.c - T};
        }
#pragma unroll 1
        for (; i < iend; i += nthr) {
          const uint2 c = s_code[i];
          float4 rk = s_rk[i];
          if (due) {  // take over the refreshed rest length
            const uint32_t mt = s_meta[i], kind = mt & 3u;
            if (kind >= MPCD_SPRING_BOND) {
              const float2 r = kind == MPCD_SPRING_BOND ? s_nl[mt >> 2] : s_dg[mt >> 2];
              rk.x = r.x;
              rk.y = r.y;
              s_rk[i] = rk;
            }
          }
          const int ea = (int)(c.x & 0x7fffu), eb = (int)(c.x >> 16);
          const bool guarded = (c.x & 0x8000u) != 0;
          const Force g = spring_force<kFloat>(own.a[ea], own.b[ea], own.c[ea], other.a[eb], other.b[eb], other.c[eb], rk,
                                               guarded);
          const int ka = (int)(c.y & 0xffffu), kb = (int)(c.y >> 16);
          s_fx[ka] = g.x;
          s_fx[ka + fw] = g.y;
          s_fx[ka + 2 * fw] = g.z;
          if (kb != 0xffff) {
            s_fx[kb] = opposite<kFloat>(g.x);
            s_fx[kb + fw] = opposite<kFloat>(g.y);
            s_fx[kb + 2 * fw] = opposite<kFloat>(g.z);
          }
        }
      }
    }
    __syncthreads();
    // every owned coordinate of the force, summed as md_df.cu's lanes, helper
    // slots and warps sum it, then the Verlet step
    const bool last = e == a.n;
    const dfloat c = e == 0 || last ? dt2 : dt;
    float ssh = 0.f, ssl = 0.f;  // a solo tile's coordinate tid / 8, in lanes 0, 8 and 16
    if (solo && warp == 0) {
      const float2* w = s_fx + min(lane32 >> 3, 2) * fw + lanes * wmax * solo_slots;
      if (solo_slots > kTreeRun) {
        slots_tree(w, solo_slots, solo_src, lane32 & 7, ssh, ssl);
      } else {
        for (int k = 0; k < solo_slots; ++k) df_acc(ssh, ssl, w[k].x, w[k].y);
      }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      float th = 0.f, tl = 0.f;
      if (solo) {
        th = ssh;
        tl = ssl;
      } else {
        const float2* F = s_fx + fat[j];
        uint32_t shape = fshape[j];
#pragma unroll 1
        for (int k = 0; k < wslots[j]; ++k, shape >>= 4) {  // slot after slot
          const int rows = (int)(shape & 15u);
          float h = 0.f, l = 0.f;
          if (rows > 0) {
            slot_sum<HALVES, kFloat>(lanes, F, fstep, rows, h, l);
            F += rows * lanes * fstep;
          }
          if constexpr (HALVES == 2) {
            const float oh = __shfl_xor_sync(0xffffffffu, h, 1), ol = __shfl_xor_sync(0xffffffffu, l, 1);
            df_acc(h, l, oh, ol);
          }
          if (k == 0) {
            th = h;
            tl = l;
          } else {
            df_acc(th, tl, h, l);
          }
        }
      }
      if (cmv[j] == 1) {
        kick(v[j], df_norm(th, tl), c);
        if (!last) coord_kick(x[j], v[j], dt);
      }
    }
    if (last) break;
  }
  __syncthreads();
  if (*s_fail) return;  // the last evaluation's packets never came
  // the final state, binned with the next shift by one thread per bead
  double* fin = reinterpret_cast<double*>(smem + L.fin);
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (pub[j] >= 0) {
      const double X = coord_to_double(x[j]), V = df_to_double(v[j]);
      const int s = base + cq[j];
      (ck[j] == 0 ? m.x[0] : (ck[j] == 1 ? m.y[0] : m.z[0]))[s] = X;
      (ck[j] == 0 ? m.vx : (ck[j] == 1 ? m.vy : m.vz))[s] = V;
      fin[ck[j] * T + cq[j]] = X;
      fin[(3 + ck[j]) * T + cq[j]] = V;
    }
  __syncthreads();
  for (int i = tid; i < T; i += nthr)
    if (m.moves[base + i] == 1) {
      const double X = fin[i], Y = fin[T + i], Z = fin[2 * T + i];
      const double VX = fin[3 * T + i], VY = fin[4 * T + i], VZ = fin[5 * T + i];
      if (a.deferred)
        bin.defer(base + i, X, Y, Z, VX, VY, VZ);
      else
        bin(X, Y, Z, VX, VY, VZ);
    }
  // refreshed bonds back to float64
  if (refreshed)
    each_bond([&](int, const CiliumDev&, int, int k) {
      const double l = df_to_double(dfloat{s_nl[k].x, s_nl[k].y});
      m.newlen[b0 + k] = l;
      m.oldlen[b0 + k] = l;
      m.diag[b0 + k] = df_to_double(dfloat{s_dg[k].x, s_dg[k].y});
    });
  // switch_logic for the cilia of this tile (the staged positions are the final ones)
  const Staged end{oa + (size_t)T * (a.n & 1), ob + (size_t)T * (a.n & 1), oc + (size_t)T * (a.n & 1)};
  for (int c = c0 + tid; c < c1; c += nthr) cilium_switch(m, a, c, a.t_end, base, end);
}

template <int NC, int HALVES, bool kFloat, typename Bin>
__global__ void __launch_bounds__(512) k_md_entries(MDState m, typename Bin::Cells c, MDStepArgs a) {
  md_entries_body<NC, HALVES, kFloat>(m, a, Bin{c, &a});
}

// the kernel for a tile width: owned coordinates per thread and threads per
// coordinate, double-float (m.df == 1) or float springs (2)
template <typename Bin>
const void* entries_kernel(const MDState& m) {
  const bool fl = m.df == 2;
  const int threads = md_entries_threads(m.tile);
  if (6 * m.tile <= threads && m.de_lanes == 8)
    return fl ? (const void*)k_md_entries<1, 2, true, Bin> : (const void*)k_md_entries<1, 2, false, Bin>;
  if (3 * m.tile <= threads)
    return fl ? (const void*)k_md_entries<1, 1, true, Bin> : (const void*)k_md_entries<1, 1, false, Bin>;
  return fl ? (const void*)k_md_entries<2, 1, true, Bin> : (const void*)k_md_entries<2, 1, false, Bin>;
}

size_t entries_smem(const MDState& m) {
  return EntSmem(m.tile, m.hmax, m.de_nent_max, m.de_ninc_max, m.df_nb_max).total;
}

template <typename Bin>
int launch_entries(const MDState& m, const typename Bin::Cells& c, const MDStepArgs& a, cudaStream_t s,
                   cudaError_t* st) {
  if (m.nslots == 0 || m.ntiles == 0) return 0;
  MDState mm = m;
  typename Bin::Cells cc = c;
  MDStepArgs aa = a;
  md_set_dt_pairs(aa);
  void* args[] = {&mm, &cc, &aa};
  const size_t smem = entries_smem(m);
  const void* k = entries_kernel<Bin>(m);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  *st = cudaLaunchCooperativeKernel(k, dim3(m.ntiles), dim3(md_entries_threads(m.tile)), args, smem, s);
  return 1;
}

}  // namespace

// entries, polls and a solo tile's list are dealt to all threads of the CTA
// (swimmer64 MD at 384 threads against 320 or 512, sums in any order: 123 us against 137)
int md_entries_threads(int tile) { return tile <= 64 ? 384 : 512; }

int launch_md_entries_f64cells(const MDState& m, const CellsF64& c, const MDStepArgs& a, cudaStream_t s,
                               cudaError_t* st) {
  return launch_entries<BinF64>(m, c, a, s, st);
}

int launch_md_entries_f32cells(const MDState& m, const CellsF32& c, const MDStepArgs& a, cudaStream_t s,
                               cudaError_t* st) {
  return launch_entries<BinF32>(m, c, a, s, st);
}

int md_entries_max_coresident_blocks(const MDState& m, int f32cells) {
  int dev = 0, sms = 0, per_sm = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t smem = entries_smem(m);
  if (smem > (size_t)optin) return 0;
  const void* k = f32cells ? entries_kernel<BinF32>(m) : entries_kernel<BinF64>(m);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, md_entries_threads(m.tile), smem);
  return per_sm * sms;
}

}  // namespace mpcd
