// MPCD fluid kernels: per-cell collision maps, fused collide + stream + bin,
// bead coupling, observables and the periodic counting-sort reorder.
//
// One MPC step of the fluid (src/libcilia/mpcd.cpp:140-247 collision,
// src/libcilia/fluid.cpp:152-167 + mpcd.cpp:340-394 streaming, mpcd.cpp:257-267
// binning) is two kernels:
//   cell_params : per cell, from the sums binned at the end of the previous step:
//                 u = P/M, E_rel = K - M u^2, thermostat factor sc, rotation R,
//                 and the affine collision map v' = A v + b (A = sc R, b = u - A u);
//                 clears the sums for the next step.
//   fluid_step  : per particle: v' = A v + b with the map of its shifted cell,
//                 x' = x + v' h with periodic wrap, bin into the next shifted cell
//                 (atomic sums).  One read and one write of the particle state.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "engine_internal.h"
#include "fluid_device.cuh"

namespace mpcd {

namespace {

constexpr int kThreads = 256;

// Persistent grid-stride sizing: a few resident CTAs per SM, every thread
// handling many particles, so per-thread set-up and reductions amortise.
inline int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  return sms;
}

inline int grid_for(long n, int threads = kThreads, int per_sm = 4) {
  long g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (per_sm <= 0) {
    // not persistent: -per_sm items per thread, short-lived CTAs, at most
    // kMaxShortCTAs of them (more rounds per thread beyond that: every CTA
    // ends with one float64 atomic into the same dissipated-energy word;
    // 128^3 boxes measured best at about 10 k CTAs, like 64^3 ones)
    constexpr long kMaxShortCTAs = 10240;
    const long per = (long)threads * (per_sm < 0 ? -per_sm : 1);
    g = (n + per - 1) / per;
    return (int)(g < 1 ? 1 : (g > kMaxShortCTAs ? kMaxShortCTAs : g));
  }
  const long cap = (long)sm_count() * per_sm;
  return (int)(g < cap ? g : cap);
}

// shifted cell along one axis from the cell index and the in-cell offset:
// floor(i + o + a) = i + (o >= 1 - a), compared in fixed point, high word then
// low word (32-bit integer instructions only)
__device__ __forceinline__ int shifted(int i, uint64_t o, uint64_t t, int L) {
  const uint32_t oh = (uint32_t)(o >> 32), th = (uint32_t)(t >> 32);
  const bool ge = oh > th || (oh == th && (uint32_t)o >= (uint32_t)t);
  const int s = i + (ge ? 1 : 0);
  return s == L ? 0 : s;
}

// cell index i back into [0, L)
__device__ __forceinline__ void wrap_cell(int& i, int L) {
  if ((unsigned)i < (unsigned)L) return;
  i += i < 0 ? L : -L;
  if ((unsigned)i >= (unsigned)L) {  // more than one box away
    i %= L;
    if (i < 0) i += L;
  }
}

// an unwrapped coordinate (any finite value below about 1e9), counted from cell i0, as
// cell and offset
__device__ __forceinline__ void split_coord(double x, int L, int& i, uint64_t& o, unsigned& bad, int i0 = 0) {
  if (!(x > -1.0e9 && x < 1.0e9)) {  // non-finite: keep the particle in its cell and report
    o = kOffOne / 2;
    bad |= kErrCellRange;
    return;
  }
  const double f = floor(x);
  const double d = x - f;
  i = (int)f;
  o = 0;
  if (d >= 1.0)
    i += 1;  // x was a tiny negative number: x - floor(x) rounded to 1
  else
    o = offset_from_double(d);
  i = (i + i0) % L;
  if (i < 0) i += L;
}

// streams one coordinate by v h and wraps it into the box; the general form
// takes displacements of four cells and more
__device__ __forceinline__ void stream_coord(int& i, uint64_t& o, double v, const StepArgs& a, int L, unsigned& bad) {
  int c;
  if (stream_fixed(o, c, v, a.xh)) {
    i += c;
    wrap_cell(i, L);
  } else {
    const int i0 = i;  // the offset alone: added to a cell index it would lose the index's bits
    split_coord(fma(v, a.h, offset_to_double(o)), L, i, o, bad, i0);
  }
}

// 1/n for the particle counts of bead-free cells, in units of 2^-62
struct InvTable {
  int64_t x[256];
};
constexpr InvTable make_inv_table() {
  InvTable t{};
  for (int i = 1; i < 256; ++i) t.x[i] = (int64_t)(((1ull << 62) + (unsigned)i / 2) / (unsigned)i);
  return t;
}
__device__ const InvTable g_inv_n = make_inv_table();

// Free-running rotation axis of the float64 path in units of 2^-60: the direction
// drawn in float (cos theta = 2u - 1, phi = 2 pi u', as generate_collision_matrix,
// src/libcilia/mpcd.cpp:269-284), normalised to more than float64 precision so that
// the rotation is orthogonal to it.
__device__ __forceinline__ void draw_axis_fixed(uint64_t seed, uint64_t step, uint32_t cid, int64_t* r) {
  const u32x4 q = draw4(seed, step, kStreamCell, cid, 0u);
  const float ct = 2.0f * u01_flt(q.y) - 1.0f;
  const float st = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
  float sp, cp;
  sincospif(2.0f * u01_flt(q.x), &sp, &cp);
  r[0] = axis_fixed(st * cp);
  r[1] = axis_fixed(st * sp);
  r[2] = axis_fixed(ct);
  axis_normalise(r);
}
// the same axis as the nearest float64 numbers
__device__ __forceinline__ void draw_axis_f64(uint64_t seed, uint64_t step, uint32_t cid, double& rx, double& ry,
                                              double& rz) {
  int64_t r[3];
  draw_axis_fixed(seed, step, cid, r);
  rx = from_fixed(r[0], kAxisBits);
  ry = from_fixed(r[1], kAxisBits);
  rz = from_fixed(r[2], kAxisBits);
}

// The thermostat factor sqrt(g / (erel / 2)) = 2g / sqrt(2g erel): one
// reciprocal square root in place of a float64 division and square root;
// outside the float range the direct form.
__device__ __forceinline__ double thermostat_factor(double g, double erel) {
  const double q = 2.0 * g, x = q * erel;
  return (x > 1e-30 && x < 1e30) ? q * rsqrt_f64(x) : sqrt(g / (erel * 0.5));
}
// the same for a float g > 0, its conversion and the range check on the bit
// patterns (they are float64 instructions otherwise)
__device__ __forceinline__ double thermostat_factor(float g, double erel) {
  const uint32_t gb = __float_as_uint(g);
  const double q = __hiloint2double((int)((gb >> 3) + (897u << 20)), (int)(gb << 29));  // 2 g
  const double x = q * erel;
  if ((uint32_t)__double2hiint(x) - (923u << 20) >= (200u << 20)) return sqrt((double)g / (erel * 0.5));
  return q * rsqrt_f64(x);
}

// A cell on its way to the map: its sums (virtual particles included), the
// real particles' momentum and mass, and the sphere that cuts it.
struct CellSums {
  double4 s;
  double M;
  int num;
  int sk;  // rigid sphere whose surface cuts the cell, or -1
  double rel[3], preal[3], mreal;
};

// Virtual particles up to rho = 10 in cells cut by a sphere's surface (moving
// with it) or in the wall layers.  Not inlined, like the float64 map below:
// the common path fits the instruction cache better without them.
__device__ __noinline__ void add_virtual(CellSums& t, long cid, const StepArgs& a) {
  const bool wall = a.walls && wall_layer_cell(a.box, cid);
  if (a.sph.n && !wall) {
    const int L0 = a.box.L[0], L1 = a.box.L[1];
    t.sk = sphere_cut_cell(a.sph, a.box, a.a_cur, (int)(cid % L0), (int)((cid / L0) % L1), (int)(cid / ((long)L0 * L1)),
                           t.rel);
  }
  if (t.sk < 0 && !wall) return;
  const int dm = 10 - t.num;
  double pv[3];
  if (t.sk >= 0) {
    t.preal[0] = t.s.x;
    t.preal[1] = t.s.y;
    t.preal[2] = t.s.z;
    t.mreal = t.M;
    sphere_virtual(a.sph.s[t.sk], t.rel, dm, a.seed, a.step, (uint32_t)cid, a.inj_virt, pv);
  } else if (a.inj_virt) {
    pv[0] = a.inj_virt[3 * cid];
    pv[1] = a.inj_virt[3 * cid + 1];
    pv[2] = a.inj_virt[3 * cid + 2];
  } else {
    virtual_momentum(a.seed, a.step, (uint32_t)cid, dm, pv);
  }
  t.s.x += pv[0];
  t.s.y += pv[1];
  t.s.z += pv[2];
  t.s.w += (pv[0] * pv[0] + pv[1] * pv[1] + pv[2] * pv[2]) / dm;
  t.M += dm;
  t.num += dm;
}

// the Gamma draw of a cell of num > 1 particles, injected or generated
__device__ __forceinline__ double injected_gamma(const StepArgs& a, long cid, unsigned& errbits) {
  const double g = a.inj_gamma[cid];
  if (g < 0) {
    errbits |= kErrGammaMissing;
    return 0.0;
  }
  return g;
}

// The map in float64, for cells whose numbers do not fit the fixed-point form
// and for cells cut by a sphere, whose impulse follows from it.
__device__ __noinline__ unsigned map_f64(const CellSums& t, long cid, float gf, uint64_t* out, const StepArgs& a) {
  unsigned errbits = 0;
  const double4 s = t.s;
  const double dinv = 1.0 / t.M;
  const double ux = s.x * dinv, uy = s.y * dinv, uz = s.z * dinv;
  const double erel = s.w - (ux * s.x + uy * s.y + uz * s.z);  // K - M u^2
  double sc = 1.0;
  if (erel > 0 && t.num > 1) sc = thermostat_factor(a.inj_gamma ? injected_gamma(a, cid, errbits) : (double)gf, erel);
  double rx, ry, rz;
  if (a.inj_axis) {
    rx = a.inj_axis[3 * cid + 0];
    ry = a.inj_axis[3 * cid + 1];
    rz = a.inj_axis[3 * cid + 2];
  } else {
    draw_axis_f64(a.seed, a.step, (uint32_t)cid, rx, ry, rz);
  }
  if (t.sk >= 0) {
    // the real particles' momentum after the collision is A P + M b; what
    // they gained came from the virtual particles, i.e. from the sphere
    double A[9], b[3], J[3];
    map_from_axis(sc, rx, ry, rz, ux, uy, uz, A, b);
    for (int q = 0; q < 3; ++q)
      J[q] = t.preal[q] -
             (A[3 * q] * t.preal[0] + A[3 * q + 1] * t.preal[1] + A[3 * q + 2] * t.preal[2] + t.mreal * b[q]);
    add_impulse(a.sph.acc + 6 * t.sk, t.rel, J);
  }
  const double d[7] = {sc, rx, ry, rz, ux, uy, uz};
  out[0] = kMapF64;
  for (int q = 0; q < 7; ++q) out[1 + q] = f64_bits(d[q]);
  for (int q = 8; q < 12; ++q) out[q] = 0;
  return errbits;
}

// The collision map of one cell (MPCD::next_tstep, src/libcilia/mpcd.cpp:
// 140-247) as twelve words (fixed_collide.cuh): in fixed point when the
// cell's numbers fit, else as float64 factor, axis and mean velocity, in two
// parts that need nothing of each other.  The cell's sum m v^2 before the
// collision goes to the sums of ke or ke_rest.
//
// The sums' part: factor and mean velocity.  False if the cell takes the
// float64 form, whose words it has written to par.
__device__ __forceinline__ bool cell_factor(double4 s, uint32_t w, long cid, const StepArgs& a, double* par, int64_t& sc,
                                            int& scale, int64_t* u, EnergySum& ke, double& ke_rest, unsigned& errbits, bool& gfail) {
  const int nf = cnt_fluid(w), nb = cnt_beads(w);
  int num = nf + nb, sk = -1;
  double M = (double)num;
  if (nb) M = (double)nf + (double)nb * a.bead_mass;
  CellSums t;
  if ((a.sph.n || a.walls) && num < 10) {
    t.s = s;
    t.M = M;
    t.num = num;
    t.sk = -1;
    add_virtual(t, cid, a);
    s = t.s;
    M = t.M;
    num = t.num;
    sk = t.sk;
  }
  // the random part first: it needs the count alone, and the sums are still on
  // their way
  float gf = 0.f;
  if (num > 1 && !a.inj_gamma) gf = gamma_mt(num, a.seed, a.step, (uint32_t)cid, &gfail);
  bool fit = sk < 0;
  if (a.inj_axis) {
    int64_t r;
#pragma unroll
    for (int q = 0; q < 3; ++q) fit = to_fixed<60, 1>(a.inj_axis[3 * cid + q], r) && fit;
  }
  // dissipated energy (src/libcilia/mpcd.cpp:166-168, 232-234, 243-246): every
  // cell adds sum m v^2 before the collision here, and every particle
  // subtracts its m v'^2 after it (fluid_step, bead_collide), so the total
  // matches the reference's bookkeeping including the rounding of its
  // rotation constants
  int64_t kin = 0;
  const int ebits = kinetic_fixed(s.w, kin);
  if (ebits) {
    energy_add_cell(ke, kin, ebits);
  } else {
    ke_rest += s.w;
    fit = false;
  }
  int64_t inv = 0, top = 0, erel = 0;
  sc = 1ll << kAxisBits;
  scale = 0;
  if (nb == 0 && num < 256) {
    inv = __ldg(g_inv_n.x + num);  // M = num without beads
    top = mean_top(ebits, num);
  } else {
    fit = to_fixed<62, 0>(1.0 / M, inv) && fit;
    top = mean_top(ebits, M);
  }
  if (fit) {
    const double p[3] = {s.x, s.y, s.z};
    fit = cell_energy(p, kin, ebits, inv, top, num == 1, u, erel);
    if (fit && num > 1) {
      const double e = from_fixed(erel, ebits);
      double f;
      if (a.inj_gamma) {
        const double g = injected_gamma(a, cid, errbits);
        f = thermostat_factor(g, e);
        fit = g < kGammaMax;
      } else {
        f = thermostat_factor(gf, e);
        fit = gf < kGammaMax;
      }
      const int hi = __double2hiint(f);
      if (hi >= 1024 << 20) {  // 2 and more: a quarter of it, where the sums leave room
#pragma unroll
        for (int q = 0; q < 3; ++q) fit = fit && u[q] < kMeanMaxHot && u[q] > -kMeanMaxHot;
        f = __hiloint2double(hi - (2 << 20), __double2loint(f));
        scale = 2;
      } else {
        fit = true;
      }
      fit = to_fixed<60, 1>(f, sc) && fit;
    }
  }
  if (!fit) {
    t.s = s;
    t.M = M;
    t.num = num;
    t.sk = sk;
    uint64_t o[12];
    errbits |= map_f64(t, cid, gf, o, a);
    ulonglong2* pm = reinterpret_cast<ulonglong2*>(par);
#pragma unroll
    for (int q = 0; q < 6; ++q) pm[q] = make_ulonglong2(o[2 * q], o[2 * q + 1]);
  }
  return fit;
}
// The axis' part: the rotation.
__device__ __forceinline__ void cell_rotation(long cid, const StepArgs& a, int64_t* R) {
  int64_t r[3] = {0, 0, 0};
  if (a.inj_axis) {
#pragma unroll
    for (int q = 0; q < 3; ++q) (void)to_fixed<60, 1>(a.inj_axis[3 * cid + q], r[q]);  // cell_factor minds the rest
  } else {
    draw_axis_fixed(a.seed, a.step, (uint32_t)cid, r);
  }
  rotation_fixed(r, kCosAlpha, kSinAlpha, R);
}
__device__ __forceinline__ void store_row(double* par, int i, const int64_t* row, int64_t sc, int scale, const int64_t* u) {
  uint64_t w[4];
  map_row(i, row, sc, u, w, scale);
  ulonglong2* p = reinterpret_cast<ulonglong2*>(par + 4 * i);
  p[0] = make_ulonglong2(w[0], w[1]);
  p[1] = make_ulonglong2(w[2], w[3]);
}

// The whole map by one thread.
__device__ __forceinline__ void collision_map(double4 s, uint32_t w, long cid, const StepArgs& a, double* par, EnergySum& ke,
                                              double& ke_rest, unsigned& errbits, bool& gfail) {
  int64_t R[9], u[3], sc;
  int scale;
  if (!cell_factor(s, w, cid, a, par, sc, scale, u, ke, ke_rest, errbits, gfail)) return;
  cell_rotation(cid, a, R);
#pragma unroll
  for (int i = 0; i < 3; ++i) store_row(par, i, R + 3 * i, sc, scale, u);
}

// The block's sum of fixed-point energies (units of 2^-bits) and a float64 rest,
// added to *dst with the given sign by the warp that comes last: no barrier at
// the end of a block, whose other warps would wait there for the slowest (0.8 to
// 1.1 of 12 cycles per instruction before).
struct BlockEnergy {
  double sum;
  unsigned warps;
};
__device__ __forceinline__ void energy_begin(BlockEnergy& b) {
  if (threadIdx.x == 0) {
    b.sum = 0.0;
    b.warps = 0;
  }
  __syncthreads();
}
__device__ __forceinline__ void energy_end(BlockEnergy& b, EnergySum ke, int bits, double rest, double sign, double* dst) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t lo = __shfl_xor_sync(0xffffffffu, ke.lo, o);
    energy_add(ke, lo, __shfl_xor_sync(0xffffffffu, ke.hi, o));
  }
  if (rest != 0.0) atomicAdd(&b.sum, rest);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&b.sum, energy_value(ke, bits));
    __threadfence_block();
    if (atomicAdd(&b.warps, 1u) == (blockDim.x >> 5) - 1) {
      __threadfence_block();
      const double tot = *reinterpret_cast<volatile double*>(&b.sum);
      if (tot != 0.0) atomicAdd(dst, sign * tot);
    }
  }
}

// ============================================================== float64 ===

// Bound by latency: the generator's Gamma loop and the map are one long chain
// per cell (1890 instructions, 12 cycles each at six warps per scheduler); the
// float64 form kept that pipe 73 % busy.  64-thread blocks fill the SMs in the
// finest steps (24 warps with 80 registers; five blocks of 128: 36 us, eight
// with 64 registers: 43).  64^3 cells 48 to 31 us, 80 x 71 x 89 96 to 50.  For
// boxes beyond one wave of the pair form below.
constexpr int kCellThreads = 64;
__global__ void __launch_bounds__(kCellThreads, 12) k_cell_params_f64(CellsF64 c, StepArgs a) {
  __shared__ BlockEnergy s_e;
  energy_begin(s_e);
  chain_begin();
  EnergySum ke;
  double ke_rest = 0.0;
  unsigned errbits = 0;
  bool gfail = false;
  constexpr int kU = 2;
  const long stride = (long)gridDim.x * blockDim.x;
  for (long cb = (long)blockIdx.x * blockDim.x + threadIdx.x; cb < c.ncell; cb += kU * stride) {
    uint32_t w[kU];
    double4 sm[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long cid = cb + u * stride;
      w[u] = cid < c.ncell ? __ldcg(c.cnt + cid) : 0u;
      sm[u] = make_double4(0.0, 0.0, 0.0, 0.0);
      if (cid < c.ncell) {
        const double2* p = reinterpret_cast<const double2*>(c.sum + cid);
        const double2 lo = __ldcg(p), hi = __ldcg(p + 1);
        sm[u] = make_double4(lo.x, lo.y, hi.x, hi.y);
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (!w[u]) continue;
      const long cid = cb + u * stride;
      c.sum[cid] = make_double4(0.0, 0.0, 0.0, 0.0);
      c.cnt[cid] = 0u;
      if (a.premapped && cnt_beads(w[u]) > 0) continue;  // mapped by k_bead_maps_f64
      collision_map(sm[u], w[u], cid, a, c.par + 12 * cid, ke, ke_rest, errbits, gfail);
    }
  }
  if (gfail) errbits |= kErrGammaLoop;
  if (errbits) atomicOr(a.err, errbits);
  energy_end(s_e, ke, kCellEnergyBits, ke_rest, 1.0, a.diss);
}

// The same by pairs of warps, 32 cells a CTA: one warp makes count, sums, Gamma
// draw and thermostat factor, the other axis and rotation, and both the rows of
// the map: half the chain, for twice the warps.  That pays while all pairs are
// on the SMs at once (10 CTAs of 92 registers each): per step 36^3 cells 29.2
// us against 29.9, 32^3 24.9 / 25.3, the channel (24 x 21 x 37) 31.1 / 32.8, 8^3
// 8.8 / 10.2; beyond, the one-thread form does: 40^3 36.5 against 38.8, 64^3
// cells 29 us against 41.
constexpr int kPairCTAs = 10;  // per SM
__global__ void __launch_bounds__(kCellThreads, kPairCTAs) k_cell_pairs_f64(CellsF64 c, StepArgs a) {
  __shared__ BlockEnergy s_e;
  __shared__ int64_t s_R[2][3][32], s_u[2][3][32], s_sc[2][32];
  __shared__ int s_fits[2][32];  // 1 + the map's scale, or 0
  energy_begin(s_e);
  chain_begin();
  const int lane = threadIdx.x & 31;
  const bool sums = threadIdx.x < 32;  // the warp of the sums; the other makes the rotations
  EnergySum ke;
  double ke_rest = 0.0;
  unsigned errbits = 0;
  bool gfail = false;
  int b = 0;  // two sets of words: one barrier per round
  for (long c0 = 32l * blockIdx.x; c0 < c.ncell; c0 += 32l * gridDim.x, b ^= 1) {
    const long cid = c0 + lane;
    double* par = c.par + 12 * cid;
    int64_t R[9], u[3] = {0, 0, 0}, sc = 0;
    if (sums) {
      int fits = 0, scale = 0;
      if (cid < c.ncell) {
        const uint32_t w = __ldcg(c.cnt + cid);
        const double2* p = reinterpret_cast<const double2*>(c.sum + cid);
        const double2 lo = __ldcg(p), hi = __ldcg(p + 1);
        if (w) {
          c.sum[cid] = make_double4(0.0, 0.0, 0.0, 0.0);
          c.cnt[cid] = 0u;
          if (!(a.premapped && cnt_beads(w) > 0))  // else mapped by k_bead_maps_f64
            fits = cell_factor(make_double4(lo.x, lo.y, hi.x, hi.y), w, cid, a, par, sc, scale, u, ke, ke_rest, errbits, gfail)
                       ? 1 + scale
                       : 0;
        }
      }
      s_fits[b][lane] = fits;
      s_sc[b][lane] = sc;
#pragma unroll
      for (int q = 0; q < 3; ++q) s_u[b][q][lane] = u[q];
    } else if (cid < c.ncell) {
      cell_rotation(cid, a, R);
#pragma unroll
      for (int q = 0; q < 3; ++q) s_R[b][q][lane] = R[q];  // the first row goes to the other warp
    }
    __syncthreads();
    if (!s_fits[b][lane]) continue;
    const int scale = s_fits[b][lane] - 1;
    if (sums) {
#pragma unroll
      for (int q = 0; q < 3; ++q) R[q] = s_R[b][q][lane];
      store_row(par, 0, R, sc, scale, u);
    } else {
      sc = s_sc[b][lane];
#pragma unroll
      for (int q = 0; q < 3; ++q) u[q] = s_u[b][q][lane];
      store_row(par, 1, R + 3, sc, scale, u);
      store_row(par, 2, R + 6, sc, scale, u);
    }
  }
  if (gfail) errbits |= kErrGammaLoop;
  if (errbits) atomicOr(a.err, errbits);
  energy_end(s_e, ke, kCellEnergyBits, ke_rest, 1.0, a.diss);
}

// Walls along z (NOSLIP / SLIP, src/libcilia/mpcd.cpp:346-376): the channel is
// 0 <= z <= Lz - 1; a particle that crossed a wall during the streaming step
// is reflected.  Returns the (possibly changed) unwrapped z.
__device__ __forceinline__ void wall_bounce(int walls, double ztop, double& x, double& y, double& z, double& vx,
                                            double& vy, double& vz) {
  if (z > ztop) {
    if (walls == 1) {
      double t2 = (z - ztop) / vz;
      vx = -vx;
      vy = -vy;
      vz = -vz;
      x += 2.0 * t2 * vx;
      y += 2.0 * t2 * vy;
      z += 2.0 * t2 * vz;
    } else {
      vz = -vz;
      z = -z + ztop * 2.0;
    }
  }
  if (z < 0) {
    double t2 = z / vz;
    vx = -vx;
    vy = -vy;
    vz = -vz;
    x += vx * 2.0 * t2;
    y += vy * 2.0 * t2;
    z += vz * 2.0 * t2;
  }
}

// kBoundary of the fluid pass: a periodic box; walls along z; rigid spheres
// (with or without walls)
constexpr int kPeriodic = 0, kWalled = 1, kSpheres = 2;

// A particle whose numbers do not fit the fixed-point form: collision, energy
// (returned), streaming and kick in float64 (no inlining: it would hold
// registers of the common path).
struct SlowParticle {
  double v[3], K;
  int i[3];
  uint64_t o[3];
  unsigned bad;
};
__device__ __forceinline__ double square_f64(const double* v) { return v[0] * v[0] + v[1] * v[1] + v[2] * v[2]; }
// the kick of a body force, and the energy that is binned
__device__ __forceinline__ void kick_f64(SlowParticle& t, const StepArgs& a) {
  if (a.gkick != 0.0) t.v[0] += a.gkick;
  t.K = square_f64(t.v);
}
__device__ __noinline__ double slow_particle(SlowParticle& t, const double* par, const StepArgs& a) {
  apply_map_f64(par, t.v[0], t.v[1], t.v[2]);
  const double k = square_f64(t.v);
  t.bad = 0;
  for (int d = 0; d < 3; ++d) stream_coord(t.i[d], t.o[d], t.v[d], a, a.box.L[d], t.bad);
  kick_f64(t, a);
  return k;
}
// The same with walls or rigid spheres: bounce-back in unwrapped float64
// coordinates; par is null if the collision is done.
__device__ __noinline__ double bounced_particle(SlowParticle& t, const double* par, const StepArgs& a) {
  double k = 0.0;
  if (par) {
    apply_map_f64(par, t.v[0], t.v[1], t.v[2]);
    k = square_f64(t.v);
  }
  double X[3];
  for (int d = 0; d < 3; ++d) X[d] = t.i[d] + offset_to_double(t.o[d]);
  if (!(a.sph.n > 0 && sphere_bounce(a.sph, a.box, a.h, X, t.v)))
    for (int d = 0; d < 3; ++d) X[d] += t.v[d] * a.h;
  if (a.walls) wall_bounce(a.walls, (double)(a.box.L[2] - 1), X[0], X[1], X[2], t.v[0], t.v[1], t.v[2]);
  t.bad = 0;
  for (int d = 0; d < 3; ++d) split_coord(X[d], a.box.L[d], t.i[d], t.o[d], t.bad);
  kick_f64(t, a);
  return k;
}

// Adds the four values of a particle to its cell's sums.  The lanes of a quad
// exchange their values first (a 4 x 4 transpose) so that each instruction adds
// the 32 contiguous bytes of eight cells instead of one word of up to 32: the
// L2 takes a quarter of the requests (80 x 71 x 89 x 10: 206 to 173 us).
__device__ __forceinline__ void add_to_cell(double* sum, uint32_t cell, double v0, double v1, double v2, double v3, bool whole) {
  if (!whole) {
    double* p = sum + 4 * (size_t)cell;
    atomicAdd(p + 0, v0);
    atomicAdd(p + 1, v1);
    atomicAdd(p + 2, v2);
    atomicAdd(p + 3, v3);
    return;
  }
  const int q = threadIdx.x & 3;
  const bool q0 = q & 1, q1 = q & 2;
  const double a0 = __shfl_xor_sync(0xffffffffu, q0 ? v0 : v1, 1), a1 = __shfl_xor_sync(0xffffffffu, q0 ? v2 : v3, 1);
  const double w0 = q0 ? a0 : v0, w1 = q0 ? v1 : a0, w2 = q0 ? a1 : v2, w3 = q0 ? v3 : a1;
  const double b0 = __shfl_xor_sync(0xffffffffu, q1 ? w0 : w2, 2), b1 = __shfl_xor_sync(0xffffffffu, q1 ? w1 : w3, 2);
  // component q of the quad's particles 0 to 3
  const double x[4] = {q1 ? b0 : w0, q1 ? b1 : w1, q1 ? w2 : b0, q1 ? w3 : b1};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    atomicAdd(sum + 4 * (size_t)__shfl_sync(0xffffffffu, cell, j, 4) + q, x[j]);
}

// I: particle index type (32-bit whenever the particle count allows).
// Collision, kinetic energy, streaming, wrap and the comparison with the grid
// shift run in 64-bit fixed point (fixed_collide.cuh, fixed_offset.cuh); float64
// appears only as the stored velocity and in the atomic sums, which the L2
// adds.  Nothing is saturated (issue 61 %, the L1 data path 69 %); 32 warps of 64
// registers per SM did best (24 of 80: 107 us against 98), and fetching the next
// particle ahead brought nothing.  64^3 x 10: 116 us with the collision in float64,
// 94 now; 80 x 71 x 89 x 10: 234, 171; 32^3 x 10: 20.
// Walls and spheres are instantiations of their own; between walls only a
// particle that would leave the channel takes the bounce-back.
constexpr int kFluidThreads = 128;
template <typename I, int kBoundary>
__global__ void __launch_bounds__(kFluidThreads, 8) k_fluid_step_f64(FluidF64 f, CellsF64 c, StepArgs a) {
  const int Lx = a.box.L[0], Ly = a.box.L[1], Lz = a.box.L[2];
  const bool kick = a.xkick != 0;  // what does not fit is in vmax
  const I n = (I)f.n;
  __shared__ BlockEnergy s_e;
  energy_begin(s_e);
  chain_begin();
  EnergySum ke;  // sum of v'^2, and the rest
  double ke_rest = 0.0;
  unsigned bad = 0;
  for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (I)gridDim.x * blockDim.x) {
    const uint32_t cp = f.cell[i];
    int ix = cell_x(cp), iy = cell_y(cp), iz = cell_z(cp);
    uint64_t ox = f.ox[i], oy = f.oy[i], oz = f.oz[i];
    double vx = f.vx[i], vy = f.vy[i], vz = f.vz[i];
    // collision with the map of the shifted cell (box cells < 2^30: 32-bit index)
    const uint32_t cid =
        (uint32_t)shifted(ix, ox, a.xta_cur[0], Lx) +
        (uint32_t)Lx * ((uint32_t)shifted(iy, oy, a.xta_cur[1], Ly) + (uint32_t)Ly * (uint32_t)shifted(iz, oz, a.xta_cur[2], Lz));
    const double* par = c.par + 12 * (size_t)cid;
    uint64_t m[12];
    {
      const ulonglong2* p = reinterpret_cast<const ulonglong2*>(par);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const ulonglong2 t = p[q];
        m[2 * q] = t.x;
        m[2 * q + 1] = t.y;
      }
    }
    int64_t x[3] = {0, 0, 0}, y[3];
    bool fit = to_fixed<58, 4>(vx, x[0]) && to_fixed<58, 4>(vy, x[1]) && to_fixed<58, 4>(vz, x[2]) &&
               (uint32_t)(m[0] >> 32) != (uint32_t)(kMapF64 >> 32);
    apply_words(m, x, y);
    const uint32_t lim = (uint32_t)a.xstep.vmax;
#pragma unroll
    for (int q = 0; q < 3; ++q) fit = fit && (uint32_t)(y[q] >> 32) + lim < 2 * lim;
    double K;
    if (fit) {
      const Limbs wx = split_limbs(y[0] << 2), wy = split_limbs(y[1] << 2), wz = split_limbs(y[2] << 2);
      const int64_t k2 = square_words(wx, wy, wz);
      energy_add(ke, (uint64_t)k2, 0u);
      if (kick) {
        const int64_t yk = y[0] + a.xkick;
        K = from_fixed(square_words(split_limbs(yk << 2), wy, wz), kSquareBits);
        vx = from_fixed(yk, kOutBits);
      } else {
        K = from_fixed(k2, kSquareBits);
        vx = from_fixed(y[0], kOutBits);
      }
      vy = from_fixed(y[1], kOutBits);
      vz = from_fixed(y[2], kOutBits);
      bool free_path = kBoundary != kSpheres;
      if (kBoundary != kSpheres) {
        int cx, cy, cz;
        uint64_t nx = ox, ny = oy, nz = oz;
        stream_words(nx, cx, wx, a.xstep);
        stream_words(ny, cy, wy, a.xstep);
        stream_words(nz, cz, wz, a.xstep);
        // between walls z stays in [0, Lz - 1], whose upper end is a cell's edge
        if (kBoundary == kWalled) free_path = iz + cz >= 0 && (iz + cz < Lz - 1 || (iz + cz == Lz - 1 && nz == 0));
        if (free_path) {
          ox = nx;
          oy = ny;
          oz = nz;
          ix += cx;
          iy += cy;
          iz += cz;
          wrap_cell(ix, Lx);
          wrap_cell(iy, Ly);
          if (kBoundary == kPeriodic) wrap_cell(iz, Lz);
        }
      }
      if (kBoundary != kPeriodic && !free_path) {
        SlowParticle t{{kick ? from_fixed(y[0], kOutBits) : vx, vy, vz}, 0.0, {ix, iy, iz}, {ox, oy, oz}, 0u};
        bounced_particle(t, nullptr, a);
        K = t.K;
        vx = t.v[0];
        vy = t.v[1];
        vz = t.v[2];
        ix = t.i[0];
        iy = t.i[1];
        iz = t.i[2];
        ox = t.o[0];
        oy = t.o[1];
        oz = t.o[2];
        bad |= t.bad;
      }
    } else {
      SlowParticle t{{vx, vy, vz}, 0.0, {ix, iy, iz}, {ox, oy, oz}, 0u};
      ke_rest += kBoundary == kPeriodic ? slow_particle(t, par, a) : bounced_particle(t, par, a);
      K = t.K;
      vx = t.v[0];
      vy = t.v[1];
      vz = t.v[2];
      ix = t.i[0];
      iy = t.i[1];
      iz = t.i[2];
      ox = t.o[0];
      oy = t.o[1];
      oz = t.o[2];
      bad |= t.bad;
    }
    // bin with the next shift
    const uint32_t cn =
        (uint32_t)shifted(ix, ox, a.xta_next[0], Lx) +
        (uint32_t)Lx * ((uint32_t)shifted(iy, oy, a.xta_next[1], Ly) + (uint32_t)Ly * (uint32_t)shifted(iz, oz, a.xta_next[2], Lz));
    const bool whole = (threadIdx.x & ~31u) + 31u - threadIdx.x + i < n;  // all lanes of the warp are here
    add_to_cell(reinterpret_cast<double*>(c.sum), cn, vx, vy, vz, K, whole);
    atomicAdd(c.cnt + cn, 1u);
    f.cell[i] = pack_cell(ix, iy, iz);
    f.ox[i] = ox;
    f.oy[i] = oy;
    f.oz[i] = oz;
    f.vx[i] = vx;
    f.vy[i] = vy;
    f.vz[i] = vz;
  }
  if (bad) atomicOr(a.err, bad);
  energy_end(s_e, ke, kSquareBits, ke_rest, -1.0, a.diss);
}

__global__ void k_bin_fluid_f64(FluidF64 f, CellsF64 c, StepArgs a) {
  const int Lx = a.box.L[0], Ly = a.box.L[1], Lz = a.box.L[2];
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t cp = f.cell[i];
    const long cid = shifted(cell_x(cp), f.ox[i], a.xta_cur[0], Lx) +
                     (long)Lx * (shifted(cell_y(cp), f.oy[i], a.xta_cur[1], Ly) + (long)Ly * shifted(cell_z(cp), f.oz[i], a.xta_cur[2], Lz));
    const double vx = f.vx[i], vy = f.vy[i], vz = f.vz[i];
    double* sp = reinterpret_cast<double*>(c.sum + cid);
    atomicAdd(sp + 0, vx);
    atomicAdd(sp + 1, vy);
    atomicAdd(sp + 2, vz);
    atomicAdd(sp + 3, vx * vx + vy * vy + vz * vz);
    atomicAdd(c.cnt + cid, 1u);
  }
}

__global__ void k_bead_collide_f64(MDState m, CellsF64 c, StepArgs a) {
  double ke_after = 0.0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      atomicOr(a.err, kErrCellRange);
      continue;
    }
    double vx = m.vx[s], vy = m.vy[s], vz = m.vz[s];
    apply_map_f64(c.par + 12 * cid, vx, vy, vz);
    ke_after += a.bead_mass * (vx * vx + vy * vy + vz * vz);
    m.vx[s] = vx;
    m.vy[s] = vy;
    m.vz[s] = vz;
  }
  const double tot = block_sum_f64(ke_after);
  if (threadIdx.x == 0 && tot != 0.0) atomicAdd(a.diss, -tot);
}

__global__ void k_bin_beads_f64(MDState m, CellsF64 c, StepArgs a) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      atomicOr(a.err, kErrCellRange);
      continue;
    }
    const double mb = a.bead_mass, vx = m.vx[s], vy = m.vy[s], vz = m.vz[s];
    double* sp = reinterpret_cast<double*>(c.sum + cid);
    atomicAdd(sp + 0, vx * mb);
    atomicAdd(sp + 1, vy * mb);
    atomicAdd(sp + 2, vz * mb);
    atomicAdd(sp + 3, mb * (vx * vx + vy * vy + vz * vz));
    atomicAdd(c.cnt + cid, 1u << 16);
  }
}

__global__ void k_observables_f64(FluidF64 f, MDState m, double bead_mass, double* out) {
  double px = 0, py = 0, pz = 0, e = 0, n = 0, ms = 0, ef = 0, nf = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const double vx = f.vx[i], vy = f.vy[i], vz = f.vz[i];
    const double v2 = vx * vx + vy * vy + vz * vz;
    px += vx;
    py += vy;
    pz += vz;
    e += v2;
    ef += v2;
    n += 1.0;
    ms += 1.0;
    nf += 1.0;
  }
  for (long s = (long)blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += (long)gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const double vx = m.vx[s], vy = m.vy[s], vz = m.vz[s];
    px += bead_mass * vx;
    py += bead_mass * vy;
    pz += bead_mass * vz;
    e += bead_mass * (vx * vx + vy * vy + vz * vz);
    n += 1.0;
    ms += bead_mass;
  }
  double vals[8] = {px, py, pz, e, n, ms, ef, nf};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double t = block_sum_f64(vals[k]);
    if (threadIdx.x == 0) atomicAdd(out + k, t);
  }
}

// Observables from the cell sums binned at the end of the last step (float64
// path): the sums hold every moving particle's m v and m v^2 once, so their
// totals are the fluid + bead momentum and energy, read from 36 B per cell
// instead of 24 B per particle.  The beads' own energy (moving beads, a few
// thousand) is summed beside it to split off the fluid's.  Per-block
// partials, added in block order by the last block to finish (no memset, no
// float atomics into the result); out = {P x, y, z, sum m v^2, n, mass,
// fluid sum v^2, fluid n, dissipated energy, error bits}, device memory or a
// mapped page-locked host slot (then no copy follows the kernel).
// GB300 runs float64 adds at a small fraction of its float32 rate, so the
// counts are summed as integers and the grid is one block per SM (fewer
// block reductions); four cells' loads are in flight per thread.
__global__ void __launch_bounds__(kThreads) k_observables_cells_f64(CellsF64 c, MDState m, double bead_mass,
                                                                    const double* diss, const unsigned* err,
                                                                    double* part, unsigned* counter, double* out) {
  double px = 0, py = 0, pz = 0, e = 0, eb = 0;
  uint32_t nf = 0, nb = 0;
  const long stride = (long)gridDim.x * blockDim.x;
  long cid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  for (; cid + 3 * stride < c.ncell; cid += 4 * stride) {
    uint32_t w[4];
    double4 s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = c.cnt[cid + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = c.sum[cid + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (w[u] != 0) {
        px += s[u].x;
        py += s[u].y;
        pz += s[u].z;
        e += s[u].w;
        nf += (uint32_t)cnt_fluid(w[u]);
        nb += (uint32_t)cnt_beads(w[u]);
      }
  }
  for (; cid < c.ncell; cid += stride) {
    const uint32_t w = c.cnt[cid];
    if (w == 0) continue;
    const double4 s = c.sum[cid];
    px += s.x;
    py += s.y;
    pz += s.z;
    e += s.w;
    nf += (uint32_t)cnt_fluid(w);
    nb += (uint32_t)cnt_beads(w);
  }
  for (long s = (long)blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += stride) {
    if (m.moves[s] != 1) continue;
    const double vx = m.vx[s], vy = m.vy[s], vz = m.vz[s];
    eb += bead_mass * (vx * vx + vy * vy + vz * vz);
  }
  // the counts as integers up to the block total, then exact in float64
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nf += __shfl_xor_sync(0xffffffffu, nf, o);
    nb += __shfl_xor_sync(0xffffffffu, nb, o);
  }
  __shared__ uint32_t s_cnt[2][32];
  if ((threadIdx.x & 31) == 0) {
    s_cnt[0][threadIdx.x >> 5] = nf;
    s_cnt[1][threadIdx.x >> 5] = nb;
  }
  const double v5[5] = {px, py, pz, e, eb};
  __shared__ bool last;
  __shared__ double t5[5];
  __shared__ double tot[7];
  block_sums_f64<5>(v5, t5);  // t5 for every thread after it (its barriers order s_cnt too)
  if (threadIdx.x < 7) {  // partial k: P x, y, z, sum m v^2, fluid n, bead n, bead sum m v^2
    double r;
    if (threadIdx.x < 4) {
      r = t5[threadIdx.x];
    } else if (threadIdx.x == 6) {
      r = t5[4];
    } else {
      uint32_t t = 0;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += s_cnt[threadIdx.x - 4][i];
      r = (double)t;
    }
    part[7 * blockIdx.x + threadIdx.x] = r;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double vals[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += __ldcg(part + 7 * b + k);
    vals[k] = v;
  }
  block_sums_f64<7>(vals, tot);
  if (threadIdx.x == 0) {
    out[0] = tot[0];
    out[1] = tot[1];
    out[2] = tot[2];
    out[3] = tot[3];
    out[4] = tot[4] + tot[5];
    out[5] = tot[4] + tot[5] * bead_mass;
    out[6] = tot[3] - tot[6];
    out[7] = tot[4];
    out[8] = *diss;
    out[9] = (double)*err;  // bit flags (below 2^16): exact
    *counter = 0u;  // ready for the next call
  }
}

// ================================================================== sort ===

__global__ void k_sort_count(const uint32_t* cell, long n, Box box, uint32_t* count, uint32_t* rank) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t cp = cell[i];
    const long c = box.lin(cell_x(cp), cell_y(cp), cell_z(cp));
    rank[i] = atomicAdd(count + c, 1u);
  }
}

__global__ void k_sort_count_f32(const float4* pos, long n, Box box, uint32_t* count, uint32_t* rank) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t cp = __float_as_uint(pos[i].w);
    const long c = box.lin(cell_x(cp), cell_y(cp), cell_z(cp));
    rank[i] = atomicAdd(count + c, 1u);
  }
}

// exclusive scan of `count` (n entries) into `start`, three passes
constexpr int kScanBlock = 1024;

__global__ void k_scan_blocks(const uint32_t* in, long n, uint32_t* blocksums) {
  __shared__ uint32_t red[32];
  long i = (long)blockIdx.x * kScanBlock + threadIdx.x;
  uint32_t v = i < n ? in[i] : 0u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t r = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (threadIdx.x == 0) blocksums[blockIdx.x] = r;
  }
}

__global__ void k_scan_blocksums(uint32_t* blocksums, int nb) {
  // single block: sequential over chunks of 1024 with an in-block scan
  __shared__ uint32_t wsum[32];
  uint32_t carry = 0;
  for (int base = 0; base < nb; base += kScanBlock) {
    int i = base + threadIdx.x;
    uint32_t v = i < nb ? blocksums[i] : 0u;
    uint32_t x = v;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      uint32_t w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    uint32_t incl = x + (wid > 0 ? wsum[wid - 1] : 0u);
    if (i < nb) blocksums[i] = carry + incl - v;  // exclusive
    uint32_t total = wsum[31];
    __syncthreads();
    carry += total;
  }
}

__global__ void k_scan_apply(const uint32_t* in, long n, const uint32_t* blockoff, uint32_t* out) {
  __shared__ uint32_t wsum[32];
  long i = (long)blockIdx.x * kScanBlock + threadIdx.x;
  uint32_t v = i < n ? in[i] : 0u;
  uint32_t x = v;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  uint32_t incl = x + (wid > 0 ? wsum[wid - 1] : 0u);
  if (i < n) out[i] = blockoff[blockIdx.x] + incl - v;
}

__global__ void k_sort_scatter_f64(FluidF64 src, FluidF64 dst, Box box, const uint32_t* start, const uint32_t* rank) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < src.n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t cp = src.cell[i];
    const long c = box.lin(cell_x(cp), cell_y(cp), cell_z(cp));
    const long d = (long)start[c] + rank[i];
    dst.id[d] = src.id[i];
    dst.cell[d] = cp;
    dst.ox[d] = src.ox[i];
    dst.oy[d] = src.oy[i];
    dst.oz[d] = src.oz[i];
    dst.vx[d] = src.vx[i];
    dst.vy[d] = src.vy[i];
    dst.vz[d] = src.vz[i];
  }
}

__global__ void k_sort_scatter_f32(FluidF32 src, FluidF32 dst, Box box, const uint32_t* start, const uint32_t* rank) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < src.n; i += (long)gridDim.x * blockDim.x) {
    const float4 p = src.pos[i];
    const uint32_t cp = __float_as_uint(p.w);
    const long c = box.lin(cell_x(cp), cell_y(cp), cell_z(cp));
    const long d = (long)start[c] + rank[i];
    dst.id[d] = src.id[i];
    dst.pos[d] = p;
    dst.vel[d] = src.vel[i];
  }
}

int scan_counts(const uint32_t* count, long ncell, uint32_t* start, uint32_t* blocksums, cudaStream_t s) {
  const int nb = (int)((ncell + kScanBlock - 1) / kScanBlock);
  k_scan_blocks<<<nb, kScanBlock, 0, s>>>(count, ncell, blocksums);
  k_scan_blocksums<<<1, kScanBlock, 0, s>>>(blocksums, nb);
  k_scan_apply<<<nb, kScanBlock, 0, s>>>(count, ncell, blocksums, start);
  return 3;
}

// ============================================================== float32 ===
// Split precision: position = packed cell + float32 offset, velocity float32,
// per-cell sums and collision maps float32.  The thermostat factor and the
// rotation are computed per cell in float64 and rounded once.

// Adds a block's sum to *dst by the warp that comes last, as energy_end.
__device__ __forceinline__ void energy_end_f32(BlockEnergy& b, float v, double* dst) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&b.sum, (double)v);
    __threadfence_block();
    if (atomicAdd(&b.warps, 1u) == (blockDim.x >> 5) - 1) {
      __threadfence_block();
      const double tot = *reinterpret_cast<volatile double*>(&b.sum);
      if (tot != 0.0) atomicAdd(dst, tot);
    }
  }
}
// Split-precision collision map: everything per cell in float (the sums
// are float); the dissipated-energy bookkeeping accumulates in float64.
// Small blocks, loads of two cells issued together before any generator runs
// (one cell's alone: 158 us, four with persistent blocks of 256 as before 59,
// at 128^3 cells); the draws come before the sums are needed.  128^3 cells 91
// to 50 us, 64^3 16.4 to 14.8.
__global__ void __launch_bounds__(kCellThreads) k_cell_params_f32(CellsF32 c, StepArgs a) {
  __shared__ BlockEnergy s_e;
  energy_begin(s_e);
  chain_begin();
  float ldiss = 0.0f;
  unsigned errbits = 0;
  bool gfail = false;
  constexpr int kU = 2;
  const long stride = (long)gridDim.x * blockDim.x;
  for (long cb = (long)blockIdx.x * blockDim.x + threadIdx.x; cb < c.ncell; cb += kU * stride) {
    uint32_t w[kU];
    float4 sm[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long cid = cb + u * stride;
      w[u] = cid < c.ncell ? __ldcg(c.cnt + cid) : 0u;
      sm[u] = cid < c.ncell ? __ldcg(c.sum + cid) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (!w[u]) continue;
      const long cid = cb + u * stride;
      c.sum[cid] = make_float4(0.f, 0.f, 0.f, 0.f);
      c.cnt[cid] = 0u;
      if (a.premapped && cnt_beads(w[u]) > 0) continue;  // mapped by k_bead_maps_f32
      cell_map_f32(sm[u], w[u], (uint32_t)cid, a.seed, a.step, a.fbead_mass, a.inj_gamma, a.inj_axis, c.par + 2 * cid, ldiss,
                 errbits, gfail, &a);
    }
  }
  if (gfail) errbits |= kErrGammaLoop;
  if (errbits) atomicOr(a.err, errbits);
  energy_end_f32(s_e, ldiss, a.diss);
}

// Particles per thread whose loads (state, then collision map) are issued
// together before any of their reductions and stores.  The pass is bound by
// the latency of the dependent chain particle -> cell -> map; the chains in
// flight per SM are bounded by the register file, so one, two and four per
// thread measured alike (two: 48.6 us on 2.6 M particles, one 47.5, four 58.8
// at half the resident CTAs).  MPCD_FLUID_BATCH selects 1, 2 or 4.
constexpr int kFluidBatch = 2;
// resident CTAs per SM the register budget of a batch size allows
template <int U>
struct FluidMinBlocks {
  static constexpr int value = U >= 4 ? 2 : 4;
};
// default options of the split-precision fluid pass (kOptPrefetch | kOptAggregate
// bits): both (2.62 M particles, persistent grid: 45.8 us against 49.2 us
// without either, 50.4 with the prefetch alone, 49.1 with the aggregation
// alone; the same order with one particle per thread)
constexpr int kFluidOpt = 3;

// Options of the split-precision fluid pass (bits of kOpt):
//   kOptPrefetch  one thread per CTA and round sends the particle state of the
//                 chunk `pf_dist` particles ahead (the chunk a later round or
//                 a later CTA takes) from HBM into L2 by a bulk prefetch, so
//                 that the dependent chain particle -> cell -> map starts
//                 from L2
//   kOptAggregate the warp's particles binned into the same next cell are
//                 summed in registers (peer_sum) and added by one vector
//                 reduction and one count add per cell and warp
//   kOptLast      a step whose cell sums nobody will read: nothing is binned,
//                 and nothing happens at all if *a.skip is set
constexpr int kOptPrefetch = 1;
constexpr int kOptAggregate = 2;
constexpr int kOptLast = 4;

// kWalls: the bounce-back path (its float64 temporaries would otherwise
// crowd the registers of the batched loads).
template <int U, bool kWalls, typename I, int kOpt>
__global__ void __launch_bounds__(kThreads, FluidMinBlocks<U>::value)
    k_fluid_step_f32(FluidF32 f, CellsF32 c, StepArgs a, long pf_dist) {
  const int Lx = a.box.L[0], Ly = a.box.L[1], Lz = a.box.L[2];
  const float tcx = a.fta_cur[0], tcy = a.fta_cur[1], tcz = a.fta_cur[2];
  const float tnx = a.fta_next[0], tny = a.fta_next[1], tnz = a.fta_next[2];
  const float h = a.fh, gk = a.fgkick;
  float ke_after = 0.0f;
  unsigned bad = 0;
  chain_begin();
  if ((kOpt & kOptLast) && *a.skip) return;
  const I n = (I)f.n;
  const I lane = (I)(threadIdx.x & 31);
  // each block takes U x blockDim consecutive particles per round; the loop
  // runs while the warp's first particle exists, so that every lane of a
  // warp takes part in the warp-wide operations of each round
  for (I base = (I)blockIdx.x * U * blockDim.x + threadIdx.x; base - lane < n; base += (I)gridDim.x * U * blockDim.x) {
    if ((kOpt & kOptPrefetch) && threadIdx.x == 0) {
      const long s = (long)base + pf_dist;
      if (s < (long)n) {
        const long cnt = min((long)U * blockDim.x, (long)n - s);
        prefetch_l2(f.pos + s, (uint32_t)(cnt * sizeof(float4)));
        prefetch_l2(f.vel + s, (uint32_t)(cnt * sizeof(float4)));
      }
    }
    float4 p[U], v[U], mk[U], mu[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const I i = base + (I)q * blockDim.x;
      if (i < n) {
        p[q] = __ldcs(f.pos + i);
        v[q] = __ldcs(f.vel + i);
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const I i = base + (I)q * blockDim.x;
      if (i < n) {
        const uint32_t cp = __float_as_uint(p[q].w);
        const uint32_t cid = (uint32_t)shifted_f(cell_x(cp), p[q].x, tcx, Lx) +
                             (uint32_t)Lx * ((uint32_t)shifted_f(cell_y(cp), p[q].y, tcy, Ly) +
                                             (uint32_t)Ly * (uint32_t)shifted_f(cell_z(cp), p[q].z, tcz, Lz));
        const float4* m = c.par + 2 * (size_t)cid;
        mk[q] = m[0];
        mu[q] = m[1];
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const I i = base + (I)q * blockDim.x;
      if (kOpt & kOptAggregate) {
        if (base + (I)q * blockDim.x - lane >= n) continue;  // warp-uniform: no particle of this warp
      } else if (i >= n) {
        continue;
      }
      const bool valid = i < n;
      if (!valid) p[q] = v[q] = mk[q] = mu[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      const uint32_t cp = __float_as_uint(p[q].w);
      int ix = cell_x(cp), iy = cell_y(cp), iz = cell_z(cp);
      float ox = p[q].x, oy = p[q].y, oz = p[q].z, vx = v[q].x, vy = v[q].y, vz = v[q].z;
      apply_map_f32(mk[q], mu[q], vx, vy, vz);
      ke_after += vx * vx + vy * vy + vz * vz;
      if (!kWalls) {
        ox = fmaf(vx, h, ox);
        oy = fmaf(vy, h, oy);
        oz = fmaf(vz, h, oz);
      } else {
        double x = ix + (double)ox, y = iy + (double)oy, z = iz + (double)oz;
        double dvx = vx, dvy = vy, dvz = vz;
        double X[3] = {x, y, z}, V[3] = {dvx, dvy, dvz};
        if (a.sph.n && sphere_bounce(a.sph, a.box, a.h, X, V)) {
          x = X[0];
          y = X[1];
          z = X[2];
          dvx = V[0];
          dvy = V[1];
          dvz = V[2];
        } else {
          x += dvx * a.h;
          y += dvy * a.h;
          z += dvz * a.h;
        }
        if (a.walls) wall_bounce(a.walls, (double)(Lz - 1), x, y, z, dvx, dvy, dvz);
        double fx = floor(x), fy = floor(y), fz = floor(z);
        ox = (float)(x - fx);
        oy = (float)(y - fy);
        oz = (float)(z - fz);
        ix = (((int)fx % Lx) + Lx) % Lx;
        iy = (((int)fy % Ly) + Ly) % Ly;
        iz = (((int)fz % Lz) + Lz) % Lz;
        vx = (float)dvx;
        vy = (float)dvy;
        vz = (float)dvz;
      }
      rewrap_f(ox, ix, Lx, bad);
      rewrap_f(oy, iy, Ly, bad);
      rewrap_f(oz, iz, Lz, bad);
      if (gk != 0.0f) vx += gk;
      const uint32_t cn = (uint32_t)shifted_f(ix, ox, tnx, Lx) +
                          (uint32_t)Lx * ((uint32_t)shifted_f(iy, oy, tny, Ly) + (uint32_t)Ly * (uint32_t)shifted_f(iz, oz, tnz, Lz));
      const float4 contrib = make_float4(vx, vy, vz, vx * vx + vy * vy + vz * vz);
      if (kOpt & kOptLast) {
      } else if (kOpt & kOptAggregate) {
        const uint32_t key = valid ? cn : 0xffffffffu;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const float4 tot = peer_sum(peers, valid ? contrib : make_float4(0.f, 0.f, 0.f, 0.f));
        if (valid && (unsigned)(__ffs(peers) - 1) == (unsigned)lane) {
          red_add_v4(c.sum + cn, tot);
          atomicAdd(c.cnt + cn, (uint32_t)__popc(peers));
        }
      } else {
        red_add_v4(c.sum + cn, contrib);
        atomicAdd(c.cnt + cn, 1u);
      }
      if (valid) {  // (a lane past the end carried a zero particle: nothing to store, nothing added to ke_after)
        __stcs(f.pos + i, make_float4(ox, oy, oz, __uint_as_float(pack_cell(ix, iy, iz))));
        __stcs(f.vel + i, make_float4(vx, vy, vz, 0.f));
      }
    }
  }
  if (bad) atomicOr(a.err, bad);
  const double tot = block_sum_f32(ke_after);
  if (threadIdx.x == 0 && tot != 0.0) atomicAdd(a.diss, -tot);
}

__global__ void k_bin_fluid_f32(FluidF32 f, CellsF32 c, StepArgs a) {
  const int Lx = a.box.L[0], Ly = a.box.L[1], Lz = a.box.L[2];
  const float tcx = a.fta_cur[0], tcy = a.fta_cur[1], tcz = a.fta_cur[2];
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const float4 p = f.pos[i];
    const float4 v = f.vel[i];
    const uint32_t cp = __float_as_uint(p.w);
    const long cid = shifted_f(cell_x(cp), p.x, tcx, Lx) +
                     (long)Lx * (shifted_f(cell_y(cp), p.y, tcy, Ly) + (long)Ly * shifted_f(cell_z(cp), p.z, tcz, Lz));
    red_add_v4(c.sum + cid, make_float4(v.x, v.y, v.z, v.x * v.x + v.y * v.y + v.z * v.z));
    atomicAdd(c.cnt + cid, 1u);
  }
}

__global__ void k_bead_collide_f32(MDState m, CellsF32 c, StepArgs a) {
  double ke_after = 0.0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      atomicOr(a.err, kErrCellRange);
      continue;
    }
    float vx = (float)m.vx[s], vy = (float)m.vy[s], vz = (float)m.vz[s];
    apply_map_f32(c.par + 2 * cid, vx, vy, vz);
    ke_after += a.bead_mass * ((double)vx * vx + (double)vy * vy + (double)vz * vz);
    m.vx[s] = vx;
    m.vy[s] = vy;
    m.vz[s] = vz;
  }
  const double tot = block_sum_f64(ke_after);
  if (threadIdx.x == 0 && tot != 0.0) atomicAdd(a.diss, -tot);
}

__global__ void k_bin_beads_f32(MDState m, CellsF32 c, StepArgs a) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      atomicOr(a.err, kErrCellRange);
      continue;
    }
    const float mb = (float)a.bead_mass;
    const float vx = (float)m.vx[s], vy = (float)m.vy[s], vz = (float)m.vz[s];
    red_add_v4(c.sum + cid, make_float4(vx * mb, vy * mb, vz * mb, mb * (vx * vx + vy * vy + vz * vz)));
    atomicAdd(c.cnt + cid, 1u << 16);
  }
}

__global__ void k_observables_f32(FluidF32 f, MDState m, double bead_mass, double* out) {
  double px = 0, py = 0, pz = 0, e = 0, n = 0, ms = 0, ef = 0, nf = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const float4 v = f.vel[i];
    const double vx = v.x, vy = v.y, vz = v.z;
    const double v2 = vx * vx + vy * vy + vz * vz;
    px += vx;
    py += vy;
    pz += vz;
    e += v2;
    ef += v2;
    n += 1.0;
    ms += 1.0;
    nf += 1.0;
  }
  for (long s = (long)blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += (long)gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const double vx = m.vx[s], vy = m.vy[s], vz = m.vz[s];
    px += bead_mass * vx;
    py += bead_mass * vy;
    pz += bead_mass * vz;
    e += bead_mass * (vx * vx + vy * vy + vz * vz);
    n += 1.0;
    ms += bead_mass;
  }
  double vals[8] = {px, py, pz, e, n, ms, ef, nf};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double t = block_sum_f64(vals[k]);
    if (threadIdx.x == 0) atomicAdd(out + k, t);
  }
}

// ====================================================== host interchange ===
// Fluid state to and from the caller's float64 arrays (positions N x 3,
// unwrapped allowed; velocities N x 3), staged in device memory as they
// are: the conversion to cell + offset, the split into the kernels' layout
// and the return to input order by particle id run here, one thread per
// particle, instead of in host loops.

// 1 for a non-finite or out-of-range (|x| > 1e12) position or velocity
__global__ void k_check_fluid(long n, const double* pos, const double* vel, unsigned* bad) {
  unsigned b = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += (long)gridDim.x * blockDim.x) {
    const double x = pos[i], v = vel[i];
    if (!(fabs(x) <= 1e12) || !isfinite(v)) b = 1u;
  }
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1u);
}

// an unwrapped coordinate as cell index + offset in [0,1); explicit
// roundings (no contraction into a fused multiply-add) so that the result is
// the same as the host's plain float64 arithmetic
__device__ __forceinline__ void wrap_coord_dev(double x, int L, int& i, double& o) {
  const double dl = (double)L;
  double xw = __dsub_rn(x, __dmul_rn(floor(__ddiv_rn(x, dl)), dl));
  if (xw >= dl) xw = __dsub_rn(xw, dl);
  if (xw < 0) xw = __dadd_rn(xw, dl);
  const double fi = floor(xw);
  i = (int)fi;
  o = __dsub_rn(xw, fi);
  if (i >= L) i -= L;
  if (o >= 1.0) {
    o = 0.0;
    i = (i + 1) % L;
  }
}

__global__ void k_load_fluid_f64(long n, const double* pos, const double* vel, Box box, FluidF64 f) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    int c[3];
    double o[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) wrap_coord_dev(pos[3 * i + q], box.L[q], c[q], o[q]);
    f.id[i] = (uint32_t)i;
    f.cell[i] = pack_cell(c[0], c[1], c[2]);
    f.ox[i] = offset_from_double(o[0]);
    f.oy[i] = offset_from_double(o[1]);
    f.oz[i] = offset_from_double(o[2]);
    f.vx[i] = vel[3 * i];
    f.vy[i] = vel[3 * i + 1];
    f.vz[i] = vel[3 * i + 2];
  }
}

__global__ void k_load_fluid_f32(long n, const double* pos, const double* vel, Box box, FluidF32 f) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    int c[3];
    float o[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double od;
      wrap_coord_dev(pos[3 * i + q], box.L[q], c[q], od);
      o[q] = __double2float_rn(od);
      if (o[q] >= 1.0f) {  // rounding up to 1: move to the next cell
        o[q] = 0.0f;
        c[q] = (c[q] + 1) % box.L[q];
      }
    }
    f.id[i] = (uint32_t)i;
    f.pos[i] = make_float4(o[0], o[1], o[2], __uint_as_float(pack_cell(c[0], c[1], c[2])));
    f.vel[i] = make_float4(__double2float_rn(vel[3 * i]), __double2float_rn(vel[3 * i + 1]),
                           __double2float_rn(vel[3 * i + 2]), 0.0f);
  }
}

// a snapshot's offsets in place: float64 ones (of an older version) into fixed
// point, integers into their range
__global__ void k_convert_offsets(long n, uint64_t* o, bool integers) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if (integers) {  // whatever the bytes were, an offset
      o[i] &= kOffOne - 1;
      continue;
    }
    double d = __longlong_as_double((long long)o[i]);
    if (!(d >= 0.0 && d < 1.0)) d = 0.5;
    o[i] = offset_from_double(d);
  }
}

// Back to input order: particle k of the caller is the one with id k.
// status: {an id is out of range, the engine's error word}, in host memory.
__device__ __forceinline__ void report_error(unsigned* status, const unsigned* err) {
  if (blockIdx.x == 0 && threadIdx.x == 0) status[1] = *err;
}
__device__ __forceinline__ void store_pos(const FluidF64& f, long i, double* p) {
  const uint32_t cp = f.cell[i];
  const uint64_t ox = f.ox[i], oy = f.oy[i], oz = f.oz[i];
  p[0] = __dadd_rn((double)cell_x(cp), offset_to_double(ox));
  p[1] = __dadd_rn((double)cell_y(cp), offset_to_double(oy));
  p[2] = __dadd_rn((double)cell_z(cp), offset_to_double(oz));
}
__device__ __forceinline__ void store_vel(const FluidF64& f, long i, double* v) {
  const double vx = f.vx[i], vy = f.vy[i], vz = f.vz[i];
  v[0] = vx;
  v[1] = vy;
  v[2] = vz;
}
__device__ __forceinline__ void store_pos(const FluidF32& f, long i, double* q) {
  const float4 p = f.pos[i];
  const uint32_t cp = __float_as_uint(p.w);
  q[0] = __dadd_rn((double)cell_x(cp), (double)p.x);
  q[1] = __dadd_rn((double)cell_y(cp), (double)p.y);
  q[2] = __dadd_rn((double)cell_z(cp), (double)p.z);
}
__device__ __forceinline__ void store_vel(const FluidF32& f, long i, double* q) {
  const float4 v = f.vel[i];
  q[0] = v.x;
  q[1] = v.y;
  q[2] = v.z;
}
// the whole fluid in one launch
template <typename F>
__global__ void k_store_fluid(F f, double* pos, double* vel, unsigned* status, const unsigned* err) {
  chain_begin();
  report_error(status, err);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const long d = f.id[i];
    if (d >= f.n) {
      status[0] = 1u;
      continue;
    }
    store_pos(f, i, pos + 3 * d);
    store_vel(f, i, vel + 3 * d);
  }
}
// a thread per bead and axis: whole rows go out, also to host memory
__global__ void k_store_beads(MDState m, long s0, int nb, double* pos, double* vel, unsigned* status,
                              const unsigned* err) {
  if (status) report_error(status, err);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 3 * nb; k += gridDim.x * blockDim.x) {
    const int d = k / 3, ax = k - 3 * d;
    const long s = s0 + m.slot_of[s0 + d];
    pos[k] = ax == 0 ? m.x[0][s] : (ax == 1 ? m.y[0][s] : m.z[0][s]);
    vel[k] = ax == 0 ? m.vx[s] : (ax == 1 ? m.vy[s] : m.vz[s]);
  }
}
// In parts of the caller's order, so that a part is copied to the host while
// the next is gathered: where each particle is kept, then positions or
// velocities of the particles d0 .. d1.
template <typename F>
__global__ void k_find_particles(F f, uint32_t* at, unsigned* status, const unsigned* err) {
  chain_begin();
  report_error(status, err);
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const long d = f.id[i];
    if (d < f.n)
      at[d] = (uint32_t)i;
    else
      status[0] = 1u;
  }
}
template <typename F>
__global__ void k_gather_fluid(F f, const uint32_t* at, long d0, long d1, bool velocity, double* out, unsigned* status) {
  for (long d = d0 + (long)blockIdx.x * blockDim.x + threadIdx.x; d < d1; d += (long)gridDim.x * blockDim.x) {
    const long i = at[d];
    if (i >= f.n)
      status[0] = 1u;
    else if (velocity)
      store_vel(f, i, out + 3 * d);
    else
      store_pos(f, i, out + 3 * d);
  }
}

// The collision maps of the cells holding moving beads (the same map
// k_cell_params_* would make from the same sums and generator keys), one
// thread per bead slot; the first bead of a cell to take the cell's claim
// word with this step's tag makes it.  The sums are left for the cell-map
// kernel to clear.
__global__ void k_bead_maps_f64(MDState m, CellsF64 c, StepArgs a, uint32_t* claim, uint32_t tag) {
  __shared__ BlockEnergy s_e;
  energy_begin(s_e);
  EnergySum ke;
  double ke_rest = 0.0;
  unsigned errbits = 0;
  bool gfail = false;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      errbits |= kErrCellRange;
      continue;
    }
    if (atomicExch(claim + cid, tag) == tag) continue;  // another bead of the cell makes it
    const uint32_t w = c.cnt[cid];
    if (w == 0) continue;
    collision_map(c.sum[cid], w, cid, a, c.par + 12 * cid, ke, ke_rest, errbits, gfail);
  }
  if (gfail) errbits |= kErrGammaLoop;
  if (errbits) atomicOr(a.err, errbits);
  energy_end(s_e, ke, kCellEnergyBits, ke_rest, 1.0, a.diss);
}

__global__ void k_bead_maps_f32(MDState m, CellsF32 c, StepArgs a, uint32_t* claim, uint32_t tag) {
  float ldiss = 0.0f;
  unsigned errbits = 0;
  bool gfail = false;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const long cid = unwrapped_cell(a.box, a.a_cur, m.x[0][s], m.y[0][s], m.z[0][s]);
    if (cid < 0) {
      errbits |= kErrCellRange;
      continue;
    }
    if (atomicExch(claim + cid, tag) == tag) continue;
    const uint32_t w = c.cnt[cid];
    if (w == 0) continue;
    cell_map_f32(c.sum[cid], w, (uint32_t)cid, a.seed, a.step, a.fbead_mass, a.inj_gamma, a.inj_axis, c.par + 2 * cid,
                 ldiss, errbits, gfail, &a);
  }
  if (gfail) errbits |= kErrGammaLoop;
  if (errbits) atomicOr(a.err, errbits);
  const double tot = block_sum_f32(ldiss);
  if (threadIdx.x == 0 && tot != 0.0) atomicAdd(a.diss, tot);
}

// the MD launch's deferred bead binning into the cell sums
__global__ void k_bead_add_f64(MDState m, CellsF64 c, const uint32_t* bcell, const double4* bsum) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const uint32_t cid = bcell[s];
    if (cid == 0xffffffffu) continue;
    const double4 v = bsum[s];
    double* sp = reinterpret_cast<double*>(c.sum + cid);
    atomicAdd(sp + 0, v.x);
    atomicAdd(sp + 1, v.y);
    atomicAdd(sp + 2, v.z);
    atomicAdd(sp + 3, v.w);
    atomicAdd(c.cnt + cid, 1u << 16);
  }
}

__global__ void k_bead_add_f32(MDState m, CellsF32 c, const uint32_t* bcell, const float4* bsum) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.nslots; s += gridDim.x * blockDim.x) {
    if (m.moves[s] != 1) continue;
    const uint32_t cid = bcell[s];
    if (cid == 0xffffffffu) continue;
    red_add_v4(c.sum + cid, bsum[s]);
    atomicAdd(c.cnt + cid, 1u << 16);
  }
}

// Rigid spheres after a step: the impulse and angular impulse the fluid gave
// them this step are added to the running force and torque sums (divided by
// h) and cleared; every sphere moves with the velocity it had during the
// step; a free sphere (mass > 0) then takes the impulses into its velocity
// and angular velocity (solid sphere, I = 2/5 m r^2).  Float64 throughout.
__global__ void k_spheres_update(RigidSphereDev* s, int n, double* acc, double* fsum, double h, Box box) {
  const int k = threadIdx.x;
  if (k >= n) return;
  RigidSphereDev S = s[k];
  double* A = acc + 6 * k;
  for (int j = 0; j < 6; ++j) fsum[6 * k + j] += A[j] / h;
  for (int q = 0; q < 3; ++q) {
    S.c[q] += S.v[q] * h;
    if (S.r < 0.5 * box.L[q]) {  // spheres with periodic images stay in [0, L)
      if (S.c[q] >= box.L[q]) S.c[q] -= box.L[q];
      if (S.c[q] < 0.0) S.c[q] += box.L[q];
    }
  }
  if (S.mass > 0.0) {
    for (int q = 0; q < 3; ++q) {
      S.v[q] += A[q] / S.mass;
      S.w[q] += A[3 + q] / S.inertia;
    }
  }
  for (int j = 0; j < 6; ++j) A[j] = 0.0;
  s[k] = S;
}

// The generator's per-cell draws, as the collision kernels take them: cell k
// of step `step` gets the Gamma(3(nc-1)/2) variate of gamma_mt and the
// float64 path's rotation axis.  Used to check the samplers' distributions.
__global__ void k_collision_draws(int nc, uint64_t seed, uint64_t step, long n, double* gamma, double* axis,
                                  unsigned* err) {
  bool gfail = false;
  for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
    if (gamma) gamma[k] = (double)gamma_mt(nc, seed, step, (uint32_t)k, &gfail);
    if (axis) draw_axis_f64(seed, step, (uint32_t)k, axis[3 * k], axis[3 * k + 1], axis[3 * k + 2]);
  }
  if (gfail) atomicOr(err, kErrGammaLoop);
}

}  // namespace

// ============================================================ launchers ===

int launch_bead_maps_f64(const MDState& m, const CellsF64& c, const StepArgs& a, uint32_t* claim, uint32_t tag,
                         cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_maps_f64<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a, claim, tag);
  return 1;
}
int launch_bead_maps_f32(const MDState& m, const CellsF32& c, const StepArgs& a, uint32_t* claim, uint32_t tag,
                         cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_maps_f32<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a, claim, tag);
  return 1;
}
int launch_bead_add_f64(const MDState& m, const CellsF64& c, const uint32_t* bcell, const void* bsum, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_add_f64<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, bcell, static_cast<const double4*>(bsum));
  return 1;
}
int launch_bead_add_f32(const MDState& m, const CellsF32& c, const uint32_t* bcell, const void* bsum, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_add_f32<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, bcell, static_cast<const float4*>(bsum));
  return 1;
}

int launch_spheres_update(RigidSphereDev* sph, int n, double* acc, double* fsum, double h, const Box& box,
                          cudaStream_t s) {
  if (n <= 0) return 0;
  k_spheres_update<<<1, 32, 0, s>>>(sph, n, acc, fsum, h, box);
  return 1;
}

// Launches a kernel that begins with chain_begin(), in a chain as a
// programmatic dependent: its CTAs are placed while the predecessor drains.
// Per step of two kernels: 8^3 cells 18.4 to 13.2 us, 32^3 30.2 to 27.2, the
// channel 37.7 to 36.0, 80 x 71 x 89 232 to 227.  Not beside an MD launch, where an
// event lies between the two.
template <typename... P, typename... A>
cudaError_t launch_in_chain(void (*kernel)(P...), int grid, int threads, cudaStream_t s, bool chained, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

int launch_collision_draws(int nc, uint64_t seed, uint64_t step, long n, double* gamma, double* axis, unsigned* err,
                           cudaStream_t s) {
  if (n == 0) return 0;
  k_collision_draws<<<grid_for(n), kThreads, 0, s>>>(nc, seed, step, n, gamma, axis, err);
  return 1;
}

int launch_cell_params_f64(const CellsF64& c, const StepArgs& a, cudaStream_t s) {
  // by warp pairs as long as all of them are on the SMs at once (figures there)
  if (c.ncell <= 32l * kPairCTAs * sm_count())
    launch_in_chain(k_cell_pairs_f64, (int)((c.ncell + 31) / 32), kCellThreads, s, a.chained, c, a);
  else
    launch_in_chain(k_cell_params_f64, grid_for(c.ncell, kCellThreads, -1), kCellThreads, s, a.chained, c, a);
  return 1;
}
int launch_fluid_step_f64(const FluidF64& f, const CellsF64& c, const StepArgs& a, cudaStream_t s, int per_sm) {
  if (f.n == 0) return 0;
  const int grid = grid_for(f.n, kFluidThreads, per_sm);
  const bool i32 = f.n + (long)grid * kThreads < (1L << 32);
  auto launch = [&](auto kernel) { launch_in_chain(kernel, grid, kFluidThreads, s, a.chained, f, c, a); };
  if (a.sph.n > 0)
    i32 ? launch(k_fluid_step_f64<uint32_t, kSpheres>) : launch(k_fluid_step_f64<long, kSpheres>);
  else if (a.walls != 0)
    i32 ? launch(k_fluid_step_f64<uint32_t, kWalled>) : launch(k_fluid_step_f64<long, kWalled>);
  else
    i32 ? launch(k_fluid_step_f64<uint32_t, kPeriodic>) : launch(k_fluid_step_f64<long, kPeriodic>);
  return 1;
}
int launch_bin_fluid_f64(const FluidF64& f, const CellsF64& c, const StepArgs& a, cudaStream_t s) {
  if (f.n == 0) return 0;
  k_bin_fluid_f64<<<grid_for(f.n), kThreads, 0, s>>>(f, c, a);
  return 1;
}
int launch_bead_collide_f64(const MDState& m, const CellsF64& c, const StepArgs& a, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_collide_f64<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a);
  return 1;
}
int launch_bin_beads_f64(const MDState& m, const CellsF64& c, const StepArgs& a, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bin_beads_f64<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a);
  return 1;
}
int launch_observables_cells_f64(const CellsF64& c, const MDState& m, double bead_mass, const double* diss,
                                 const unsigned* err, double* part, unsigned* counter, double* out, cudaStream_t s) {
  const long n = c.ncell > m.nslots ? c.ncell : m.nslots;
  const int g1 = grid_for(n, kThreads, 1);  // at most one block per SM
  const int g = g1 < kObsBlocks ? g1 : kObsBlocks;
  k_observables_cells_f64<<<g, kThreads, 0, s>>>(c, m, bead_mass, diss, err, part, counter, out);
  return 1;
}
int launch_observables_f64(const FluidF64& f, const MDState& m, double bead_mass, double* out, cudaStream_t s) {
  long n = f.n > m.nslots ? f.n : m.nslots;
  k_observables_f64<<<grid_for(n) < 1024 ? grid_for(n) : 1024, kThreads, 0, s>>>(f, m, bead_mass, out);
  return 1;
}
int launch_sort_f64(FluidF64& f, FluidF64& tmp, const Box& box, uint32_t* count, uint32_t* start, uint32_t* rank,
                    uint32_t* blocksums, cudaStream_t s) {
  const long ncell = (long)box.L[0] * box.L[1] * box.L[2];
  cudaMemsetAsync(count, 0, ncell * sizeof(uint32_t), s);
  k_sort_count<<<grid_for(f.n), kThreads, 0, s>>>(f.cell, f.n, box, count, rank);
  int k = 1 + scan_counts(count, ncell, start, blocksums, s);
  tmp.n = f.n;
  k_sort_scatter_f64<<<grid_for(f.n), kThreads, 0, s>>>(f, tmp, box, start, rank);
  FluidF64 t = f;
  f = tmp;
  tmp = t;
  return k + 1;
}

int scan_counts_ext(const uint32_t* count, long ncell, uint32_t* start, uint32_t* blocksums, cudaStream_t s) {
  return scan_counts(count, ncell, start, blocksums, s);
}

int launch_cell_params_f32(const CellsF32& c, const StepArgs& a, cudaStream_t s) {
  launch_in_chain(k_cell_params_f32, grid_for(c.ncell, kCellThreads, -1), kCellThreads, s, a.chained, c, a);
  return 1;
}
template <int U, int kOpt>
void launch_fluid_f32_opt(const FluidF32& f, const CellsF32& c, const StepArgs& a, cudaStream_t s, int per_sm) {
  const int ps = per_sm <= 0 ? per_sm : std::min(per_sm, FluidMinBlocks<U>::value);
  const int gb = grid_for((f.n + U - 1) / U, kThreads, ps);
  const bool i32 = f.n + 4L * gb * kThreads < (1L << 32);
  long pf = 0;
  if (kOpt & kOptPrefetch) {
    // the chunk the CTA starting after the current wave (or this CTA's next
    // round, for a grid of at most one wave) will take
    static int resident = 0;
    if (resident == 0) {
      int per = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fluid_step_f32<U, false, uint32_t, kOpt>, kThreads, 0);
      resident = std::max(1, per) * sm_count();
    }
    pf = (long)std::min(gb, resident) * U * kThreads;
  }
  if (i32)
    launch_in_chain(k_fluid_step_f32<U, false, uint32_t, kOpt>, gb, kThreads, s, a.chained, f, c, a, pf);
  else
    launch_in_chain(k_fluid_step_f32<U, false, long, kOpt>, gb, kThreads, s, a.chained, f, c, a, pf);
}

int launch_fluid_step_f32(const FluidF32& f, const CellsF32& c, const StepArgs& a, cudaStream_t s, int per_sm) {
  if (f.n == 0) return 0;
  if (a.walls != 0 || a.sph.n > 0) {
    const int g1 = grid_for(f.n, kThreads, per_sm);
    const bool i32 = f.n + 4L * g1 * kThreads < (1L << 32);
    i32 ? k_fluid_step_f32<1, true, uint32_t, 0><<<g1, kThreads, 0, s>>>(f, c, a, 0)
        : k_fluid_step_f32<1, true, long, 0><<<g1, kThreads, 0, s>>>(f, c, a, 0);
    return 1;
  }
  // particles per thread and round: kFluidBatch unless MPCD_FLUID_BATCH (1, 2) says otherwise;
  // options: kFluidOpt unless MPCD_FLUID_OPT (0..3: bit 0 prefetch, bit 1 aggregation) says otherwise
  static const int batch = [] {
    const char* e = std::getenv("MPCD_FLUID_BATCH");
    const int b = e ? std::atoi(e) : kFluidBatch;
    return b == 1 ? 1 : 2;
  }();
  static const int opt = [] {
    const char* e = std::getenv("MPCD_FLUID_OPT");
    const int o = e ? std::atoi(e) : kFluidOpt;
    return o & 3;
  }();
  switch (batch * 4 + opt) {
    case 4: launch_fluid_f32_opt<1, 0>(f, c, a, s, per_sm); break;
    case 5: launch_fluid_f32_opt<1, 1>(f, c, a, s, per_sm); break;
    case 6: launch_fluid_f32_opt<1, 2>(f, c, a, s, per_sm); break;
    case 7: launch_fluid_f32_opt<1, 3>(f, c, a, s, per_sm); break;
    case 8: launch_fluid_f32_opt<2, 0>(f, c, a, s, per_sm); break;
    case 9: launch_fluid_f32_opt<2, 1>(f, c, a, s, per_sm); break;
    case 10: launch_fluid_f32_opt<2, 2>(f, c, a, s, per_sm); break;
    default: launch_fluid_f32_opt<2, 3>(f, c, a, s, per_sm); break;
  }
  return 1;
}
int launch_last_fluid_step_f32(const FluidF32& f, const CellsF32& c, const StepArgs& a, cudaStream_t s) {
  launch_fluid_f32_opt<kFluidBatch, kOptPrefetch | kOptLast>(f, c, a, s, 4);
  return 1;
}
int launch_bin_fluid_f32(const FluidF32& f, const CellsF32& c, const StepArgs& a, cudaStream_t s) {
  if (f.n == 0) return 0;
  k_bin_fluid_f32<<<grid_for(f.n), kThreads, 0, s>>>(f, c, a);
  return 1;
}
int launch_bead_collide_f32(const MDState& m, const CellsF32& c, const StepArgs& a, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bead_collide_f32<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a);
  return 1;
}
int launch_bin_beads_f32(const MDState& m, const CellsF32& c, const StepArgs& a, cudaStream_t s) {
  if (m.nslots == 0) return 0;
  k_bin_beads_f32<<<grid_for(m.nslots), kThreads, 0, s>>>(m, c, a);
  return 1;
}
int launch_observables_f32(const FluidF32& f, const MDState& m, double bead_mass, double* out, cudaStream_t s) {
  long n = f.n > m.nslots ? f.n : m.nslots;
  k_observables_f32<<<grid_for(n) < 1024 ? grid_for(n) : 1024, kThreads, 0, s>>>(f, m, bead_mass, out);
  return 1;
}
int launch_sort_f32(FluidF32& f, FluidF32& tmp, const Box& box, uint32_t* count, uint32_t* start, uint32_t* rank,
                    uint32_t* blocksums, cudaStream_t s) {
  const long ncell = (long)box.L[0] * box.L[1] * box.L[2];
  cudaMemsetAsync(count, 0, ncell * sizeof(uint32_t), s);
  k_sort_count_f32<<<grid_for(f.n), kThreads, 0, s>>>(f.pos, f.n, box, count, rank);
  int k = 1 + scan_counts(count, ncell, start, blocksums, s);
  tmp.n = f.n;
  k_sort_scatter_f32<<<grid_for(f.n), kThreads, 0, s>>>(f, tmp, box, start, rank);
  FluidF32 t = f;
  f = tmp;
  tmp = t;
  return k + 1;
}

int launch_check_fluid(long n, const double* pos, const double* vel, unsigned* bad, cudaStream_t s) {
  if (n == 0) return 0;
  k_check_fluid<<<grid_for(3 * n), kThreads, 0, s>>>(n, pos, vel, bad);
  return 1;
}
int launch_load_fluid_f64(long n, const double* pos, const double* vel, const Box& box, const FluidF64& f,
                          cudaStream_t s) {
  if (n == 0) return 0;
  k_load_fluid_f64<<<grid_for(n), kThreads, 0, s>>>(n, pos, vel, box, f);
  return 1;
}
int launch_load_fluid_f32(long n, const double* pos, const double* vel, const Box& box, const FluidF32& f,
                          cudaStream_t s) {
  if (n == 0) return 0;
  k_load_fluid_f32<<<grid_for(n), kThreads, 0, s>>>(n, pos, vel, box, f);
  return 1;
}
int launch_convert_offsets(long n, uint64_t* o, bool integers, cudaStream_t s) {
  if (n == 0) return 0;
  k_convert_offsets<<<grid_for(n), kThreads, 0, s>>>(n, o, integers);
  return 1;
}
cudaError_t launch_store_beads(const MDState& m, long s0, long nb, double* pos, double* vel, unsigned* status,
                       const unsigned* err, cudaStream_t s) {
  return launch_in_chain(k_store_beads, grid_for(3 * nb, 128), 128, s, false, m, s0, (int)nb, pos, vel, status, err);
}
template <typename F>
cudaError_t launch_store_fluid(const F& f, double* pos, double* vel, unsigned* status, const unsigned* err, cudaStream_t s) {
  return launch_in_chain(k_store_fluid<F>, grid_for(f.n), kThreads, s, true, f, pos, vel, status, err);
}
template <typename F>
cudaError_t launch_find_particles(const F& f, uint32_t* at, unsigned* status, const unsigned* err, cudaStream_t s) {
  return launch_in_chain(k_find_particles<F>, grid_for(f.n, kThreads, 8), kThreads, s, true, f, at, status, err);
}
template <typename F>
cudaError_t launch_gather_fluid(const F& f, const uint32_t* at, long d0, long d1, bool velocity, double* out, unsigned* status,
                        cudaStream_t s) {
  return launch_in_chain(k_gather_fluid<F>, grid_for(d1 - d0, kThreads, 8), kThreads, s, false, f, at, d0, d1, velocity, out,
                         status);
}
#define MPCD_READ_BACK(F)                                                                                        \
  template cudaError_t launch_store_fluid(const F&, double*, double*, unsigned*, const unsigned*, cudaStream_t);         \
  template cudaError_t launch_find_particles(const F&, uint32_t*, unsigned*, const unsigned*, cudaStream_t);             \
  template cudaError_t launch_gather_fluid(const F&, const uint32_t*, long, long, bool, double*, unsigned*, cudaStream_t)
MPCD_READ_BACK(FluidF64);
MPCD_READ_BACK(FluidF32);
#undef MPCD_READ_BACK

}  // namespace mpcd
