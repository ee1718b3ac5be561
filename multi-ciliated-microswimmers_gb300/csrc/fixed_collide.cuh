// The SRD collision of the float64 fluid in 64-bit fixed point: the collision
// map of a cell from its sums, and its application to a particle.
//
// GB300 issues about one float64 operation per clock and SM against 64 and
// more 32-bit integer ones, so that a float64 multiply-add costs as much as
// about fifty integer instructions: with the map, the kinetic energy and the
// streaming in float64 the fluid pass and the cell maps were bound by that
// pipe (73-82 % busy, everything else idle).  A 64 x 64 product takes three or
// four 32 x 32 -> 64 multiply-adds here.
//
// All quantities are two's-complement integers times a power of two chosen so
// that the thermal range has bits to spare: velocities and mean velocities in
// units of 2^-58, new velocities 2^-56, map entries 2^-59, axis components and
// the thermostat factor 2^-60, a cell's kinetic energy and momentum 2^-55 (2^-50 and
// 2^-52 from 128 on).  What enters is truncated (less than one unit), a product is
// within one unit, against half of 2^-53 for float64 numbers of one half and more:
// results are at least as close to the exact ones as the float64 form's wherever
// the terms of a sum are of order one.  What does not fit (velocities of 16
// thermal velocities and more, mean velocities of 8, thermostat factors of 8, of 2
// where the mean velocity is 2, kinetic energies of a cell of 4096, momenta of
// 512, cells colder than 1/16, non-finite values) takes the float64 form, about
// half as fast; a warp with one such particle makes both.  The factor's limit is what
// counts at low densities: with 2 in place of 8, 4 % of the particles of a box with
// three per cell were beyond it, in half of the warps, and 0.1 % with ten per cell
// (64^3 cells, us per step, limit 2 / limit 8 / all in float64: two per cell 92 / 58 / 77,
// three 109 / 66 / 90, ten 125 / 120 / 182, twenty 201 / 207 / 313).
//
// Host and device code alike (tests run it on the CPU).
#pragma once
#include "fixed_offset.cuh"

namespace mpcd {

MPCD_HD double bits_f64(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, sizeof x);
  return x;
#endif
}
MPCD_HD int clz64(uint64_t x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// x in units of 2^-BITS, truncated towards zero; |x| < 2^EMAX, BITS + EMAX <= 62.
// False (r unchanged) for larger values, infinities and NaN.
template <int BITS, int EMAX>
MPCD_HD bool to_fixed(double x, int64_t& r) {
  static_assert(BITS + EMAX <= 62 && BITS + EMAX >= 53, "significand shifted left, sign kept");
  const uint64_t b = f64_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
  if ((hi & 0x7fffffffu) >= (uint32_t)(1023 + EMAX) << 20) return false;
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << (BITS + EMAX - 53);
  const int s = 1022 + EMAX - (int)((hi >> 20) & 0x7ffu);
  const int64_t d = s < 64 ? (int64_t)(m >> s) : 0;
  const int64_t sg = -(int64_t)(hi >> 31);
  r = (d ^ sg) - sg;
  return true;
}

// x 2^-bits to the nearest float64
MPCD_HD double from_fixed(int64_t x, int bits) {
  const uint64_t sg = (uint64_t)x >> 63;
  const uint64_t m = sg ? 0ull - (uint64_t)x : (uint64_t)x;
  if (m == 0) return 0.0;
  const int lz = clz64(m);
  const uint64_t n = m << lz;
  const uint64_t mant = (n >> 11) + ((n >> 10) & 1u);  // 2^52 .. 2^53
  return bits_f64((sg << 63) | (((uint64_t)(1023 + 63 - lz - bits - 1) << 52) + mant));
}

// h 2^32 + l with a signed low half: products of halves need no correction
struct Limbs {
  int32_t h, l;
};
MPCD_HD Limbs split_limbs(int64_t x) {
  const int32_t l = (int32_t)(uint32_t)x;
  return {(int32_t)((uint64_t)x >> 32) + (l < 0 ? 1 : 0), l};
}
MPCD_HD int64_t wide(int32_t a, int32_t b) { return (int64_t)a * b; }
MPCD_HD uint64_t uwide(int32_t a, int32_t b) { return (uint64_t)((int64_t)a * b); }

// a b 2^-S, rounded to within one unit; |a|, |b| <= 2^62 and the result within 2^62
template <int S>
MPCD_HD int64_t mul_sh(Limbs a, Limbs b) {
  static_assert(S >= 34 && S <= 63, "shift");
  const int64_t mid = wide(a.h, b.l) + wide(a.l, b.h) + (wide(a.l, b.l) >> 32) + (1ll << (S - 33));
  return (int64_t)((uint64_t)wide(a.h, b.h) << (64 - S)) + (mid >> (S - 32));
}

// ------------------------------------------------------------ the map ---
// Twelve words per cell, four per row i: A_i0, A_i1, A_i2 (units of 2^-59, each a
// Limbs) and b_i (units of 2^-56) of v' = A v + b.  A cell whose numbers do not
// fit holds kMapF64 in its first word instead, and the thermostat factor, the
// rotation axis and the mean velocity as float64 in the next seven.
constexpr int kVelBits = 58;         // velocities that go in, up to 16; mean velocities
constexpr int kMapBits = 59;         // entries of A
constexpr int kAxisBits = 60;        // axis components, thermostat factor
constexpr int kOutBits = 56;         // velocities that come out, below 128 (apply_words)
constexpr int64_t kMeanMax = 1ll << 61;  // 8, mean velocities
constexpr int64_t kMeanMaxHot = 1ll << 59;  // 2, where the thermostat factor is 2 or more
constexpr float kGammaMax = 4096.f;         // and the Gamma variate there
constexpr uint64_t kMapF64 = 0x7fffffff00000000ull;

MPCD_HD Limbs word_limbs(uint64_t w) { return {(int32_t)(w >> 32), (int32_t)(uint32_t)w}; }
// The first word of a map: an entry of A is below 2 (29 bits and a sign in its
// high limb), so that bit 62 differs from the sign only where it was flipped to say
// that A is held divided by four.  kMapF64 is neither.
MPCD_HD int word_scale(uint64_t w) { return (int)((w ^ (w << 1)) >> 62) & 2; }
MPCD_HD Limbs first_limbs(uint64_t w) {
  return {(int32_t)((uint32_t)(w >> 32) << 2) >> 2, (int32_t)(uint32_t)w};
}

// 8 M in units of 2^-PB, for whole numbers of particles and for any mass, as far
// as it matters to momenta in 62 bits.
constexpr int kMomentumBits = 52;
template <int PB = kMomentumBits>
MPCD_HD int64_t mean_limit(int num) {
  constexpr int most = 1 << (59 - PB);
  return (int64_t)(num < most ? num : most) << (PB + 3);
}
template <int PB = kMomentumBits>
MPCD_HD int64_t mean_limit(double mass) {
  constexpr double most = 1 << (59 - PB);
  return (int64_t)((mass < most ? mass : most) * (double)(1ll << (PB + 3)));
}
// The mean velocity u (units of 2^-58) and the kinetic energy K - M u^2 relative
// to it (units of 2^-KB) of a cell with momentum p (each below 2^PE), kinetic energy kin
// (units of 2^-KB, below 2^62) and mass M, inv = 1 / M in units of 2^-62.  top: 8 M in
// units of 2^-PB; a momentum that reaches it is refused before the product can
// wrap.  False if the numbers do not fit.
template <int PB = kMomentumBits, int PE = 9, int KB = 50>
MPCD_HD bool cell_mean(const double* p, int64_t kin, int64_t inv, int64_t top, int64_t* u, int64_t& erel) {
  int64_t q[3];
  if (!(to_fixed<PB, PE>(p[0], q[0]) && to_fixed<PB, PE>(p[1], q[1]) && to_fixed<PB, PE>(p[2], q[2]))) return false;
  bool fit = true;
#pragma unroll
  for (int i = 0; i < 3; ++i) fit = fit && q[i] < top && q[i] > -top;
  if (!fit) return false;
  const Limbs iv = split_limbs(inv);
  uint64_t rel = (uint64_t)kin;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const Limbs l = split_limbs(q[i]);
    u[i] = mul_sh<PB + 4>(l, iv);
    fit = fit && u[i] < kMeanMax && u[i] > -kMeanMax;
    rel -= (uint64_t)mul_sh<58 + PB - KB>(split_limbs(u[i]), l);
  }
  erel = (int64_t)rel;
  return fit;
}
// A cell's kinetic energy in units of 2^-55 below 128 (ten thermal particles hold
// 30), else of 2^-50; 0 if it does not fit.
MPCD_HD int kinetic_fixed(double K, int64_t& kin) { return to_fixed<55, 7>(K, kin) ? 55 : (to_fixed<50, 12>(K, kin) ? 50 : 0); }
// 8 M in the units of the momenta that go with it
template <typename M>
MPCD_HD int64_t mean_top(int bits, M mass) { return bits == 55 ? mean_limit<55>(mass) : mean_limit(mass); }
// cell_mean in the units of kinetic_fixed.  A cell whose particles differ by too
// little from each other (a single one: from rest) is refused: below an energy of
// 1/16 the units are coarser than float64, and below one unit nothing would be left
// for the thermostat to scale.
MPCD_HD bool cell_energy(const double* p, int64_t kin, int bits, int64_t inv, int64_t top, bool single, int64_t* u,
                         int64_t& erel) {
  const bool fit = bits == 55 ? cell_mean<55, 7, 55>(p, kin, inv, top, u, erel) : cell_mean(p, kin, inv, top, u, erel);
  return fit && (single ? kin : erel) >= 1ll << (bits - 4);
}

// a float in (-2, 2) in units of 2^-60
MPCD_HD int64_t axis_fixed(float f) {
#ifdef __CUDA_ARCH__
  const uint32_t u = __float_as_uint(f);
#else
  uint32_t u;
  std::memcpy(&u, &f, sizeof u);
#endif
  const int s = 127 - (int)((u >> 23) & 0xffu);
  const int64_t d = s < 64 ? (int64_t)((uint64_t)((u & 0x7fffffu) | 0x800000u) << 37 >> s) : 0;
  return (u >> 31) ? -d : d;
}
// r (units of 2^-60, |r|^2 = 1 + e with |e| < 2^-20) to unit length: r (1 - e/2 + 3 e^2/8)
MPCD_HD void axis_normalise(int64_t* r) {
  const Limbs x = split_limbs(r[0]), y = split_limbs(r[1]), z = split_limbs(r[2]);
  const int64_t e = mul_sh<60>(x, x) + mul_sh<60>(y, y) + mul_sh<60>(z, z) - (1ll << 60);
  const int32_t e8 = (int32_t)(e >> 12);
  const int64_t e2 = wide(e8, e8) >> 36;  // e^2
  const Limbs d = split_limbs((e >> 1) - ((3 * e2) >> 3));
  r[0] -= mul_sh<60>(x, d);
  r[1] -= mul_sh<60>(y, d);
  r[2] -= mul_sh<60>(z, d);
}

// constants in units of 2^-60: cos and sin of the rotation angle as the
// reference uses them (src/libcilia/mpcd.h:72-76)
MPCD_HD int64_t unit60(double x) { return (int64_t)(x * 1152921504606846976.0); }

// The rotation (units of 2^-60) about the axis r (2^-60), with the entries of
// src/libcilia/mpcd.cpp:285-293 (R_ii = r_i^2 (1 - ca) + ca, R_ij = r_i r_j (1 -
// ca) -+ r_k sa).
MPCD_HD void rotation_fixed(const int64_t* r, double cos_a, double sin_a, int64_t* R) {
  const Limbs x = split_limbs(r[0]), y = split_limbs(r[1]), z = split_limbs(r[2]);
  const Limbs oc = split_limbs(unit60(1.0 - cos_a)), sa = split_limbs(unit60(sin_a));
  const int64_t ca = unit60(cos_a);
  const Limbs tx = split_limbs(mul_sh<60>(x, oc)), ty = split_limbs(mul_sh<60>(y, oc)), tz = split_limbs(mul_sh<60>(z, oc));
  const int64_t sx = mul_sh<60>(x, sa), sy = mul_sh<60>(y, sa), sz = mul_sh<60>(z, sa);
  const int64_t xy = mul_sh<60>(tx, y), xz = mul_sh<60>(tx, z), yz = mul_sh<60>(ty, z);
  R[0] = mul_sh<60>(tx, x) + ca;
  R[1] = xy - sz;
  R[2] = xz + sy;
  R[3] = xy + sz;
  R[4] = mul_sh<60>(ty, y) + ca;
  R[5] = yz - sx;
  R[6] = xz - sy;
  R[7] = yz + sx;
  R[8] = mul_sh<60>(tz, z) + ca;
}
// Row i of the map's words from that row of R, the factor sc (2^-60) and the
// mean velocity u (2^-58): A = sc R, b = u - A u.  With s = 2 the factor is 4 sc: A is
// held divided by four (word_scale).
MPCD_HD void map_row(int i, const int64_t* row, int64_t sc, const int64_t* u, uint64_t* w, int s = 0) {
  const Limbs f = split_limbs(sc);
  int64_t b = (u[i] + 1) >> 1;  // 2^-57
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const Limbs a = split_limbs(mul_sh<61>(split_limbs(row[j]), f));
    w[j] = (uint64_t)(uint32_t)a.h << 32 | (uint32_t)a.l;
    b -= (int64_t)((uint64_t)mul_sh<60>(a, split_limbs(u[j])) << s);
  }
  w[3] = (uint64_t)((b + 1) >> 1);
  if (i == 0 && s) w[0] ^= 1ull << 62;
}
MPCD_HD void map_words(const int64_t* r, int64_t sc, const int64_t* u, double cos_a, double sin_a, uint64_t* w, int s = 0) {
  int64_t R[9];
  rotation_fixed(r, cos_a, sin_a, R);
#pragma unroll
  for (int i = 0; i < 3; ++i) map_row(i, R + 3 * i, sc, u, w + 4 * i, s);
}

// v' = A v + b in units of 2^-56, for |v_i| < 16 of a particle that is in the cell.
// The sums are taken modulo 2^64; the result, |u| + sc |v - u|, is below 2^7: with sc < 2
// and |u_i| < 8 by these limits, with sc < 8 because sc |v - u| is at most the root of sc^2
// E_rel = 2 g, g < kGammaMax.  The products of low halves are left out (up to two units
// each, 1.2 together in the mean square; four times that where A is held divided
// by four, whose float64 form rounds as much more coarsely).
MPCD_HD void apply_words(const uint64_t* w, const int64_t* v, int64_t* out) {
  const Limbs x = split_limbs(v[0]), y = split_limbs(v[1]), z = split_limbs(v[2]);
  const int s = word_scale(w[0]);
  const uint32_t half = 1u << (28 - s);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const Limbs a = i ? word_limbs(w[4 * i]) : first_limbs(w[0]), b = word_limbs(w[4 * i + 1]), c = word_limbs(w[4 * i + 2]);
    const uint64_t top = uwide(a.h, x.h) + uwide(b.h, y.h) + uwide(c.h, z.h);
    const uint64_t mid = uwide(a.h, x.l) + uwide(b.h, y.l) + uwide(c.h, z.l) + uwide(a.l, x.h) + uwide(b.l, y.h) + uwide(c.l, z.h);
    out[i] = (int64_t)((top << (3 + s)) + (uint64_t)((int64_t)(mid + half) >> (29 - s)) + w[4 * i + 3]);
  }
}

// sum of v_i^2 in units of 2^-52, v_i in units of 2^-58 with |v_i| < 16
constexpr int kSquareBits = 52;
// A sum of such squares, or of cells' kinetic energies in units of 2^-55: 96 bits,
// every addend whole, so that the sum is exact whatever the number of addends.
struct EnergySum {
  uint64_t lo = 0;
  uint32_t hi = 0;
};
MPCD_HD void energy_add(EnergySum& e, uint64_t lo, uint32_t hi) {
  e.lo += lo;
  e.hi += hi + (e.lo < lo ? 1u : 0u);
}
constexpr int kCellEnergyBits = 55;
MPCD_HD void energy_add_cell(EnergySum& e, int64_t kin, int bits) {  // of kinetic_fixed
  const int sh = kCellEnergyBits - bits;
  energy_add(e, (uint64_t)kin << sh, sh ? (uint32_t)((uint64_t)kin >> (64 - sh)) : 0u);
}
MPCD_HD double energy_value(const EnergySum& e, int bits) {
  const double unit = 1.0 / (double)(1ull << bits);
  return (double)e.lo * unit + (double)e.hi * (18446744073709551616.0 * unit);
}
MPCD_HD int64_t square_words(Limbs x, Limbs y, Limbs z) {
  const int64_t top = wide(x.h, x.h) + wide(y.h, y.h) + wide(z.h, z.h);
  const int64_t mid = wide(x.h, x.l) + wide(y.h, y.l) + wide(z.h, z.l);
  return top + (mid >> 31);
}

// The time step for stream_words in units of 2^-61 (exact for 2^-9 <= h < 2),
// and the high word of the velocity bound (units of 2^-56) below which |v| < 16
// and |v| h < 4.  The bound is zero for larger steps: all in float64.
struct StreamStep {
  Limbs h = {0, 0};
  int32_t vmax = 0;
};
// kick: a change of the velocity that is added after the bound was checked,
// returned in units of 2^-56.
inline StreamStep stream_step(double h, double kick, int64_t* xkick) {
  StreamStep s;
  *xkick = 0;
  if (!(h >= 0 && h < 2 && std::fabs(kick) < 8)) return s;
  s.h = split_limbs(std::llround(std::ldexp(h, 61)));
  *xkick = std::llround(std::ldexp(kick, kOutBits));
  s.vmax = (int32_t)std::floor(std::ldexp(std::fmin(16.0 - std::fabs(kick), 4.0 / h), kOutBits - 32));
  return s;
}
// Streams an offset by v h, v in units of 2^-58.
MPCD_HD void stream_words(uint64_t& k, int& cells, Limbs v, const StreamStep& s) {
  const int64_t u = (int64_t)k + mul_sh<59>(v, s.h);
  cells = (int)(u >> kOffBits);
  k = (uint64_t)u & (kOffOne - 1);
}

}  // namespace mpcd
