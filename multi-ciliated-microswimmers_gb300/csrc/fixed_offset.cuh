// In-cell offsets of the float64 fluid as 64-bit fixed point, and the few
// operations on them that the fluid pass needs, in integer arithmetic.
//
// An offset o in [0, 1) is the integer k = o 2^60.  GB300 completes about one
// float64 operation per clock and SM against 64 integer ones, and in float64 the
// fluid pass is bound by that pipe; streaming (x += v h), the wrap into the next cell
// and the comparison with the grid shift need none of it this way.  An offset that
// is not a multiple of 2^-60 (below 2^-7, so only in the first row of cells, where a
// position has more bits) is rounded to one when it is uploaded.
// The displacement v h is the truncated high part of the exact product of the
// two float64 significands, so its error is below 2 units of 2^-60 where the
// fused multiply-add on a float64 offset rounds to 2^-54 (offsets of one half
// and more).
//
// Host and device code alike (tests run it on the CPU).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef MPCD_HD
#ifdef __CUDACC__
#define MPCD_HD __host__ __device__ __forceinline__
#else
#define MPCD_HD inline
#endif
#endif

namespace mpcd {

constexpr int kOffBits = 60;
constexpr uint64_t kOffOne = 1ull << kOffBits;

MPCD_HD uint64_t f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, sizeof u);
  return u;
#endif
}
MPCD_HD uint64_t mul_hi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// The bits of the float nearest to x (ties to even, as a conversion rounds), for
// 2^-100 <= x < 2^100: the conversion itself is a float64 instruction.
MPCD_HD uint32_t nearest_float_bits(double x) {
  const uint64_t u = f64_bits(x);
  const uint64_t w = u + 0x0fffffffu + ((u >> 29) & 1u);
  return (uint32_t)((w - (896ull << 52)) >> 29);
}

// o in [0, 1) to the nearest unit (exact for o >= 2^-7: 53 bits end above 2^-60)
MPCD_HD uint64_t offset_from_double(double o) {
  const uint64_t k = (uint64_t)rint(o * (double)kOffOne);
  return k < kOffOne ? k : kOffOne - 1;
}
// the nearest float64 below 1
MPCD_HD double offset_to_double(uint64_t k) {
  const double o = (double)k * (1.0 / (double)kOffOne);
  return o < 1.0 ? o : 0x1.fffffffffffffp-1;
}

// Threshold t in [0, 1] of a comparison o >= t: the smallest k with k 2^-60 >= t.
MPCD_HD uint64_t offset_threshold(double t) { return (uint64_t)ceil(t * (double)kOffOne); }

// The time step as a normalised 64-bit significand m (2^63 <= m < 2^64) and
// exponent e: h = m 2^(e - 63).
struct FixedStep {
  uint64_t m = 0;
  int e = 0;
};
inline FixedStep fixed_step(double h) {
  FixedStep s;
  int ex = 0;
  const double f = std::frexp(h, &ex);  // h = f 2^ex, 1/2 <= f < 1
  s.m = (uint64_t)std::ldexp(f, 53) << 11;
  s.e = ex - 1;
  return s;
}

// Streams one coordinate: offset k, velocity v; the whole cells moved go to
// `cells`.  Returns false (k and cells unchanged) when |v| h may reach four
// cells or v is not finite.
MPCD_HD bool stream_fixed(uint64_t& k, int& cells, double v, const FixedStep& h) {
  const uint64_t b = f64_bits(v);
  const uint32_t hi = (uint32_t)(b >> 32);
  const int ev = (int)((hi >> 20) & 0x7ffu) - 1023 + h.e;  // |v| h < 2^(ev + 2)
  if (ev > 0) return false;
  // |v| = m 2^(e_v - 63) with m = significand << 11 (a subnormal v moves nothing)
  const uint64_t m = ((uint64_t)(((hi & 0xfffffu) | 0x100000u) << 11 | (uint32_t)b >> 21) << 32) | ((uint32_t)b << 11);
  const uint64_t p = mul_hi64(m, h.m);  // |v| h = p 2^(ev - 62) = (p >> (2 - ev)) units
  const int s = 2 - ev;
  const uint64_t d = s < 64 ? p >> s : 0ull;
  const int64_t sg = -(int64_t)(hi >> 31);
  const int64_t u = (int64_t)k + (((int64_t)d ^ sg) - sg);
  cells = (int)(u >> kOffBits);  // arithmetic: rounds down
  k = (uint64_t)u & (kOffOne - 1);
  return true;
}

}  // namespace mpcd
