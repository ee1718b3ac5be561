// Exchange of bead positions between the tiles of the entries kernel
// (md_entries.cu) as tagged packets through L2.
#pragma once
#include <cstdint>

#include "df32.cuh"
#include "engine_internal.h"

namespace mpcd {

namespace {

// polls of a packet before giving up (each an L2 round trip: a second or two)
constexpr uint32_t kPollLimit = 1u << 21;
// packets one thread polls at a time (their loads in flight together)
constexpr int kPollBatch = 3;

// the launch arguments' dt and dt / 2 as pairs
inline void md_set_dt_pairs(MDStepArgs& a) {
  const dfloat d = df_from_double(a.dt), h = df_from_double(a.dt / 2.0);
  a.dt_pair = {d.h, d.l};
  a.dt2_pair = {h.h, h.l};
}

// A position buffer holds the packets of coordinate k of all slots at
// k nslots: threads polling neighbouring beads read neighbouring packets (a
// warp's loads of 48-byte strided packets took three times as long).

// One coordinate of a bead as it travels between tiles: the offset's pair,
// the cell, and the tag of the evaluation; stored and loaded by single
// 128-bit accesses (single-copy atomic), so that the tag vouches for the rest.
struct Packet {
  uint32_t h, l, c, tag;
};
__device__ __forceinline__ void packet_store(uint4* p, const Packet& k) {
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\t.reg .b128 t;\n\t"
      "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b128 t, {a, b};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "r"(k.h), "r"(k.l), "r"(k.c), "r"(k.tag)
      : "memory");
}
__device__ __forceinline__ Packet packet_load(const uint4* p) {
  Packet k;
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\t.reg .b128 t;\n\t"
      "ld.relaxed.gpu.global.b128 t, [%4];\n\tmov.b128 {a, b}, t;\n\t"
      "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
      : "=r"(k.h), "=r"(k.l), "=r"(k.c), "=r"(k.tag)
      : "l"(p)
      : "memory");
  return k;
}

// true once a poll has run for kPollLimit turns, or another thread of the CTA
// has given up: reports kErrBarrier and sets *fail
__device__ __forceinline__ bool poll_given_up(uint32_t spins, unsigned* err, int* fail) {
  if (spins <= kPollLimit && ((spins & 1023u) != 1023u || *(volatile int*)fail == 0)) return false;
  atomicOr(err, kErrBarrier);
  *fail = 1;
  return true;
}

// polls the three packets of two beads (slots s1, s2) until all six carry `tag`
__device__ __forceinline__ void receive_two(const uint4* src, int nslots, uint32_t tag, int s1, int s2, Packet (&d)[6],
                                            unsigned* err, int* fail) {
  bool ok = false;
  for (uint32_t spins = 0; !ok; ++spins) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      d[k] = packet_load(src + (size_t)k * nslots + s1);
      d[3 + k] = packet_load(src + (size_t)k * nslots + s2);
    }
    ok = true;
#pragma unroll
    for (int k = 0; k < 6; ++k) ok = ok && d[k].tag == tag;
    if (!ok && poll_given_up(spins, err, fail)) break;
  }
}

// Polls the packets of hn halo beads (packet p: coordinate p / hn of halo bead
// p mod hn) of evaluation `tag` until all have come and hands each to
// put(bead, coordinate, packet).  `first`: this thread's first packet, nthr apart from
// the next; kPollBatch of them are in flight together (indices past the end
// read the last packet again).  Bounded, as poll_given_up.
template <typename Put>
__device__ __forceinline__ void receive_packets(const uint4* src, int nslots, uint32_t tag, int hn, const int* hslot,
                                                int first, int nthr, unsigned* err, int* fail, Put&& put) {
  const int np = 3 * hn;
#pragma unroll 1
  for (int p0 = first; p0 < np; p0 += kPollBatch * nthr) {
    Packet d[kPollBatch];
    const uint4* at[kPollBatch];
#pragma unroll
    for (int u = 0; u < kPollBatch; ++u) {
      const int p = min(p0 + u * nthr, np - 1);
      const int k = (p >= hn) + (p >= 2 * hn);
      at[u] = src + (size_t)k * nslots + hslot[p - k * hn];
    }
    bool ok = false;
    for (uint32_t spins = 0; !ok; ++spins) {
#pragma unroll
      for (int u = 0; u < kPollBatch; ++u) d[u] = packet_load(at[u]);
      ok = true;
#pragma unroll
      for (int u = 0; u < kPollBatch; ++u) ok = ok && d[u].tag == tag;
      if (!ok && poll_given_up(spins, err, fail)) break;
    }
#pragma unroll
    for (int u = 0; u < kPollBatch; ++u) {
      const int p = p0 + u * nthr;
      const int k = (p >= hn) + (p >= 2 * hn);
      if (p < np) put(p - k * hn, k, d[u]);
    }
  }
}

}  // namespace

}  // namespace mpcd
