// mpcd_fluid_step_noalloc: one split-precision MPC step of a plain fluid on
// caller-owned device arrays, for callers that cannot allocate device memory
// themselves (code running inside another runtime's memory pool or allocator,
// or plug-ins that are only handed pointers and a stream).  It calls no
// cudaMalloc, cudaFree or allocating library routine.
//
// Its per-cell scratch (velocity sums, counts and collision maps) lives in one
// file-scope static device array sized for kMaxCells cells.  Every GPU that
// loads the library holds that array until the process exits; every call
// shares it, so calls that overlap on the GPU (different streams or threads)
// race, and the array keeps the last call's contents (the sums are cleared at
// the start of each call).  A particle that breaks the layout (a cell index
// beyond the box, an offset outside [0,1)) is never binned, and the step then
// leaves every particle as it was.
//
// Bound by launches and by the wait for the result on all but the largest
// boxes.  One clear, three kernels and one copy back, with the check and the
// binning in one kernel, the refusal decided on the device and no sums made
// for a step that follows (3 clears, 4 kernels, 3 copies and a wait in the
// middle before): 11 x 9 x 13 cells 83 to 48 us, 39 x 40 x 42 106 to 61.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/mpcd_gpu.h"
#include "engine_internal.h"
#include "fluid_device.cuh"

using namespace mpcd;

namespace {

constexpr long kMaxCells = MPCD_NOALLOC_MAX_CELLS;
// layout: sums (float4 per cell) | counts (uint32 per cell) | Outcome, for the
// cells of the call and contiguous so that one clear covers them; maps (2
// float4 per cell) behind the room of the largest box
struct alignas(16) Outcome {
  double diss;        // dissipated energy
  unsigned err;       // error word
  unsigned rejected;  // a particle breaks the layout
};
constexpr size_t kSumBytes = sizeof(float4) * kMaxCells;
constexpr size_t kParBytes = 2 * sizeof(float4) * kMaxCells;
constexpr size_t kCntBytes = sizeof(uint32_t) * kMaxCells;
constexpr size_t kScratchBytes = kSumBytes + kParBytes + kCntBytes + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

struct DeviceScratch {
  bool ready = false;
  unsigned char* base = nullptr;  // device address of g_noalloc_scratch
};

std::mutex g_setup_mutex;
DeviceScratch g_scratch[64];

// Resolves the array's device address on the current device, once per device.
cudaError_t scratch_for_device(int dev, unsigned char** out) {
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch[dev].ready) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_scratch[dev].base = static_cast<unsigned char*>(p);
    g_scratch[dev].ready = true;
  }
  *out = g_scratch[dev].base;
  return cudaSuccess;
}

// Sums of the current shift.  Caller-packed particles are checked before they
// index the scratch: every axis' cell index below the box edge and every offset
// in [0,1) (NaN fails).  A bad particle sets *rejected.
__global__ void k_check_bin_f32(FluidF32 f, CellsF32 c, StepArgs a, unsigned* rejected) {
  const Box box = a.box;
  const float tcx = a.fta_cur[0], tcy = a.fta_cur[1], tcz = a.fta_cur[2];
  unsigned bad = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += (long)gridDim.x * blockDim.x) {
    const float4 p = f.pos[i], v = f.vel[i];
    const uint32_t cp = __float_as_uint(p.w);
    const bool ok = (cp >> 30) == 0u && cell_x(cp) < box.L[0] && cell_y(cp) < box.L[1] && cell_z(cp) < box.L[2] &&
                    p.x >= 0.0f && p.x < 1.0f && p.y >= 0.0f && p.y < 1.0f && p.z >= 0.0f && p.z < 1.0f;
    if (!ok) {
      bad = 1u;
      continue;
    }
    const long cid = shifted_f(cell_x(cp), p.x, tcx, box.L[0]) +
                     (long)box.L[0] * (shifted_f(cell_y(cp), p.y, tcy, box.L[1]) +
                                       (long)box.L[1] * shifted_f(cell_z(cp), p.z, tcz, box.L[2]));
    red_add_v4(c.sum + cid, make_float4(v.x, v.y, v.z, v.x * v.x + v.y * v.y + v.z * v.z));
    atomicAdd(c.cnt + cid, 1u);
  }
  if (bad) *rejected = 1u;
}

}  // namespace

extern "C" int mpcd_fluid_step_noalloc(const int* sizes, long n, void* pos, void* vel, double tstep,
                                       const double* a_cur, const double* a_next, unsigned long long seed,
                                       unsigned long long step, double* diss, void* stream) {
  if (!sizes || !a_cur || !a_next || n < 0 || (n > 0 && (!pos || !vel)) || !(tstep > 0)) return MPCD_EINVAL;
  long ncell = 1;
  for (int q = 0; q < 3; ++q) {
    if (sizes[q] < 2 || sizes[q] > 1024) return MPCD_EINVAL;
    ncell *= sizes[q];
  }
  if (ncell > kMaxCells) return MPCD_EINVAL;  // the box exceeds the static scratch
  for (int q = 0; q < 3; ++q)
    if (!(a_cur[q] >= 0.0 && a_cur[q] < 1.0) || !(a_next[q] >= 0.0 && a_next[q] < 1.0)) return MPCD_EINVAL;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return MPCD_ECUDA;
  unsigned char* base = nullptr;
  if (scratch_for_device(dev, &base) != cudaSuccess) return MPCD_ECUDA;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CellsF32 cells;
  cells.ncell = ncell;
  const size_t cnt_at = sizeof(float4) * (size_t)ncell;
  const size_t outcome_at = (cnt_at + sizeof(uint32_t) * (size_t)ncell + 15) & ~(size_t)15;
  cells.sum = reinterpret_cast<float4*>(base);
  cells.cnt = reinterpret_cast<uint32_t*>(base + cnt_at);
  cells.par = reinterpret_cast<float4*>(base + kSumBytes + kCntBytes + 256);
  Outcome* d_out = reinterpret_cast<Outcome*>(base + outcome_at);
  FluidF32 f;
  f.n = n;
  f.pos = static_cast<float4*>(pos);
  f.vel = static_cast<float4*>(vel);
  // clear what must start at zero: the sums, counts, energy and error words
  if (cudaMemsetAsync(base, 0, outcome_at + sizeof(Outcome), s) != cudaSuccess) return MPCD_ECUDA;
  StepArgs a{};
  for (int q = 0; q < 3; ++q) {
    a.box.L[q] = sizes[q];
    a.a_cur[q] = a_cur[q];
    a.a_next[q] = a_next[q];
    a.ta_cur[q] = 1.0 - a_cur[q];
    a.ta_next[q] = 1.0 - a_next[q];
    a.fta_cur[q] = (float)a.ta_cur[q];
    a.fta_next[q] = (float)a.ta_next[q];
  }
  a.h = tstep;
  a.fh = (float)tstep;
  a.bead_mass = 5.0;
  a.fbead_mass = 5.0f;
  a.seed = seed;
  a.step = step;
  a.err = &d_out->err;
  a.diss = &d_out->diss;
  a.skip = &d_out->rejected;
  a.chained = true;
  if (n > 0) {
    const long g = std::min<long>((n + 255) / 256, 4096);
    k_check_bin_f32<<<(int)g, 256, 0, s>>>(f, cells, a, &d_out->rejected);
    if (cudaGetLastError() != cudaSuccess) return MPCD_ECUDA;
  }
  launch_cell_params_f32(cells, a, s);  // collision maps
  if (n > 0) launch_last_fluid_step_f32(f, cells, a, s);  // collide, stream
  if (cudaGetLastError() != cudaSuccess) return MPCD_ECUDA;
  Outcome out{};
  if (cudaMemcpyAsync(&out, d_out, sizeof out, cudaMemcpyDeviceToHost, s) != cudaSuccess) return MPCD_ECUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return MPCD_ECUDA;
  if (out.rejected) return MPCD_EDEVICE;  // nothing was changed
  if (diss) *diss = out.diss;
  return out.err ? MPCD_EDEVICE : MPCD_OK;
}
