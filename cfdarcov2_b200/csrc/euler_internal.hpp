// Shared state of the compressible Euler solver (euler.cu, euler_plain.cu).
//
// The time step lives on the device.  Launch s (counted from cfdb_euler_begin)
// reads the clock slot s%2 and the per-direction maximum signal speeds of ring
// slot s%3 (the state it advances), computes
//   dt = cfl / (lam_x/dx + lam_y/dy + lam_z/dz), clipped onto t_end,
// writes the speeds of the new state into ring slot (s+1)%3 and zeroes slot
// (s+2)%3 for launch s+1, and advances the clock into slot (s+1)%2.  The
// FP64 Neumaier totals of the new state: the plain path's reduction launch
// folds them itself (its last CTA); a fused launch leaves per-CTA partials
// (buffer s%2) and records its step in pending[s%2], and the next launch, or
// the report before the host reads the totals, folds them, so no launch
// ends waiting for a fold.  Once t_end is reached every further launch only
// copies the clock forward, so the host can enqueue steps without reading dt
// back (the reference syncs and copies a scalar every step,
// src/fvm3d.cpp:641-662, src/cuda_operators.cu:184-189).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "cfdb_internal.hpp"

struct EulerClock {
  double t[2];
  unsigned long long lam[3][3];  // non-negative doubles as ordered bit patterns
  long long steps[2];
  int finished[2];
  unsigned int counter;  // last-CTA counter of the plain path's reduction, reset by the last CTA
  int pad;
  long long pending[2];  // fused launch s: the step whose partials (buffer s%2) are not folded yet, 0 for none
};

// Neumaier pair, two fields (rho, E).
struct Comp2 {
  double s0, c0, s1, c1;
};

struct cfdb_euler {
  cfdb_ctx* ctx = nullptr;
  cfdb_mesh* mesh = nullptr;
  int dtype = CFDB_F32;
  int path = CFDB_PATH_FUSED;
  double gamma = 1.4, cfl = 0.4, t_end = 0.2;
  int64_t max_steps = 0;
  EulerClock* clock = nullptr;
  double* totals = nullptr;  // 2 * (max_steps + 1)
  Comp2* part = nullptr;     // per-CTA partials: two buffers of part_cap (the fused path alternates them)
  int part_cap = 0;
  int fused_grid = 0;     // CTAs of the last fused launch (the partials it left)
  int fused_threads = 0;  // and their size (the fold runs in the same order)
  int64_t launches = 0;
};

// The host-visible snapshot of the clock after `launches` launches.
inline int euler_slot(int64_t launches) { return int(launches & 1); }

// box_ops.cu: the plain step on structured meshes without face arrays
int box_euler_step(cfdb_euler* e, const void* U, void* Un, int64_t step);

__host__ __device__ inline double euler_dt(const double lam[3], double dx, double dy, double dz, double cfl,
                                           double t, double t_end, bool* last) {
  const double rate = (lam[0] / dx + lam[1] / dy) + lam[2] / dz;
  double dt = cfl / rate;
  *last = false;
  if (dt >= t_end - t) {
    dt = t_end - t;
    *last = true;
  }
  return dt;
}

#if defined(__CUDACC__)
__device__ __forceinline__ double bits_to_double(unsigned long long b) { return __longlong_as_double((long long)b); }

__device__ __forceinline__ void comp_add(double& s, double& c, double x) {
  const double t = s + x;
  if (fabs(s) >= fabs(x)) c += (s - t) + x; else c += (x - t) + s;
  s = t;
}

// Folds the per-CTA FP64 partials part[0 .. nblocks) into totals row `step`
// with every thread of the calling CTA, in a fixed order: thread t takes
// partials t, t + blockDim, ..., the lanes of each warp merge through
// shuffles in a fixed pattern and thread 0 merges the warps in order, so the
// totals do not depend on timing (one thread folding every partial serially
// had cost ~13 us per fused step and ~20 us per reduction launch).  Partials
// written by the same launch are read from L2.
static __device__ void fold_partials(const Comp2* __restrict__ part, int nblocks, double* totals, long long step) {
  __shared__ double sh[32][4];
  double S0 = 0, C0 = 0, S1 = 0, C1 = 0;
  for (int k = int(threadIdx.x); k < nblocks; k += int(blockDim.x)) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(part + k)), b = __ldcg(reinterpret_cast<const double2*>(part + k) + 1);
    comp_add(S0, C0, a.x); C0 += a.y;
    comp_add(S1, C1, b.x); C1 += b.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double a0 = __shfl_xor_sync(0xffffffffu, S0, o), b0 = __shfl_xor_sync(0xffffffffu, C0, o);
    const double a1 = __shfl_xor_sync(0xffffffffu, S1, o), b1 = __shfl_xor_sync(0xffffffffu, C1, o);
    comp_add(S0, C0, a0); C0 += b0;
    comp_add(S1, C1, a1); C1 += b1;
  }
  const int w = int(threadIdx.x) >> 5;
  if ((threadIdx.x & 31) == 0) {
    sh[w][0] = S0; sh[w][1] = C0; sh[w][2] = S1; sh[w][3] = C1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    S0 = C0 = S1 = C1 = 0;
    for (int k = 0; k < int(blockDim.x / 32); ++k) {
      comp_add(S0, C0, sh[k][0]); C0 += sh[k][1];
      comp_add(S1, C1, sh[k][2]); C1 += sh[k][3];
    }
    totals[2 * step] = S0 + C0;
    totals[2 * step + 1] = S1 + C1;
  }
}
#endif

// euler_plain.cu
int euler_plain_step(cfdb_euler* e, const void* U, void* Un, int64_t s);
int euler_reduce(cfdb_euler* e, const void* U, int64_t s, int begin_mode);
int euler_reduce_grid(const cfdb_euler* e);
// euler.cu
int euler_fused_step(cfdb_euler* e, const void* U, void* Un, int64_t s);
int euler_fused_grid(const cfdb_euler* e);
