// Cluster-resident heat solver for meshes small enough to live on chip: the
// whole field stays in the registers and the distributed shared memory of one
// thread-block cluster of up to 16 CTAs, every time step runs inside ONE launch
// and the steps are separated by the cluster barrier instead of a kernel boundary.
//
// CTA c owns the x slab [c X / CL, (c+1) X / CL).  A thread owns four z cells of
// two rows on every plane of the slab and keeps them in registers from step to
// step: its x neighbours are its own registers (the slab's end planes read the
// adjacent CTAs' planes through distributed shared memory), z neighbours are the
// adjacent lanes, and only the rows beside its own come from shared memory, where
// every plane is published each step (two buffers).  The plane that waits for the
// lower neighbour's copy is computed last, behind the others.
//
// What bounds a step is shared-memory bandwidth on the cluster's SMs: a thread
// that read all of its neighbours from shared memory and one row at a time moved
// 26 B per cell and step (64^3: 3.1 us per step); now it is 10 B and a step takes 2.1 us, half of it
// issue on the cluster's SMs, the rest the cluster barrier and one remote load.  The cell update is
// heat_update() (heat_cell.cuh) in packed pairs, operation by operation, so the
// results are those of the one-step sweep bit for bit.
//
// Long thin fields (more planes than the registers hold, few cells in each) keep
// both buffers in shared memory alone (heat_slab_k), where that is faster than several
// steps per pass over all SMs (heat_blocked.cu), which take the larger ones.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "cfdb_internal.hpp"
#include "f32x2.cuh"
#include "heat_cell.cuh"

CFDB_MODULE_ANCHOR

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;    // at most: row pairs x z groups
constexpr int kMaxCluster = 16;  // non-portable cluster size
constexpr int kMaxPlanes = 4;    // planes per slab (eight spill registers)
constexpr int kSlabThreads = 1024;
constexpr int kMaxGroups = 8;    // heat_slab_k: groups of four z cells per thread and step

struct ResidentArgs {
  int X, Y, Z;
  int P;  // planes per buffer (the largest slab)
  int steps;
  float cx, cy, cz;
};

struct Quad {
  float2 a, b;  // cells 0, 1 and 2, 3
};
__device__ __forceinline__ Quad ldq(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void stq(float* p, const Quad& c) {
  *reinterpret_cast<float4*>(p) = make_float4(c.a.x, c.a.y, c.b.x, c.b.y);
}
__device__ __forceinline__ Quad operator-(const Quad& x, const Quad& y) { return {f2::sub(x.a, y.a), f2::sub(x.b, y.b)}; }
__device__ __forceinline__ Quad operator+(const Quad& x, const Quad& y) { return {f2::add(x.a, y.a), f2::add(x.b, y.b)}; }

template <int P>
__global__ void __launch_bounds__(kThreads, 1)
    heat_resident_k(const float* __restrict__ in, float* __restrict__ out, ResidentArgs a) {
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int c = int(cl.block_rank());
  const int CL = int(cl.num_blocks());
  const int x0 = int((long long)c * a.X / CL), x1 = int((long long)(c + 1) * a.X / CL);
  const int np = x1 - x0;
  const int plane = a.Y * a.Z;
  const int buf = a.P * plane;  // floats per buffer
  const int zq = a.Z / 4;
  const int tid = int(threadIdx.x), lane = tid & 31;
  const int pair = tid / zq;
  const bool act = 2 * pair < a.Y;       // the last warp may be ragged
  const int y = act ? 2 * pair : 0, z = 4 * (tid - pair * zq);
  const bool two = y + 1 < a.Y;          // the pair's second row exists
  const int at = y * a.Z + z;
  const int second = two ? at + a.Z : at;
  const int below = y > 0 ? at - a.Z : at, above = y + 2 < a.Y ? at + 2 * a.Z : second;
  const bool zlo = z == 0, zhi = z + 4 == a.Z;
  const bool first = lane == 0 && !zlo, last = lane == 31 && !zhi;
  const float2 cx = f2::splat(a.cx), cy = f2::splat(a.cy), cz = f2::splat(a.cz);

  Quad v[P][2];
  {
    const float* src = in + (long long)x0 * plane;
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (p < np) {
        v[p][0] = ldq(src + (long long)p * plane + at);
        v[p][1] = ldq(src + (long long)p * plane + second);
        if (act) {
          stq(sm + p * plane + at, v[p][0]);
          if (two) stq(sm + p * plane + second, v[p][1]);
        }
      }
  }
  // the planes next to ours in the neighbour slabs
  const float* lo = c > 0 ? cl.map_shared_rank(sm, c - 1) + ((x0 - 1) - int((long long)(c - 1) * a.X / CL)) * plane : nullptr;
  const float* hi = c < CL - 1 ? cl.map_shared_rank(sm, c + 1) : nullptr;
  cl.sync();

  // one plane: t and its x neighbours m, q in registers, rows beside the pair in A
  auto update = [&](const Quad t[2], const Quad m[2], const Quad q[2], const float* A, Quad n[2]) __attribute__((always_inline)) {
    const Quad yb = ldq(A + below), ya = ldq(A + above);
    const Quad dy = two ? t[1] - t[0] : t[0] - t[0];
    const Quad ly[2] = {dy + (yb - t[0]), (ya - t[1]) - dy};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const Quad& w = t[r];
      float l = __shfl_up_sync(0xffffffffu, w.b.y, 1), h = __shfl_down_sync(0xffffffffu, w.a.x, 1);
      const int o = r ? second : at;
      if (first) l = A[o - 1];  // the neighbour is in another warp
      if (last) h = A[o + 4];
      l = zlo ? w.a.x : l;
      h = zhi ? w.b.y : h;
      const float d0 = __fsub_rn(w.a.y, w.a.x), d1 = __fsub_rn(w.b.x, w.a.y), d2 = __fsub_rn(w.b.y, w.b.x);
      const Quad lz = {make_float2(__fadd_rn(d0, __fsub_rn(l, w.a.x)), __fsub_rn(d1, d0)),
                       make_float2(__fsub_rn(d2, d1), __fsub_rn(__fsub_rn(h, w.b.y), d2))};
      const Quad lx = (q[r] - w) + (m[r] - w);
      n[r].a = f2::add(w.a, f2::fma(cx, lx.a, f2::fma(cy, ly[r].a, f2::mul(cz, lz.a))));
      n[r].b = f2::add(w.b, f2::fma(cx, lx.b, f2::fma(cy, ly[r].b, f2::mul(cz, lz.b))));
    }
  };

  for (int s = 0; s < a.steps; ++s) {
    const float* A = sm + (s & 1) * buf;
    float* B = sm + ((s + 1) & 1) * buf;
    // planes x0 - 1 and x1 from the neighbour slabs, the end planes themselves on
    // a wall
    const float* const below_x = lo ? lo + (s & 1) * buf : A;
    const float* const above_x = hi ? hi + (s & 1) * buf : A + (np - 1) * plane;
    const Quad L[2] = {ldq(below_x + at), ldq(below_x + second)}, H[2] = {ldq(above_x + at), ldq(above_x + second)};
    auto put = [&](int p, const Quad n[2]) __attribute__((always_inline)) {
      if (act) {
        stq(B + p * plane + at, n[0]);
        if (two) stq(B + p * plane + second, n[1]);
      }
      v[p][0] = n[0];
      v[p][1] = n[1];
    };
    // planes 1 .. np - 1 first: they need registers and the upper copy; then
    // plane 0 with the lower copy
    Quad prev[2] = {v[0][0], v[0][1]}, next0[2] = {H[0], H[1]};
    if (P > 1 && np > 1) {
      next0[0] = v[P > 1 ? 1 : 0][0];
      next0[1] = v[P > 1 ? 1 : 0][1];
    }
#pragma unroll
    for (int p = 1; p < P; ++p)
      if (p < np) {
        const Quad t[2] = {v[p][0], v[p][1]};
        Quad q[2] = {H[0], H[1]}, n[2];
        if (p + 1 < P && p + 1 < np) {
          q[0] = v[p + 1 < P ? p + 1 : p][0];
          q[1] = v[p + 1 < P ? p + 1 : p][1];
        }
        update(t, prev, q, A + p * plane, n);
        prev[0] = t[0];
        prev[1] = t[1];
        put(p, n);
      }
    {
      const Quad t[2] = {v[0][0], v[0][1]};
      Quad n[2];
      update(t, L, next0, A, n);
      put(0, n);
    }
    cl.sync();  // step s written everywhere, and nobody reads buffer s & 1 any more
  }

  float* dst = out + (long long)x0 * plane;
#pragma unroll
  for (int p = 0; p < P; ++p)
    if (p < np && act) {
      stq(dst + (long long)p * plane + at, v[p][0]);
      if (two) stq(dst + (long long)p * plane + second, v[p][1]);
    }
}

// The slab in shared memory: a thread updates up to kMaxGroups groups of four z
// cells wherever they lie in its slab, all neighbours from shared memory (the x
// neighbours of the slab's end planes from the adjacent CTAs').  Bound by shared
// memory, 26 B per cell and step on 16 SMs; us per step against passes: 1000x4x4 0.78
// and 2.80, 96x24x24 1.09 and 1.70, 512x16x16 1.67 and 2.12, 2048x8x16 2.72 and 4.18.
__global__ void __launch_bounds__(kSlabThreads, 1)
    heat_slab_k(const float* __restrict__ in, float* __restrict__ out, ResidentArgs a) {
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int c = int(cl.block_rank());
  const int CL = int(cl.num_blocks());
  const int x0 = int((long long)c * a.X / CL), x1 = int((long long)(c + 1) * a.X / CL);
  const int np = x1 - x0;
  const int plane = a.Y * a.Z;
  const int buf = a.P * plane;  // floats per buffer
  const int zq = a.Z / 4;
  const int groups = np * a.Y * zq;
  const int tid = int(threadIdx.x);

  // the slab into buffer 0
  {
    const float4* src = reinterpret_cast<const float4*>(in + (long long)x0 * plane);
    float4* dst = reinterpret_cast<float4*>(sm);
    for (int i = tid; i < np * plane / 4; i += kSlabThreads) dst[i] = src[i];
  }
  // this thread's groups: offset in a buffer, offset within the plane and
  // which neighbours are walls
  int off[kMaxGroups], inpl[kMaxGroups], flags[kMaxGroups];
#pragma unroll
  for (int k = 0; k < kMaxGroups; ++k) {
    const int g = tid + k * kSlabThreads;
    off[k] = -1;
    inpl[k] = 0;
    flags[k] = 0;
    if (g < groups) {
      const int p = g / (a.Y * zq);
      const int r = g - p * (a.Y * zq);
      const int y = r / zq;
      const int z = 4 * (r - y * zq);
      inpl[k] = y * a.Z + z;
      off[k] = p * plane + inpl[k];
      flags[k] = (p == 0 ? 1 : 0) | (p == np - 1 ? 2 : 0) | (y == 0 ? 4 : 0) | (y == a.Y - 1 ? 8 : 0) |
                 (z == 0 ? 16 : 0) | (z + 4 == a.Z ? 32 : 0);
    }
  }
  // neighbour slabs' shared memory (the plane next to ours in each)
  const float* lo = c > 0 ? cl.map_shared_rank(sm, c - 1) : sm;
  const float* hi = c < CL - 1 ? cl.map_shared_rank(sm, c + 1) : sm;
  const int lo_plane = c > 0 ? (x0 - 1) - int((long long)(c - 1) * a.X / CL) : 0;
  cl.sync();

  for (int s = 0; s < a.steps; ++s) {
    const float* A = sm + (s & 1) * buf;
    float* B = sm + ((s + 1) & 1) * buf;
    const float* Alo = lo + (s & 1) * buf + lo_plane * plane;  // x0 - 1 in the lower slab
    const float* Ahi = hi + (s & 1) * buf;                      // x1 in the upper slab
#pragma unroll
    for (int k = 0; k < kMaxGroups; ++k) {
      if (off[k] < 0) continue;
      const int o = off[k], f = flags[k], yz = inpl[k];
      const float4 C = *reinterpret_cast<const float4*>(A + o);
      float4 XM, XP;
      if (!(f & 1)) XM = *reinterpret_cast<const float4*>(A + o - plane);
      else if (c > 0) XM = *reinterpret_cast<const float4*>(Alo + yz);
      else XM = C;
      if (!(f & 2)) XP = *reinterpret_cast<const float4*>(A + o + plane);
      else if (c < CL - 1) XP = *reinterpret_cast<const float4*>(Ahi + yz);
      else XP = C;
      const float4 YM = (f & 4) ? C : *reinterpret_cast<const float4*>(A + o - a.Z);
      const float4 YP = (f & 8) ? C : *reinterpret_cast<const float4*>(A + o + a.Z);
      const float zl = (f & 16) ? C.x : A[o - 1];
      const float zr = (f & 32) ? C.w : A[o + 4];
      float4 R;
      R.x = heat_update(C.x, XM.x, XP.x, YM.x, YP.x, zl, C.y, a.cx, a.cy, a.cz);
      R.y = heat_update(C.y, XM.y, XP.y, YM.y, YP.y, C.x, C.z, a.cx, a.cy, a.cz);
      R.z = heat_update(C.z, XM.z, XP.z, YM.z, YP.z, C.y, C.w, a.cx, a.cy, a.cz);
      R.w = heat_update(C.w, XM.w, XP.w, YM.w, YP.w, C.z, zr, a.cx, a.cy, a.cz);
      *reinterpret_cast<float4*>(B + o) = R;
    }
    cl.sync();  // step s written everywhere, and nobody reads buffer s & 1 any more
  }

  // the final state to global memory
  {
    const float4* src = reinterpret_cast<const float4*>(sm + (a.steps & 1) * buf);
    float4* dst = reinterpret_cast<float4*>(out + (long long)x0 * plane);
    for (int i = tid; i < np * plane / 4; i += kSlabThreads) dst[i] = src[i];
  }
}

using Kernel = void (*)(const float*, float*, ResidentArgs);

int run_cluster(cfdb_ctx* ctx, Kernel kern, const void* Ta, void* out, const ResidentArgs& a, int CL, int threads,
                long long smem) {
  // per-device kernel attributes; cheap enough to set on every call
  CFDB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CFDB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(CL));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = size_t(smem);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(CL);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return CFDB_EUNSUPPORTED;
  }
  CFDB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, static_cast<const float*>(Ta), static_cast<float*>(out), a));
  ++ctx->launches;
  return CFDB_OK;
}

// Whether a slab of P planes in shared memory beats the passes.  A step costs 1075 SM
// cycles (cluster barrier), 112 for every 1024 cells of a plane that the neighbours
// read remotely, and per 1024 groups of the CTA 731 and, begun ones, 331; the launch and
// the field's way in and out 4500 more than passes' (12000 more than the single pass of
// three steps).  Fitted to 48 long shapes at 200 steps (within 8 %); the choice is the
// faster form or within 3 % of it but for 65x16x128 (8 %).  Slabs of few wide planes
// (their x neighbours all remote) lose at any size: 12x100x60 2.5 us against 1.7.
bool slab_wins(cfdb_ctx* ctx, cfdb_mesh* m, long long P, int32_t steps) {
  if (P <= kMaxPlanes) return false;
  const double plane = double(m->ny * m->nz), groups = double(P) * plane / (4.0 * kSlabThreads);
  const double step = 1075.0 + 112.0 * plane / 1024.0 + 731.0 * groups + 331.0 * std::ceil(groups);
  if (steps <= 2) return steps == 2 && step < 3300.0;  // against single steps: the second launch costs about 2 us
  return double(steps) * (1.03 * heat_pass_cycles(ctx, m) - step) > (steps == 3 ? 12000.0 : 4500.0);
}

}  // namespace

// Runs `steps` heat steps in one launch when the mesh fits one cluster and that is
// the faster form.  In registers: planes of at most 512 (row pair, four cells)
// threads, 4 planes per CTA, two buffers in shared memory.  Beyond that in shared
// memory alone (slab_wins).  CFDB_EUNSUPPORTED (nothing launched, no error recorded)
// otherwise, and the caller takes another path.  The result goes to Tb for odd
// `steps`, else to Ta, as with the ping-pong of the per-step path; the other buffer
// is left as it was.
int heat_resident_run(cfdb_ctx* ctx, cfdb_mesh* m, const void* Ta, void* Tb, double k, double dt, int32_t steps,
                      int* launched) {
  *launched = 0;
  if (!m->uniform || m->nz % 4 != 0 || steps < 1) return CFDB_EUNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(Ta) | reinterpret_cast<uintptr_t>(Tb)) & 15u) return CFDB_EUNSUPPORTED;
  const long long plane = m->ny * m->nz, pairs = (m->ny + 1) / 2 * (m->nz / 4);
  int max_smem = 0;
  CFDB_CUDA(ctx, cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  ResidentArgs a;
  a.X = int(m->nx); a.Y = int(m->ny); a.Z = int(m->nz);
  a.steps = steps;
  a.cx = float(dt * k / (m->dx * m->dx));
  a.cy = float(dt * k / (m->dy * m->dy));
  a.cz = float(dt * k / (m->dz * m->dz));
  void* out = (steps & 1) ? Tb : const_cast<void*>(Ta);
  for (int CL = int(std::min<long long>(kMaxCluster, m->nx)); CL >= 2; CL /= 2) {
    const long long P = (m->nx + CL - 1) / CL;
    const long long smem = 2 * P * plane * 4;
    if (smem > max_smem) break;  // fewer CTAs only make the slabs larger
    a.P = int(P);
    int rc = CFDB_EUNSUPPORTED;
    if (P <= kMaxPlanes && pairs <= kThreads) {
      rc = run_cluster(ctx, P <= 2 ? heat_resident_k<2> : heat_resident_k<4>, Ta, out, a, CL, int((pairs + 31) / 32 * 32), smem);
    } else if (P * plane / 4 <= (long long)kMaxGroups * kSlabThreads) {
      if (!slab_wins(ctx, m, P, steps)) break;
      rc = run_cluster(ctx, heat_slab_k, Ta, out, a, CL, kSlabThreads, smem);
    }
    if (rc == CFDB_OK) *launched = CL;
    if (rc != CFDB_EUNSUPPORTED) return rc;
  }
  return CFDB_EUNSUPPORTED;
}
