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
// results are those of the one-step sweep bit for bit.  Larger fields take several
// steps per pass over all SMs (heat_blocked.cu).
#include <cooperative_groups.h>

#include <algorithm>

#include "cfdb_internal.hpp"
#include "f32x2.cuh"

CFDB_MODULE_ANCHOR

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;    // at most: row pairs x z groups
constexpr int kMaxCluster = 16;  // non-portable cluster size
constexpr int kMaxPlanes = 4;    // planes per slab (eight spill registers)

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

template <int P>
int run_cluster(cfdb_ctx* ctx, const cfdb_mesh* m, const void* Ta, void* out, const ResidentArgs& a, int CL, long long smem) {
  auto kern = heat_resident_k<P>;
  // per-device kernel attributes; cheap enough to set on every call
  CFDB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CFDB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(CL));
  cfg.blockDim = dim3(unsigned(((m->ny + 1) / 2 * (m->nz / 4) + 31) / 32 * 32));
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

}  // namespace

// Runs `steps` heat steps in one launch when the mesh fits one cluster: planes
// of at most 512 (row pair, four cells) threads, 4 planes per CTA, two buffers in
// shared memory.  CFDB_EUNSUPPORTED (nothing launched, no error recorded)
// otherwise, and the caller takes another path.  The result goes to Tb for odd
// `steps`, else to Ta, as with the ping-pong of the per-step path; the other buffer
// is left as it was.
int heat_resident_run(cfdb_ctx* ctx, cfdb_mesh* m, const void* Ta, void* Tb, double k, double dt, int32_t steps,
                      int* launched) {
  *launched = 0;
  if (!m->uniform || m->nz % 4 != 0 || steps < 1) return CFDB_EUNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(Ta) | reinterpret_cast<uintptr_t>(Tb)) & 15u) return CFDB_EUNSUPPORTED;
  if ((m->ny + 1) / 2 * (m->nz / 4) > kThreads) return CFDB_EUNSUPPORTED;
  int max_smem = 0;
  CFDB_CUDA(ctx, cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const long long plane = m->ny * m->nz;
  ResidentArgs a;
  a.X = int(m->nx); a.Y = int(m->ny); a.Z = int(m->nz);
  a.steps = steps;
  a.cx = float(dt * k / (m->dx * m->dx));
  a.cy = float(dt * k / (m->dy * m->dy));
  a.cz = float(dt * k / (m->dz * m->dz));
  void* out = (steps & 1) ? Tb : const_cast<void*>(Ta);
  for (int CL = std::min<long long>(kMaxCluster, m->nx); CL >= 2; CL /= 2) {
    const long long P = (m->nx + CL - 1) / CL;
    const long long smem = 2 * P * plane * 4;
    if (smem > max_smem || P > kMaxPlanes) break;  // fewer CTAs only make the slabs larger
    a.P = int(P);
    const int rc = P <= 2 ? run_cluster<2>(ctx, m, Ta, out, a, CL, smem) : run_cluster<4>(ctx, m, Ta, out, a, CL, smem);
    if (rc == CFDB_OK) *launched = CL;
    if (rc != CFDB_EUNSUPPORTED) return rc;
  }
  return CFDB_EUNSUPPORTED;
}
