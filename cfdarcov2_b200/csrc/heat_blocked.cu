// Several heat steps per pass over the field (FP32, uniform meshes): a CTA
// marches an extended (z, y) tile along x once and carries K time levels
// behind one another, so a pass reads and writes the field once for K steps.
//
// A step of the one-step sweep is bound by HBM beyond L2 (8 B per cell and
// step) and by launch and pipeline fill below it; what remains here is
// instruction issue (about 11 per cell and step) and the tile's halo.  Level s
// runs one plane behind level s - 1: at iteration i level 0 receives plane i and
// level s computes plane i - s.  Per level a thread keeps the current plane's
// value of its cells and the difference towards the plane below in registers;
// the plane above is what level s - 1 has just computed.  Neighbours in z are the
// adjacent lanes, neighbours in y come from shared memory, where every level's
// plane is published for the next iteration (two buffers per level, level 0
// in the ring slots its TMA copies land in): one barrier per iteration serves all
// levels.  A thread owns four z cells of R = 2 rows, which share the face between
// them.  The tile is extended by K rows and four z cells towards every side that
// is not a wall; what the outer cells compute from neighbours that are not there
// spreads one cell per level and never reaches the cells that are stored.  Along x
// a chunk starts K planes early and ends K planes late in the same way.
//
// Each cell update is heat_update() (heat_cell.cuh) operation by operation
// (packed pairs round per lane like the scalar operations; a difference that two
// cells share is formed once and enters the other with the opposite sign, which is exact), so results are those
// of the one-step sweep bit for bit.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "f32x2.cuh"
#include "tma_host.hpp"

CFDB_MODULE_ANCHOR

namespace {

using namespace stencil;

constexpr int kRows = 2;   // rows per thread
constexpr int kHaloZ = 4;  // z cells beyond an inner tile edge (a 16-byte step; K <= 4: three steps at most)

struct BlockedArgs {
  int X, Y, Z;
  int ztiles, chunks;
  float cx, cy, cz;
  float* out;
  long long wait_cycles;
  int missing_plane;  // test hook as in the sweeps: CTA (0, 0) issues no copy for its plane of this index
  int* err;
};

// Tiles of an axis of n cells with `ext` extended cells and a halo h: the first
// and last tile need no halo on the wall side.
__host__ __device__ inline int tiles_of(int n, int ext, int h) {
  return n <= ext ? 1 : 2 + (std::max(0, n - 2 * (ext - h)) + (ext - 2 * h) - 1) / (ext - 2 * h);
}
struct Tile {
  int start, lo, hi;  // first extended cell, stored cells [lo, hi)
};
__host__ __device__ inline Tile tile_of(int t, int n, int ext, int h) {
  Tile r;
  r.lo = t == 0 ? 0 : (ext - h) + (t - 1) * (ext - 2 * h);
  r.start = t == 0 ? 0 : r.lo - h;
  r.hi = r.start + ext >= n ? n : r.start + ext - h;
  return r;
}

template <int K, int ZL, int WARPS> struct Shape {
  static constexpr int ROWS = WARPS * (32 / ZL) * kRows;
  static constexpr int EZ = 4 * ZL;
  static constexpr int TILE = ROWS * EZ;           // floats of one plane (a multiple of 32)
  static constexpr int S = 4;                      // ring slots of level 0
  static constexpr size_t SMEM = size_t(S + 2 * (K - 1)) * TILE * 4;
  static constexpr uint32_t BYTES = TILE * 4;
  static constexpr int THREADS = WARPS * 32;
};

struct Cells {
  float2 a, b;  // cells 0, 1 and 2, 3
};
__device__ __forceinline__ Cells ld(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void st(float* p, const Cells& c) {
  *reinterpret_cast<float4*>(p) = make_float4(c.a.x, c.a.y, c.b.x, c.b.y);
}
__device__ __forceinline__ Cells operator-(const Cells& x, const Cells& y) { return {f2::sub(x.a, y.a), f2::sub(x.b, y.b)}; }
__device__ __forceinline__ Cells operator+(const Cells& x, const Cells& y) { return {f2::add(x.a, y.a), f2::add(x.b, y.b)}; }
__device__ __forceinline__ Cells operator-(const Cells& x) { return {f2::neg(x.a), f2::neg(x.b)}; }

template <int K, int ZL, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 512 / (WARPS * 32))
    heat_blocked_k(const __grid_constant__ CUtensorMap tm, const __grid_constant__ BlockedArgs g) {
  using L = Shape<K, ZL, WARPS>;
  extern __shared__ __align__(128) float smem[];
  __shared__ __align__(8) uint64_t bars[L::S];
  const Tile tz = tile_of(int(blockIdx.x) % g.ztiles, g.Z, L::EZ, kHaloZ);
  const Tile ty = tile_of(int(blockIdx.x) / g.ztiles, g.Y, L::ROWS, K);
  const int x0 = int((long long)blockIdx.y * g.X / g.chunks), x1 = int((long long)(blockIdx.y + 1) * g.X / g.chunks);
  const int ib = max(x0 - K, 0);                 // first plane of level 0
  const int last = min(x1 - 1 + K, g.X - 1);     // last plane of level 0
  if (threadIdx.x == 0) {
    prefetch_tmap(&tm);
    for (int s = 0; s < L::S; ++s) mbar_init(&bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_dep_wait();
  grid_dep_launch();
  if (smem_u32(smem) & 127u) {
    if (threadIdx.x == 0) atomicExch(g.err, kErrSmemAlign);
    return;
  }
  {
    uint32_t dyn;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if (dyn < L::SMEM) {
      if (threadIdx.x == 0) atomicExch(g.err, kErrSmemSize);
      return;
    }
  }
  // A wait that gives up ends the staging as in the sweeps: nothing more is
  // issued, later waits are skipped, and the copies in flight are waited for
  // (bounded) before the CTA exits.
  bool bad = false;
  int issued = ib - 1, waited = ib - 1;  // last plane issued (thread 0), last plane waited for
  auto issue = [&](int x) {
    if (bad || x > last) return;
    uint64_t* bar = &bars[(x - ib) % L::S];
    mbar_expect_tx(bar, L::BYTES);
    issued = x;
    if (x - ib == g.missing_plane && blockIdx.x == 0 && blockIdx.y == 0) return;
    tma_load_3d(smem + ((x - ib) % L::S) * L::TILE, &tm, tz.start, ty.start, x, bar);
  };
  if (threadIdx.x == 0)
    for (int j = 0; j < L::S; ++j) issue(ib + j);
  auto wait_plane = [&](int x) {
    waited = x;
    if (!bad && !mbar_wait_bounded(&bars[(x - ib) % L::S], unsigned((x - ib) / L::S) & 1u, g.wait_cycles)) bad = true;
  };

  const int lane = int(threadIdx.x) & 31;
  const int zl = lane % ZL, row = ((int(threadIdx.x) >> 5) * (32 / ZL) + lane / ZL) * kRows;
  const int z = tz.start + 4 * zl, y = ty.start + row;
  const bool zlo = z == 0, zhi = z + 4 == g.Z;
  const int at = row * L::EZ + 4 * zl;  // the thread's cells in a tile
  // rows beside the thread's (a wall row sees itself; the tile's own edges read
  // any row, their results are not stored)
  const int below = y == 0 || row == 0 ? at : at - L::EZ;
  const int above = y + 1 >= g.Y - 1 || row + kRows >= L::ROWS ? at + L::EZ : at + 2 * L::EZ;
  const bool wall0 = y == g.Y - 1;  // the thread's first row is the last of the mesh
  const float2 cx = f2::splat(g.cx), cy = f2::splat(g.cy), cz = f2::splat(g.cz);
  const bool zok = z >= tz.lo && z < tz.hi;
  bool store[kRows];
  float* out[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    store[r] = zok && y + r >= ty.lo && y + r < ty.hi;
    out[r] = g.out + (long long)(y + r) * g.Z + z;
  }
  const long long plane = (long long)g.Y * g.Z;
  float* const levels = smem + L::S * L::TILE;

  // level s: values of its centre plane, and the centre minus the plane below
  Cells c[K][kRows], e[K][kRows];
#pragma unroll
  for (int s = 0; s < K; ++s)
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      c[s][r] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      e[s][r] = c[s][r];
    }

  // Iteration i.  STEADY: every level has a centre plane, none of them on an x
  // wall, and plane i exists, so nothing but the updates is left; ODD is then the
  // parity of i (the level buffers alternate with it), known at compile time.
  auto iteration = [&](int i, auto steady_, auto odd_) {
    constexpr bool STEADY = decltype(steady_)::value;
    const int odd = STEADY ? int(decltype(odd_)::value) : i & 1;
    Cells up[kRows];  // the plane above the centre plane of the level at hand
    if (STEADY || i <= last) {
      wait_plane(i);
      const float* src = smem + ((i - ib) % L::S) * L::TILE + at;
#pragma unroll
      for (int r = 0; r < kRows; ++r) up[r] = ld(src + r * L::EZ);
    } else {
#pragma unroll
      for (int r = 0; r < kRows; ++r) up[r] = c[0][r];
    }
#pragma unroll
    for (int s = 0; s < K; ++s) {
      const int x = i - 1 - s;  // level s + 1 computes plane x
      if constexpr (!STEADY) {
        if (x == ib - 1) {      // level s receives its first plane
#pragma unroll
          for (int r = 0; r < kRows; ++r) c[s][r] = up[r];
        }
        if (x < ib || x >= g.X) continue;  // not begun, or ended (uniform over the CTA)
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          if (x == g.X - 1) up[r] = c[s][r];
          if (x == 0) e[s][r] = c[s][r] - c[s][r];  // the wall neighbour is the cell itself (NaN for an infinity)
        }
      }
      const float* lev =
          s == 0 ? smem + ((i - 1 - ib) % L::S) * L::TILE : levels + ((s - 1) * 2 + ((odd + 1 + s) & 1)) * L::TILE;
      const Cells yb = ld(lev + below), ya = ld(lev + above);
      // y: (above - t) + (below - t); the difference between the rows serves both
      Cells dy01 = c[s][1] - c[s][0];
      if (wall0) dy01 = c[s][0] - c[s][0];
      const Cells ly[kRows] = {dy01 + (yb - c[s][0]), (ya - c[s][1]) - dy01};
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const Cells t = c[s][r];
        float l = __shfl_up_sync(0xffffffffu, t.b.y, 1, ZL), h = __shfl_down_sync(0xffffffffu, t.a.x, 1, ZL);
        l = zlo ? t.a.x : l;
        h = zhi ? t.b.y : h;
        const float d0 = __fsub_rn(t.a.y, t.a.x), d1 = __fsub_rn(t.b.x, t.a.y), d2 = __fsub_rn(t.b.y, t.b.x);
        const Cells lz = {make_float2(__fadd_rn(d0, __fsub_rn(l, t.a.x)), __fsub_rn(d1, d0)),
                          make_float2(__fsub_rn(d2, d1), __fsub_rn(__fsub_rn(h, t.b.y), d2))};
        const Cells d = up[r] - t;
        const Cells lx = d - e[s][r];
        Cells n;
        n.a = f2::add(t.a, f2::fma(cx, lx.a, f2::fma(cy, ly[r].a, f2::mul(cz, lz.a))));
        n.b = f2::add(t.b, f2::fma(cx, lx.b, f2::fma(cy, ly[r].b, f2::mul(cz, lz.b))));
        e[s][r] = d;
        c[s][r] = up[r];
        up[r] = n;
      }
      if (s + 1 < K) {
        float* dst = levels + (s * 2 + ((odd + 1 + s) & 1)) * L::TILE + at;
#pragma unroll
        for (int r = 0; r < kRows; ++r) st(dst + r * L::EZ, up[r]);
      } else if (x >= x0) {
#pragma unroll
        for (int r = 0; r < kRows; ++r)
          if (store[r]) st(out[r] + x * plane, up[r]);
      }
    }
    __syncthreads();
    // plane i - 1 of level 0 has been read by every thread
    if (threadIdx.x == 0 && i > ib) {
      fence_proxy_async();
      issue(i - 1 + L::S);
    }
  };
  using Yes = std::true_type;
  using No = std::false_type;
  int i = ib;
  const int steady = (max(ib + K, K + 1) + 1) & ~1, end = x1 + K;
  for (; i < end && i < steady; ++i) iteration(i, No{}, No{});
#pragma unroll 1
  for (; i + 1 <= last; i += 2) {
    iteration(i, Yes{}, No{});
    iteration(i + 1, Yes{}, Yes{});
  }
#pragma unroll 1
  for (; i < end; ++i) iteration(i, No{}, No{});
  if (bad) {
    if (threadIdx.x == 0)
      for (int x = waited + 1; x <= issued; ++x)
        mbar_wait_bounded(&bars[(x - ib) % L::S], unsigned((x - ib) / L::S) & 1u, g.wait_cycles);
    atomicExch(g.err, kErrWaitTimeout);
  }
}

// A pass: K steps, tiles of ZL lanes along z and `warps` warps, x chunks.
struct Plan {
  int K = 0, ZL = 0, warps = 0, chunks = 1;
  double cost = 0;  // estimated SM cycles per step
};

template <int K, int ZL, int WARPS> int launch(cfdb_ctx* ctx, const cfdb_mesh* m, const void* src, void* dst, BlockedArgs a) {
  using L = Shape<K, ZL, WARPS>;
  auto fn = encode_fn();
  if (!fn) return cfdb_fail(ctx, CFDB_ECUDA, "cuTensorMapEncodeTiled entry point unavailable");
  CUtensorMap tm;
  cuuint64_t dims[3] = {cuuint64_t(m->nz), cuuint64_t(m->ny), cuuint64_t(m->nx)};
  cuuint64_t strides[2] = {cuuint64_t(m->nz) * 4, cuuint64_t(m->nz * m->ny) * 4};
  cuuint32_t box[3] = {cuuint32_t(L::EZ), cuuint32_t(L::ROWS), 1};
  cuuint32_t es[3] = {1, 1, 1};
  const CUresult r = fn(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(src), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cfdb_fail(ctx, CFDB_ECUDA, "cuTensorMapEncodeTiled (heat) failed with %d", int(r));
  auto kern = heat_blocked_k<K, ZL, WARPS>;
  // a setting of the CUDA context; cheap enough for every pass
  CFDB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::SMEM)));
  a.ztiles = tiles_of(a.Z, L::EZ, kHaloZ);
  a.out = static_cast<float*>(dst);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.ztiles * tiles_of(a.Y, L::ROWS, K), a.chunks);
  cfg.blockDim = dim3(L::THREADS);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CFDB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, tm, a));
  ++ctx->launches;
  return CFDB_OK;
}

template <int K, int ZL> int launch_warps(cfdb_ctx* ctx, const cfdb_mesh* m, const Plan& p, const void* s, void* d, const BlockedArgs& a) {
  if (p.warps == 16) return launch<K, ZL, 16>(ctx, m, s, d, a);
  if (p.warps == 8) return launch<K, ZL, 8>(ctx, m, s, d, a);
  return launch<K, ZL, 4>(ctx, m, s, d, a);
}
template <int K> int launch_zl(cfdb_ctx* ctx, const cfdb_mesh* m, const Plan& p, const void* s, void* d, const BlockedArgs& a) {
  if (p.ZL == 32) return launch_warps<K, 32>(ctx, m, p, s, d, a);
  if (p.ZL == 16) return launch_warps<K, 16>(ctx, m, p, s, d, a);
  return launch_warps<K, 8>(ctx, m, p, s, d, a);
}

// The cheapest plan for passes of K steps.  A CTA marches its chunk and K planes
// on each side; an iteration takes about 450 cycles of latency (copy, barrier)
// plus, per level, a dependent chain of 130 and 21 for every warp of the SM,
// 1500 to fill a wave of CTAs and 3500 around a launch.  Fitted to 384x400x392,
// where it is right (43.8 us per step by the rule, 44 measured); passes that
// follow one another hide most of the last two terms, so small fields take less
// than it says (64^3 3.1 by the rule and 2.2 measured, 128^3 5.1 and 3.8, 160^3 6.8
// and 5.1).  The search weighs the tiles' halo and padding, how evenly the CTAs
// fill the SMs, and the chunks' overlap.  Of the chunk counts with equally long
// chunks the smallest costs least (no other term falls as they grow), so only
// those are looked at: 2 sqrt(nx) of them.
Plan plan_search(const cfdb_ctx* ctx, const cfdb_mesh* m, int K) {
  Plan best;
  const int64_t sms = std::max(1, ctx->num_sms);
  for (int ZL : {32, 16, 8})
    for (int warps : {16, 8, 4}) {
      const int rows = warps * (32 / ZL) * kRows;
      if (rows <= 2 * K && rows < m->ny) continue;  // the halo would leave no rows
      const int64_t tiles = int64_t(tiles_of(int(m->nz), 4 * ZL, kHaloZ)) * tiles_of(int(m->ny), rows, K);
      const int64_t slots = sms * (16 / warps);
      const int64_t most = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(m->nx / 2, 4096), 16 * slots / tiles));
      for (int64_t chunks = 1; chunks <= most;) {
        const int64_t waves = (tiles * chunks + slots - 1) / slots;
        const int64_t longest = (m->nx + chunks - 1) / chunks;
        const double planes = double(longest) + (chunks > 2 ? 2 * K : chunks > 1 ? K : 0) + K;
        const int64_t per_sm = (std::min(slots, tiles * chunks) + sms - 1) / sms;
        const double cycles = 3500.0 + double(waves) * (1500.0 + planes * (450.0 + K * (130.0 + 21.0 * double(warps * per_sm))));
        if (best.K == 0 || cycles / K < best.cost) best = Plan{K, ZL, warps, int(chunks), cycles / K};
        if (longest == 1) break;
        chunks = (m->nx + longest - 2) / (longest - 1);
      }
    }
  return best;
}

// The same, kept on the mesh (the search takes 2 to 10 us of host time, as much as a
// short call): one word, so that threads that come together store the same.
Plan plan_for(const cfdb_ctx* ctx, cfdb_mesh* m, int K) {
  std::atomic<uint64_t>& word = m->heat_plan[K - 2];
  uint64_t w = word.load(std::memory_order_relaxed);
  if (w == 0) {
    const Plan p = plan_search(ctx, m, K);
    const float cost = float(p.cost);
    uint32_t bits;
    std::memcpy(&bits, &cost, sizeof(bits));
    w = uint64_t(bits) << 32 | uint64_t(p.chunks) << 16 | uint64_t(p.ZL) << 8 | uint64_t(p.warps);
    word.store(w, std::memory_order_relaxed);
  }
  const uint32_t bits = uint32_t(w >> 32);
  float cost;
  std::memcpy(&cost, &bits, sizeof(cost));
  return Plan{K, int(w >> 8 & 255), int(w & 255), int(w >> 16 & 65535), double(cost)};
}

}  // namespace

// SM cycles per step of passes in a row over a field that a cluster would hold: the
// rule's, less what the passes hide of one another (fitted to 48 thin fields at 1.7 to
// 5.5 us per step: within 19 %, most within 5).
double heat_pass_cycles(const cfdb_ctx* ctx, cfdb_mesh* m) {
  return 1.234 * std::min(plan_for(ctx, m, 2).cost, plan_for(ctx, m, 3).cost) - 3655.0;
}

// `steps` steps (1 .. 3) in one pass src -> dst.
static int blocked_pass(cfdb_ctx* ctx, cfdb_mesh* m, const void* src, void* dst, double k, double dt, int steps,
                        const Plan plans[4]) {
  if (steps == 1) return fused_heat_step(ctx, m, CFDB_F32, src, dst, k, dt);
  const Plan& p = plans[steps];
  BlockedArgs a{};
  a.X = int(m->nx); a.Y = int(m->ny); a.Z = int(m->nz);
  a.chunks = p.chunks;
  a.cx = float(dt * k / (m->dx * m->dx));
  a.cy = float(dt * k / (m->dy * m->dy));
  a.cz = float(dt * k / (m->dz * m->dz));
  a.wait_cycles = ctx->wait_cycles;
  a.missing_plane = ctx->missing_plane;
  a.err = ctx->d_error;
  return steps == 2 ? launch_zl<2>(ctx, m, p, src, dst, a) : launch_zl<3>(ctx, m, p, src, dst, a);
}

// `steps` steps, the state alternating between Ta and Tb per pass, the last one
// where the one-step sweep would have left it (Tb for odd `steps`); with
// keep_other the buffer that does not receive the result is left as it was,
// a workspace taking its part where one can be had.  CFDB_EUNSUPPORTED (nothing
// launched) when the mesh or the pointers are not what the TMA kernels take, and for
// one or two steps that need no workspace.
int heat_blocked_run(cfdb_ctx* ctx, cfdb_mesh* m, void* Ta, void* Tb, double k, double dt, int32_t steps, int use_graph,
                     bool keep_other) {
  if (steps < 1 || check_sweep(ctx, m, {Ta, Tb}) != CFDB_OK) return CFDB_EUNSUPPORTED;
  // passes of two or three steps (four spill registers), as even as possible,
  // as many as the parity wants; one or two steps are single passes
  Plan plans[4];
  int most = 1;
  if (steps > 2) {
    for (int K : {2, 3}) plans[K] = plan_for(ctx, m, K);
    most = plans[3].cost < plans[2].cost ? 3 : 2;
  }
  int32_t n = steps / most + (steps % most != 0);
  if ((n ^ steps) & 1) ++n;
  const int per = int(steps / n), more = int(steps % n);  // the first `more` passes do per + 1
  void* ws = nullptr;
  if (keep_other && n > 1) {
    const int rc = cfdb_ws_alloc(ctx, m->n * 4, &ws);
    if (rc && rc != CFDB_ENOMEM) return rc;
    keep_other = rc == CFDB_OK;
  }
  if (!keep_other && steps <= 2) return CFDB_EUNSUPPORTED;  // the caller's single steps
  if (!keep_other) {
    auto run = [&](void* a, void* b, int32_t passes, int each) {
      return cfdb_run_steps(
          ctx, a, b, passes, use_graph, [&](const void* s, void* d) { return blocked_pass(ctx, m, s, d, k, dt, each, plans); },
          graph_key("heat-pass", m, CFDB_F32, CFDB_PATH_FUSED, a, b, nullptr, {k, dt, double(each)}));
    };
    if (more)
      if (int rc = run(Ta, Tb, more, per + 1)) return rc;
    return (more & 1) ? run(Tb, Ta, n - more, per) : run(Ta, Tb, n - more, per);
  }
  void* const result = (steps & 1) ? Tb : Ta;
  const void* src = Ta;
  int rc = CFDB_OK;
  for (int32_t j = 0; j < n && !rc; ++j) {
    void* dst = ((n - 1 - j) & 1) ? ws : result;
    rc = blocked_pass(ctx, m, src, dst, k, dt, j < more ? per + 1 : per, plans);
    src = dst;
  }
  cfdb_ws_free(ctx, ws);
  return rc;
}
