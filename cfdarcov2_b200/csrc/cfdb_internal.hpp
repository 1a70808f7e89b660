// Internal declarations shared by the host runtime and the kernel files of
// libcfdb.  Nothing here is part of the C ABI (include/cfdb.h).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <functional>
#include <initializer_list>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "cfdb.h"

// ---------------------------------------------------------------------------
// Host-side geometry in double: the reference's flattened N x 6 arrays
// (entry (i, f) at f*n + i; per-dimension arrays stacked d*6n + f*n + i).
// ---------------------------------------------------------------------------
struct HostGeom {
  int64_t nx = 0, ny = 0, nz = 0, n = 0;
  std::vector<double> normal, normal_alt;  // 3 * 6n
  std::vector<double> area, alpha, len;    // 6n
  std::vector<double> volume, center, isb; // n, 3n, n
  std::vector<int64_t> ids, ibf;           // 6n
};

// Builds HostGeom (geometry.cpp).  verts may be null (uniform lattice).  mode:
// 0 reference formulas, 1 reference with component-sum areas, 2 exact vector
// areas (default of vertex meshes).  Returns false if memory runs out.
bool cfdb_build_geometry(HostGeom& g, int64_t nx, int64_t ny, int64_t nz, double dx, double dy, double dz,
                         const double* verts, int mode);

// Device copy of the geometry for the plain (per-operator) kernels in one
// precision.  ids are int32 (self on boundary faces, as the reference's _ids).
struct PlainGeomDev {
  bool ready = false;
  void* normal = nullptr;      // 3 * 6n
  void* normal_alt = nullptr;  // 3 * 6n
  void* area = nullptr;        // 6n
  void* alpha = nullptr;       // 6n
  void* len = nullptr;         // 6n
  void* volume = nullptr;      // n
  void* isb = nullptr;         // n
  void* stab_tmp = nullptr;    // 3 * 6n, allocated on first stab call
};

// Geometry of a structured mesh along one axis, in double: edge lengths (n),
// face-plane coordinates (n + 1), alpha of the face below cell i (n + 1) and
// |x_f - x_P| of a cell's lower and upper face (n each).
struct AxisTables {
  std::vector<double> h, g, alpha, len_lo, len_hi;
};
// Fills t[0..2] (x, y, z) and returns the magnitude up to which an operand
// overflows in no intermediate of the operators; NaN when the face arrays of
// this mesh do not follow exactly from values per axis (geometry.cpp).
double axis_tables(int64_t nx, int64_t ny, int64_t nz, double dx, double dy, double dz, bool f64, AxisTables t[3]);

// The same tables on the device in one precision (box_ops.cu), in place of
// the face arrays: h in double, the rest in the storage type; vol (n) is null
// when every cell's volume rounds to v.
struct BoxGeomDev {
  int state = 0;  // 0 not built, 1 usable, 2 this mesh keeps the face arrays
  void* tab = nullptr;
  void* vol = nullptr;
  const double* h[3] = {};
  const void* alpha[3] = {};
  const void* len[6] = {};  // x-, x+, y-, y+, z-, z+
  double v = 0, limit = 0;
  // every cell's volume, areas, interior alphas and lengths round to one value
  // per direction (uA: the face normal to x, y, z)
  bool uni = false;
  double uA[3] = {}, ual[3] = {}, ulm[3] = {}, ulp[3] = {};
};

// Geometry of a vertex mesh with every face held once (box_ops.cu), in one
// precision: per axis the faces' unit normals along +axis (3 count), areas and
// alphas (count each; the face below cell i along its axis is entry i, one more
// entry than cells), per cell the six |x_f - x_P| (slot after slot) and the volume.
struct FaceGeomDev {
  int state = 0;  // 0 not built, 1 usable, 2 this mesh keeps the N x 6 arrays
  int64_t count[3] = {};
  void* block = nullptr;  // holds all of the following
  void* normal[3] = {};
  void* area[3] = {};
  void* alpha[3] = {};
  void* len = nullptr;
  void* vol = nullptr;
  void* grad = nullptr;  // 3 n, the stabilisation's first stage: there with the
                         // geometry, so that a recorded or budgeted call needs nothing more
};

// Compact FP32 geometry of vertex meshes for the fused kernels: per cell the
// outward area vector of its +x/+y/+z face and 1/V (10 fields), stored on
// the lattice padded by one ghost layer below each axis (x and y) and by four
// cells below z (so the z origin of every row stays 16-byte aligned):
// cell (x, y, z) sits at ((x + 1) Yp + y + 1) Zp + z + 4 with Yp = ny + 1,
// Zp = nz + 4.  The -faces of a cell are its minus neighbours' +faces
// negated; on the -x/-y/-z walls that neighbour is a ghost entry holding the
// wall face's outward area vector negated, so no kernel needs a wall table.
// Ghost entries of the other fields are zero.
struct CompactGeomDev {
  bool ready = false;
  float* S = nullptr;  // 10 np: [Sx.x|Sx.y|Sx.z|Sy.x|...|Sz.z|1/V] over the padded lattice
  int64_t np = 0;      // padded entries per field: (nx + 1) Yp Zp
  int64_t yp = 0, zp = 0;
};

struct cfdb_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  int64_t budget = 0;
  int64_t allocated = 0;
  std::unordered_map<void*, int64_t> allocs;
  // Stream-ordered pool for per-call workspaces (checkpoint slots, adjoint
  // buffers, reduction scratch): freed blocks stay in the pool, so a repeated
  // call of the same size neither allocates nor frees device memory.
  cudaMemPool_t pool = nullptr;
  std::unordered_map<void*, int64_t> ws;
  // Scratch of the synchronous reductions (CFL step, FP64 totals): per-CTA
  // partials, the last-CTA ticket and a page-locked word the kernel stores the
  // result to.  A call holds the mutex until it has read its result, so calls
  // on any stream or thread never share the scratch.
  struct Reduce {
    void* part = nullptr;
    unsigned int* ticket = nullptr;
    void* host = nullptr;
    unsigned long long host_id = 0;  // the CUDA context `host` was locked in
    std::mutex mu;
  } reduce;
  int* d_error = nullptr;  // device error word written by bounded waits
  // Bound of the sweep kernels' mbarrier waits (SM clock cycles) and the
  // missing-copy test hook (cfdb_ctx_set_wait_limit).
  long long wait_cycles = 4000000000LL;
  int missing_plane = -1;
  cudaStream_t capture_stream = nullptr;  // private stream used to record CUDA graphs
  // Kernels launched on this context so far (graph replays count every
  // kernel node they run).
  int64_t launches = 0;
  // Instantiated step graphs of cfdb_run_steps, keyed by everything the
  // recorded launches depend on; least recently used beyond kGraphCache.
  struct GraphEntry {
    std::string key;
    cudaGraphExec_t exec = nullptr;
    int32_t chunk = 0;        // steps per replay
    int64_t per_replay = 0;   // kernels per replay
    uint64_t last_use = 0;
  };
  std::vector<GraphEntry> graphs;
  uint64_t graph_clock = 0;
  // Objects created on this context (meshes, Euler solvers, batches) with a
  // callback that detaches them when the context is destroyed first: their
  // device memory goes with the context, their own destroy then frees only
  // host memory.
  std::unordered_map<void*, std::function<void()>> children;
};

inline void cfdb_adopt(cfdb_ctx* ctx, void* child, std::function<void()> orphan) {
  if (ctx) ctx->children[child] = std::move(orphan);
}
inline void cfdb_release(cfdb_ctx* ctx, void* child) {
  if (ctx) ctx->children.erase(child);
}

// Runs `steps` calls of step(src, dst) alternating a -> b -> a ..., eagerly or
// replayed from a captured CUDA graph (graphs.cpp).  `key` names everything
// the recorded launches depend on (kernel, mesh uid, buffers, parameters); a
// graph recorded under the same key by an earlier call is replayed without
// recording again.  An empty key records a fresh graph every call.
#include <functional>
int cfdb_run_steps(cfdb_ctx* ctx, void* a, void* b, int32_t steps, int use_graph,
                   const std::function<int(const void*, void*)>& step, const std::string& key = std::string());
void cfdb_graphs_clear(cfdb_ctx* ctx);
void cfdb_jit_release(cfdb_ctx* ctx);  // unloads the context's run-time compiled modules (jit.cpp)
// Key of a cached step graph: the step kind, the mesh (by uid), dtype, path,
// the three buffers and the scalar parameters, bit for bit.
std::string graph_key(const char* kind, const struct cfdb_mesh* m, int dtype, int path, const void* a, const void* b,
                      const void* c, std::initializer_list<double> params);

// Marching kernels whose chunk count a mesh keeps (box_ops.cu has 49).
constexpr int kMarches = 64;

struct cfdb_mesh {
  cfdb_ctx* ctx = nullptr;
  uint64_t uid = 0;  // process-unique, never reused (keys of cached step graphs)
  int64_t nx = 0, ny = 0, nz = 0, n = 0;
  double dx = 0, dy = 0, dz = 0;
  bool uniform = true;
  int geom_mode = 0;  // see cfdb_build_geometry
  std::vector<double> verts;  // vertex meshes only
  std::unique_ptr<HostGeom> geom;
  int32_t* d_ids = nullptr;
  PlainGeomDev plain[2];
  CompactGeomDev compact;
  BoxGeomDev box[2];  // structured meshes, by precision
  FaceGeomDev faces[2];  // vertex meshes, by precision
  std::atomic<uint32_t> march_chunks[kMarches] = {};  // by kernel; 0: not chosen
  std::atomic<uint64_t> heat_plan[2] = {};  // passes of 2 and 3 heat steps (heat_blocked.cu); 0: not searched
  int lattice_state = 0;  // 0 not checked, 1 exact lattice, 2 not one
  cfdb_lattice_geometry lattice{};
};

// Device ordinals the per-device caches of kernel attributes cover.
constexpr int kMaxDevices = 64;

// ---- tracing -----------------------------------------------------------------
// An NVTX range over a library call (the reference times Equation::evaluate
// with std::chrono only, examples/main_3d_heat.cpp:96-99): profilers and
// timeline tools show each run / build / gradient phase by name.  NVTX 3 is
// header-only; without a tool attached a range costs a few nanoseconds.
#include <nvtx3/nvToolsExt.h>
struct CfdbRange {
  explicit CfdbRange(const char* name) { nvtxRangePushA(name); }
  ~CfdbRange() { nvtxRangePop(); }
  CfdbRange(const CfdbRange&) = delete;
  CfdbRange& operator=(const CfdbRange&) = delete;
};

// ---- error plumbing --------------------------------------------------------
int cfdb_fail(cfdb_ctx* ctx, int code, const char* fmt, ...);
int cfdb_cuda_fail(cfdb_ctx* ctx, cudaError_t e, const char* what);
// Reads and clears the device error word (bounded waits, sweep launch
// checks); synchronises ctx->stream.  CFDB_ETIMEOUT for a wait that gave up.
int cfdb_check_device_error(cfdb_ctx* ctx);

#define CFDB_CUDA(ctx, call)                                       \
  do {                                                             \
    cudaError_t e__ = (call);                                      \
    if (e__ != cudaSuccess) return cfdb_cuda_fail((ctx), e__, #call); \
  } while (0)

// Checks for a launch error right after a kernel launch.
#define CFDB_LAUNCHED(ctx)                   \
  do {                                       \
    ++(ctx)->launches;                       \
    CFDB_CUDA(ctx, cudaGetLastError());      \
  } while (0)

// ---- memory ---------------------------------------------------------------
int cfdb_dev_alloc(cfdb_ctx* ctx, int64_t bytes, void** out);
void cfdb_dev_free(cfdb_ctx* ctx, void* p);
// Workspace from the context's pool, ordered on ctx->stream (usable by work
// enqueued after the call; freed after the work enqueued before the free).
// Counts toward the allocation budget while live.
int cfdb_ws_alloc(cfdb_ctx* ctx, int64_t bytes, void** out);
void cfdb_ws_free(cfdb_ctx* ctx, void* p);
// CFDB_ENOMEM when a workspace of `bytes` would exceed the allocation budget
// (calls that use scratch the context already owns keep answering as if they
// allocated it).
int cfdb_ws_budget(cfdb_ctx* ctx, int64_t bytes);

// ---- module loading ---------------------------------------------------------
// CUDA loads a kernel at its first launch by default (lazy loading), which
// puts 0.1-1.5 ms of module work inside a caller's first step.  Each
// translation unit with kernels registers an empty anchor kernel at library
// load; context creation loads every kernel of the anchors' modules.
int cfdb_register_module(const void* anchor_kernel);
#define CFDB_MODULE_ANCHOR                                                                      \
  namespace {                                                                                   \
  __global__ void cfdb_module_anchor_k() {}                                                     \
  const int cfdb_module_anchor_reg_ = cfdb_register_module(reinterpret_cast<const void*>(&cfdb_module_anchor_k)); \
  }

// ---- geometry helpers ------------------------------------------------------
int cfdb_mesh_need_host_geom(cfdb_mesh* m);
int cfdb_mesh_need_plain(cfdb_mesh* m, int dtype);
// The geometry a per-operator kernel of dtype runs on, built where it is not yet.
// All give the same bits: the tables of a structured mesh (box_ops.cu), a vertex
// mesh's faces held once (vertex_faces: the operator has such a kernel), or the
// N x 6 arrays.  Where the arrays are there already, they serve while the stream
// records a graph; a failed allocation of the others falls back to them.  Other
// calls on the mesh may want the arrays later, so where the budget or the device has
// room for the arrays (and `array_scratch` bytes that the operator needs with them)
// but not for both, the arrays serve from the start.
enum class Geom { Arrays, Box, Faces };
int cfdb_mesh_geometry(cfdb_mesh* m, int dtype, bool vertex_faces, Geom* geom, int64_t array_scratch = 0);
// fills the plain arrays of dtype on the device (geometry_dev.cu)
int cfdb_build_plain_device(cfdb_mesh* m, int dtype, PlainGeomDev& p);
// Device bytes that the arrays still want (0 when they are there), and those of the
// tables or the faces held once (geometry_dev.cu).
int64_t cfdb_plain_bytes(const cfdb_mesh* m, int dtype);
int64_t cfdb_table_bytes(const cfdb_mesh* m, int dtype);
// samples and checks the lattice constants on the device (geometry_dev.cu)
int cfdb_check_lattice_device(cfdb_mesh* m, cfdb_lattice_geometry* out);
int cfdb_mesh_need_compact(cfdb_mesh* m);

inline size_t dtype_size(int dtype) { return dtype == CFDB_F64 ? 8 : 4; }
inline bool dtype_ok(int dtype) { return dtype == CFDB_F32 || dtype == CFDB_F64; }

int cfdb_check_mesh(cfdb_ctx* ctx, cfdb_mesh* m);
void cfdb_mesh_orphan(cfdb_mesh* m);

// ---- launchers implemented in the kernel files ------------------------------
// plain_ops.cu
int plain_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
int plain_heat_update(cfdb_ctx* ctx, int dtype, const void* L, const void* T, double k, double dt, void* Tn,
                      int64_t n);
int plain_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c,
                    double cconst, int mode, double dt);
int plain_wave_adjoint(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, const void* lam1, void* lam0,
                       const void* c, void* gc, double dt);
// box_ops.cu: the same operators on structured meshes without face arrays.
// *usable = false: this mesh takes the array kernels.
int cfdb_mesh_need_box(cfdb_mesh* m, int dtype, bool* usable);
int box_grad(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
int box_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
int box_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt);
int box_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c, double cconst, int mode,
                  double dt);
int box_stab(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
// The same on vertex meshes with every face's geometry held once.  *usable =
// false: this mesh takes the array kernels.
int cfdb_mesh_need_faces(cfdb_mesh* m, int dtype, bool* usable);
int cfdb_build_faces_device(cfdb_mesh* m, int dtype, FaceGeomDev& b);  // geometry_dev.cu
int vert_grad(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
int vert_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
int vert_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt);
int vert_stab(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask);
// fused_tma.cu
int fused_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt,
                    const void* fixed = nullptr);
int fused_d2t_step(cfdb_ctx* ctx, cfdb_mesh* m, const void* u, const void* u_prev, void* u_next, double k,
                   const int32_t* masks, int32_t n_terms, double dt, int first_step);
// All `steps` FP32 heat steps in one thread-block-cluster launch with the
// field resident in distributed shared memory (resident.cu); CFDB_EUNSUPPORTED
// when the mesh does not fit or passes are faster (nothing launched).
int heat_resident_run(cfdb_ctx* ctx, cfdb_mesh* m, const void* Ta, void* Tb, double k, double dt, int32_t steps,
                      int* launched);
// The same with several steps per pass over the field (heat_blocked.cu).
int heat_blocked_run(cfdb_ctx* ctx, cfdb_mesh* m, void* Ta, void* Tb, double k, double dt, int32_t steps, int use_graph,
                     bool keep_other);
double heat_pass_cycles(const cfdb_ctx* ctx, cfdb_mesh* m);
int fused_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c,
                    double cconst, int mode, double dt);
// distorted.cu
int compact_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c,
                      double cconst, int mode, double dt);
// adjoint.cu
int fused_wave_adjoint(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, const void* lam1, void* lam0,
                       const void* c, void* gc, double dt);

// Shared launch-size helper: a grid-stride grid of at most `per_sm` CTAs per SM.
inline int grid_for(const cfdb_ctx* ctx, int64_t n, int threads, int per_sm = 8) {
  int64_t want = (n + threads - 1) / threads;
  int64_t cap = int64_t(ctx->num_sms > 0 ? ctx->num_sms : 148) * per_sm;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return int(want);
}
