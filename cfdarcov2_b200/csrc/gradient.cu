// Gradient of J = 0.5 |p_T - p_target|^2 with respect to the sound-speed
// field c and the initial pressure p0, through the discrete adjoint of the
// acoustic step (speed_mode 1).  With snapshots >= steps every forward state
// is written straight into its own slot (the forward step's output IS the
// checkpoint: no copies) and the reverse sweep reads them back; with fewer
// slots the binomial schedule of revolve.cpp recomputes the missing states.
#include <algorithm>
#include <cmath>
#include <vector>

#include "cfdb_internal.hpp"

CFDB_MODULE_ANCHOR

int cfdb_revolve_build(int32_t steps, int32_t snapshots, std::vector<int32_t>& act, std::vector<int32_t>& arg,
                       std::vector<int32_t>& at, int64_t* forward);

namespace {

constexpr int kThreads = 256;

// J's partial sum of the CTA, and with `lam` the adjoint seed (p_T - p_target, 0, 0, 0)
// in the same pass; the last CTA to finish folds the partials in a fixed order.
// Bound by memory: 2 fields read, 4 written.
template <class R>
__global__ void __launch_bounds__(kThreads) misfit_k(const R* __restrict__ qT, const R* __restrict__ target, R* __restrict__ lam,
                                                     long long n, double* __restrict__ part, unsigned* __restrict__ ticket,
                                                     double* __restrict__ out) {
  __shared__ double red[kThreads / 32];
  __shared__ bool last;
  double s = 0;
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kThreads) {
    const R q = qT[i], t = target[i];
    const double d = double(q) - double(t);
    s += d * d;
    if (lam) {
      lam[i] = q - t;
      lam[n + i] = R(0);
      lam[2 * n + i] = R(0);
      lam[3 * n + i] = R(0);
    }
  }
  auto cta_sum = [&](double v) {  // on thread 0
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0;
    if (threadIdx.x == 0)
      for (int w = 0; w < kThreads / 32; ++w) v += red[w];
    return v;
  };
  s = cta_sum(s);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  s = 0;
  for (int k = threadIdx.x; k < int(gridDim.x); k += kThreads) s += __ldcg(part + k);
  s = cta_sum(s);
  if (threadIdx.x == 0) out[0] = 0.5 * s;
}

struct Run {
  cfdb_ctx* ctx;
  cfdb_mesh* m;
  int dtype, path;
  const void* c;
  double dt;
  size_t esz;
  int64_t n;

  int step(const void* src, void* dst) const {
    return cfdb_wave_step(ctx, m, dtype, path, src, dst, c, 0.0, 1, dt);
  }
  int adjoint(const void* q, const void* lam1, void* lam0, void* gc) const {
    return cfdb_wave_adjoint_step(ctx, m, dtype, path, q, lam1, lam0, c, gc, dt);
  }
  int copy(void* dst, const void* src) const {
    CFDB_CUDA(ctx, cudaMemcpyAsync(dst, src, 4 * n * esz, cudaMemcpyDeviceToDevice, ctx->stream));
    return CFDB_OK;
  }
  // J to the end of `scratch` (misfit_bytes()) and, when lam != nullptr, the adjoint
  // seed; read_misfit() waits for it and returns it.
  int64_t misfit_bytes() const { return int64_t(8) * (grid_for(ctx, n, kThreads, 2) + 2); }
  int misfit(const void* qT, const void* target, void* lam, void* scratch) const {
    const int grid = grid_for(ctx, n, kThreads, 2);
    double* part = static_cast<double*>(scratch);
    unsigned* ticket = reinterpret_cast<unsigned*>(part + grid + 1);
    CFDB_CUDA(ctx, cudaMemsetAsync(ticket, 0, sizeof(unsigned), ctx->stream));
    if (dtype == CFDB_F64)
      misfit_k<double><<<grid, kThreads, 0, ctx->stream>>>((const double*)qT, (const double*)target, (double*)lam, n, part, ticket, part + grid);
    else
      misfit_k<float><<<grid, kThreads, 0, ctx->stream>>>((const float*)qT, (const float*)target, (float*)lam, n, part, ticket, part + grid);
    CFDB_LAUNCHED(ctx);
    return CFDB_OK;
  }
  int read_misfit(const void* scratch, double* host) const {
    const double* res = static_cast<const double*>(scratch) + grid_for(ctx, n, kThreads, 2);
    CFDB_CUDA(ctx, cudaMemcpyAsync(host, res, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CFDB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CFDB_OK;
  }
};

int check_args(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, int path, const void* q0, const void* c, const void* target,
               int32_t steps, double dt, const char* fn) {
  if (int rc = cfdb_check_mesh(ctx, m)) return rc;
  if (!dtype_ok(dtype)) return cfdb_fail(ctx, CFDB_EINVAL, "%s: unknown dtype %d", fn, dtype);
  if (path != CFDB_PATH_PLAIN && path != CFDB_PATH_FUSED) return cfdb_fail(ctx, CFDB_EINVAL, "%s: unknown path", fn);
  if (!q0 || !c || !target) return cfdb_fail(ctx, CFDB_EINVAL, "%s: NULL input", fn);
  if (steps < 1 || !(dt > 0) || !std::isfinite(dt)) return cfdb_fail(ctx, CFDB_EINVAL, "%s: need steps >= 1 and dt > 0", fn);
  CFDB_CUDA(ctx, cudaSetDevice(ctx->device));
  return CFDB_OK;
}

// Workspaces of one call, taken from the context's pool and returned to it
// (stream-ordered) when the call ends.
struct Bufs {
  cfdb_ctx* ctx;
  std::vector<void*> v;
  ~Bufs() {
    for (void* p : v) cfdb_ws_free(ctx, p);
  }
  int get(int64_t bytes, void** out) {
    int rc = cfdb_ws_alloc(ctx, bytes, out);
    if (!rc) v.push_back(*out);
    return rc;
  }
};

}  // namespace

extern "C" int cfdb_wave_objective(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, int path, const void* q0, const void* c,
                                   const void* target, int32_t steps, double dt, double* J_out) {
  CfdbRange range_("cfdb_wave_objective");
  if (int rc = check_args(ctx, m, dtype, path, q0, c, target, steps, dt, "cfdb_wave_objective")) return rc;
  if (!J_out) return cfdb_fail(ctx, CFDB_EINVAL, "cfdb_wave_objective: J_out is NULL");
  Run R{ctx, m, dtype, path, c, dt, dtype_size(dtype), m->n};
  Bufs B{ctx, {}};
  void *a, *b, *scratch;
  if (int rc = B.get(int64_t(4 * R.esz) * R.n, &a)) return rc;
  if (int rc = B.get(int64_t(4 * R.esz) * R.n, &b)) return rc;
  if (int rc = B.get(R.misfit_bytes(), &scratch)) return rc;
  if (int rc = R.copy(a, q0)) return rc;
  if (int rc = cfdb_run_steps(ctx, a, b, steps, 1, [&](const void* s, void* d) { return R.step(s, d); },
                              graph_key("wave", m, dtype, path, a, b, c, {0.0, 1.0, dt})))
    return rc;
  if (int rc = R.misfit((steps & 1) ? b : a, target, nullptr, scratch)) return rc;
  return R.read_misfit(scratch, J_out);
}

extern "C" int cfdb_wave_gradient(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, int path, const void* q0, const void* c,
                                  const void* target, int32_t steps, double dt, int32_t snapshots, double* J_out,
                                  void* grad_c, void* grad_p0, cfdb_gradient_stats* stats) {
  CfdbRange range_("cfdb_wave_gradient");
  if (int rc = check_args(ctx, m, dtype, path, q0, c, target, steps, dt, "cfdb_wave_gradient")) return rc;
  if (!J_out || !grad_c || !grad_p0) return cfdb_fail(ctx, CFDB_EINVAL, "cfdb_wave_gradient: NULL output");
  if (snapshots < 1) return cfdb_fail(ctx, CFDB_EINVAL, "cfdb_wave_gradient: snapshots must be >= 1");
  Run R{ctx, m, dtype, path, c, dt, dtype_size(dtype), m->n};
  const int64_t sb = int64_t(4 * R.esz) * R.n;  // one state
  Bufs B{ctx, {}};
  void *lamA, *lamB, *scratch;
  if (int rc = B.get(sb, &lamA)) return rc;
  if (int rc = B.get(sb, &lamB)) return rc;
  if (int rc = B.get(R.misfit_bytes(), &scratch)) return rc;
  CFDB_CUDA(ctx, cudaMemsetAsync(grad_c, 0, R.esz * R.n, ctx->stream));
  cudaEvent_t e0, e1, e2;
  CFDB_CUDA(ctx, cudaEventCreate(&e0));
  CFDB_CUDA(ctx, cudaEventCreate(&e1));
  CFDB_CUDA(ctx, cudaEventCreate(&e2));
  struct EvGuard {
    cudaEvent_t a, b, c;
    ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); cudaEventDestroy(c); }
  } evg{e0, e1, e2};
  cfdb_gradient_stats st{};
  int rc = CFDB_OK;
  void* lam = lamA;
  void* lam_next = lamB;
  auto adj = [&](const void* q) {
    int r = R.adjoint(q, lam, lam_next, grad_c);
    std::swap(lam, lam_next);
    ++st.adjoint_steps;
    return r;
  };

  if (snapshots >= steps) {
    // every state in its own slot; the forward step writes the checkpoint
    char* states = nullptr;
    if ((rc = B.get(sb * (int64_t(steps) + 1), reinterpret_cast<void**>(&states))))
      return cfdb_fail(ctx, rc, "cfdb_wave_gradient: %d stored states (%lld bytes) do not fit; pass fewer snapshots",
                       steps + 1, (long long)(sb * (int64_t(steps) + 1)));
    auto slot = [&](int t) { return static_cast<void*>(states + sb * int64_t(t)); };
    if ((rc = R.copy(slot(0), q0))) return rc;
    cudaEventRecord(e0, ctx->stream);
    {
      CfdbRange forward("cfdb_wave_gradient: forward sweep");
      for (int t = 0; t < steps && !rc; ++t) rc = R.step(slot(t), slot(t + 1));
    }
    cudaEventRecord(e1, ctx->stream);
    if (rc) return rc;
    st.forward_steps = steps;
    st.snapshots_used = steps + 1;
    if ((rc = R.misfit(slot(steps), target, lam, scratch))) return rc;
    CfdbRange reverse("cfdb_wave_gradient: reverse sweep");
    for (int t = steps - 1; t >= 0 && !rc; --t) rc = adj(slot(t));
  } else {
    std::vector<int32_t> act, arg, at;
    int64_t fwd = 0;
    cfdb_revolve_build(steps, snapshots, act, arg, at, &fwd);
    char* slots = nullptr;
    void *cur, *tmp;
    if ((rc = B.get(sb * snapshots, reinterpret_cast<void**>(&slots)))) return rc;
    if ((rc = B.get(sb, &cur))) return rc;
    if ((rc = B.get(sb, &tmp))) return rc;
    auto slot = [&](int k) { return static_cast<void*>(slots + sb * int64_t(k)); };
    if ((rc = R.copy(cur, q0))) return rc;
    cudaEventRecord(e0, ctx->stream);
    bool first_turn_seen = false;
    for (size_t k = 0; k < act.size() && !rc; ++k) {
      switch (act[k]) {
        case CFDB_RV_TAKESHOT: rc = R.copy(slot(arg[k]), cur); break;
        case CFDB_RV_RESTORE: rc = R.copy(cur, slot(arg[k])); break;
        case CFDB_RV_ADVANCE:
          for (int j = 0; j < arg[k] && !rc; ++j) {
            rc = R.step(cur, tmp);
            std::swap(cur, tmp);
            ++st.forward_steps;
          }
          break;
        case CFDB_RV_FIRSTURN:
          cudaEventRecord(e1, ctx->stream);
          first_turn_seen = true;
          if ((rc = R.step(cur, tmp))) break;  // q_T
          ++st.forward_steps;
          if ((rc = R.misfit(tmp, target, lam, scratch))) break;
          rc = adj(cur);
          break;
        case CFDB_RV_YOUTURN: rc = adj(cur); break;
        default: rc = cfdb_fail(ctx, CFDB_EINVAL, "corrupt checkpoint schedule"); break;
      }
    }
    if (!first_turn_seen && !rc) rc = cfdb_fail(ctx, CFDB_EINVAL, "checkpoint schedule has no first turn");
    st.snapshots_used = snapshots;
  }
  if (rc) return rc;
  // dJ/dp0 = the pressure block of lam_0
  CFDB_CUDA(ctx, cudaMemcpyAsync(grad_p0, lam, R.esz * R.n, cudaMemcpyDeviceToDevice, ctx->stream));
  cudaEventRecord(e2, ctx->stream);
  if ((rc = R.read_misfit(scratch, J_out))) return rc;  // the call's one wait
  float f = 0, r = 0;
  cudaEventElapsedTime(&f, e0, e1);
  cudaEventElapsedTime(&r, e1, e2);
  st.forward_ms = f;
  st.reverse_ms = r;
  if (stats) *stats = st;
  return CFDB_OK;
}
