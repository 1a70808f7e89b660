// The plain operators and the plain acoustic step on structured meshes,
// without the reference's N x 6 geometry arrays.
//
// What bounds the array kernels of plain_ops.cu is the geometry they read: 62
// values per cell around the one or four field values that a step needs (200^3
// FP32: gradient 200 us, Laplacian 381 us, stabilisation 1092 us; the fields
// alone take 10 us of HBM time each).  On a structured mesh all of it follows
// from three short tables: every face is axis-aligned, so its unit normal is
// +-e_d exactly, its area is the rounded product of two edge lengths, alpha
// and |x_f - x_P| depend on one index each, and only the cell volume (a sum of
// six rounded terms) may differ from cell to cell: it is one value when all
// cells round to the same, and one array otherwise.  axis_tables() (host,
// geometry.cpp) evaluates the formulas of geometry_cell.hpp per axis, in the
// same operation order, and refuses meshes for which the reduction to one
// axis is not exact; those keep the array kernels.
//
// Results are the array kernels' bits.  The products by the zero components of
// a normal are left out: each is +-0 for finite operands, and adding +-0 to an
// accumulator that starts at +0 changes nothing.  For an operand that is not
// finite the array form turns such a product into NaN, so the kernels look at
// every value the array form would have multiplied by zero and give NaN (or,
// where more than one stage is chained, evaluate the cell by the full sums:
// *_full below).
//
// Layout: what bounds these kernels once the geometry is gone is instruction
// issue, so every face is evaluated once.  A thread owns NY consecutive rows at
// one z and marches a chunk of x planes: the face above a plane is carried in
// registers as the next plane's face below, the faces between a thread's rows
// are shared by them, and the z neighbours are the adjacent lanes of the warp.
// The lanes run along z across row groups (32 consecutive (group, z) pairs,
// the outer HZ on each side computing for their neighbours only), so rows of
// any length waste no lanes; a lane at a z wall uses no neighbour.  Warps never
// wait for one another.  (One cell per thread with neighbours through L1, the
// first form, took 45, 50 and 262 us for the gradient, Laplacian and
// stabilisation at 200^3 FP32, 139 and 565 instructions per cell.)
// Compiled with --fmad=false like plain_ops.cu.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <limits>

#include "euler_internal.hpp"

CFDB_MODULE_ANCHOR

namespace {

constexpr int kThreads = 128;

template <class R> struct Box {
  int nx, ny, nz;
  unsigned plane;           // ny nz
  int groups;               // row groups of NY rows
  unsigned tiles, chunks;   // warps across (group, z) and along x
  const double *hx, *hy, *hz;   // edge lengths
  const R *ax, *ay, *az;        // alpha of the face below cell i (entry i), 0 .. n
  const R *lmx, *lpx, *lmy, *lpy, *lmz, *lpz;  // |x_f - x_P| of the - and + faces
  const R* vol;                 // cell volumes, or null: v for every cell
  R v, rv;                      // rv = 1 / v
  R limit;                      // magnitudes up to this overflow in no intermediate
  // one value per direction for the whole mesh (UNI kernels)
  R A[3], al[3], lm[3], lp[3];
  __device__ R volume(int64_t i) const { return vol ? vol[i] : v; }
};

template <class R> __device__ __forceinline__ bool finite(R v) { return fabs(v) <= std::numeric_limits<R>::max(); }

// ---- the array form of one cell, for operands that are not finite ------------

struct Cell {
  int x, y, z;
};
template <class R> __device__ int64_t id_of(const Box<R>& g, Cell c) { return int64_t(c.x) * g.plane + c.y * g.nz + c.z; }
// neighbour through slot f, the cell itself on a wall
template <class R> __device__ Cell beyond(const Box<R>& g, Cell c, int f) {
  switch (f) {
    case 0: c.z = max(c.z - 1, 0); break;
    case 1: c.z = min(c.z + 1, g.nz - 1); break;
    case 2: c.y = max(c.y - 1, 0); break;
    case 3: c.y = min(c.y + 1, g.ny - 1); break;
    case 4: c.x = max(c.x - 1, 0); break;
    default: c.x = min(c.x + 1, g.nx - 1); break;
  }
  return c;
}
template <class R> __device__ R area_of(const Box<R>& g, Cell c, int f) {
  return f < 2 ? R(g.hx[c.x] * g.hy[c.y]) : f < 4 ? R(g.hx[c.x] * g.hz[c.z]) : R(g.hy[c.y] * g.hz[c.z]);
}
template <class R> __device__ R length_of(const Box<R>& g, Cell c, int f) {
  switch (f) {
    case 0: return g.lmz[c.z];
    case 1: return g.lpz[c.z];
    case 2: return g.lmy[c.y];
    case 3: return g.lpy[c.y];
    case 4: return g.lmx[c.x];
    default: return g.lpx[c.x];
  }
}
// component d of the outward normal of slot f
template <class R> __device__ R outward(int f, int d) { return d == 2 - f / 2 ? (f & 1 ? R(1) : R(-1)) : R(0); }

template <class R> __device__ R grad_full(const Box<R>& g, const R* phi, Cell c, int d) {
  const int64_t i = id_of(g, c);
  R acc = R(0);
  for (int f = 0; f < 6; ++f) {
    const R itp = (phi[i] + phi[id_of(g, beyond(g, c, f))]) * R(0.5);
    acc = acc + itp * outward<R>(f, d) * area_of(g, c, f);
  }
  return acc / g.volume(i);
}

template <class R> __device__ __noinline__ R stab_full(const Box<R>& g, const R* phi, int x, int y, int z, int mask) {
  const Cell c{x, y, z};
  const int64_t i = id_of(g, c);
  R res = R(0);
  for (int d = 0; d < 3; ++d) {
    if (!(mask & (1 << d))) continue;
    const R gd = grad_full(g, phi, c, d);
    R acc = R(0);
    for (int f = 0; f < 6; ++f) {
      const Cell nb = beyond(g, c, f);
      const R up = phi[i] + length_of(g, c, f) * gd * outward<R>(f, d);
      const R col = phi[id_of(g, nb)] + length_of(g, nb, f ^ 1) * grad_full(g, phi, nb, d) * outward<R>(f ^ 1, d);
      const R s = R(0.5) * (up - col);
      acc = acc + s * fabs(outward<R>(f, d)) * area_of(g, c, f);
    }
    res = res + acc / g.volume(i);
  }
  return res;
}

template <class R> __device__ __noinline__ R grad_sum_full(const Box<R>& g, const R* phi, int x, int y, int z, int mask) {
  R res = R(0);
  for (int d = 0; d < 3; ++d)
    if (mask & (1 << d)) res = res + grad_full(g, phi, Cell{x, y, z}, d);
  return res;
}

template <class R> __device__ __noinline__ R lapl_full(const Box<R>& g, const R* phi, int x, int y, int z, int mask) {
  const Cell c{x, y, z};
  const int64_t i = id_of(g, c);
  const R alpha[6] = {g.az[z], g.az[z + 1], g.ay[y], g.ay[y + 1], g.ax[x], g.ax[x + 1]};
  R res = R(0);
  for (int d = 0; d < 3; ++d) {
    if (!(mask & (1 << d))) continue;
    R acc = R(0);
    for (int f = 0; f < 6; ++f) {
      const R sn = (phi[id_of(g, beyond(g, c, f))] - phi[i]) * alpha[f];
      acc = acc + sn * fabs(outward<R>(f, d)) * area_of(g, c, f);
    }
    res = res + acc / g.volume(i);
  }
  return res;
}

// Division by a cell volume. The volume divides several sums of a cell, so its
// reciprocal r = fl(1 / v) is formed once and each quotient takes a product and
// two corrections by the exact remainder: with r correctly rounded and the
// quotient within one unit in the last place, fl(q + fl(a - q v) r) is the
// correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34(1), 1990).  That
// needs remainders that do not underflow: a smaller nonzero dividend is divided
// directly, and volumes are in [2^-80, 2^24] (other meshes keep the array
// kernels).  A result that is not finite is computed again by the callers.
// (Three IEEE divisions had been about 60 of the gradient's 102 instructions
// per cell.)
template <class R> struct Volume {
  R v, r;
  __device__ __forceinline__ R quot(R a) const {
    R q = a * r;
    q = fma(fma(-q, v, a), r, q);
    return fma(fma(-q, v, a), r, q);
  }
  // a[d] = fl(a[d] / v) for N sums of one cell, one branch for all of them
  template <int N> __device__ __forceinline__ void divide(R a[N]) const {
    R least = fabs(a[0]);
#pragma unroll
    for (int d = 1; d < N; ++d) least = fmin(least, fabs(a[d]));
    bool direct = false;
    if (least < (sizeof(R) == 8 ? R(1e-288) : R(1e-30))) {  // zero divides exactly
#pragma unroll
      for (int d = 0; d < N; ++d) direct = direct || (fabs(a[d]) < (sizeof(R) == 8 ? R(1e-288) : R(1e-30)) && a[d] != R(0));
    }
    if (direct) {
#pragma unroll
      for (int d = 0; d < N; ++d) a[d] = a[d] / v;
    } else {
#pragma unroll
      for (int d = 0; d < N; ++d) a[d] = quot(a[d]);
    }
  }
};

// ---- the march ------------------------------------------------------------------

constexpr unsigned kWarp = 0xffffffffu;

// A thread's place: NY rows from y0 at one z, planes [x0, x1).  off[HY + r] is
// row y0 + r within a plane, r = -HY .. NY + HY - 1, walls repeated (a wall
// face's neighbour is the cell itself, and so are rows beyond the last).
template <int NY, int HY, int HZ> struct March {
  int y0, z, x0, x1;
  int off[NY + 2 * HY];
  bool out, zlo, zhi;
  template <class G> __device__ __forceinline__ bool start(const G& g) {
    const unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= g.tiles * g.chunks) return false;  // whole warps
    const unsigned chunk = w / g.tiles, tile = w - chunk * g.tiles;
    const int64_t S = int64_t(g.groups) * g.nz, at = int64_t(tile) * (32 - 2 * HZ) + int(lane) - HZ;
    out = int(lane) >= HZ && int(lane) < 32 - HZ && at < S;
    const int s = int(min(max(at, int64_t(0)), S - 1));
    const int grp = s / g.nz;
    z = s - grp * g.nz;
    y0 = grp * NY;
#pragma unroll
    for (int r = -HY; r < NY + HY; ++r) off[r + HY] = min(max(y0 + r, 0), g.ny - 1) * g.nz + z;
    x0 = int(int64_t(chunk) * g.nx / g.chunks);
    x1 = int(int64_t(chunk + 1) * g.nx / g.chunks);
    zlo = z == 0;
    zhi = z == g.nz - 1;
    return true;
  }
};

enum { OP_GRAD = 0, OP_LAPL = 1, OP_HEAT = 2 };

// GradVar (grad_k): sum over the masked directions of (sum_f itp_f n_d A) / V,
// itp = (phi_P + phi_N) / 2, and Grad2Var (lapl_k): the same with
// sn_f = (phi_N - phi_P) alpha_f and the unsigned normal +e_d on both faces.
// With F the face value between the lower and the upper cell times the area,
// both sum to ((0 - F_lower) + F_upper) / V per direction: the lower face enters
// with the opposite sign, which rounds alike.  HEAT: the update dt (k L) + phi
// of heat_update_k in the same pass.  UNI: one area, alpha and volume for the
// whole mesh.  A result that is not finite (every face value reaches it: FULL
// sums all three directions, and the others are summed to look at) is computed
// again by the full sums.
// 200^3 FP32 (64 MB): floor 10 us.
template <class R, int OP, int NY, bool UNI, bool FULL>
__global__ void __launch_bounds__(kThreads) box_sum_k(const __grid_constant__ Box<R> g, const R* __restrict__ phi, R* __restrict__ out, int mask_,
                                                      R k, R dt) {
  March<NY, 1, 1> w;
  if (!w.start(g)) return;
  const int mask = FULL ? 7 : mask_;
  const int64_t pl = g.plane;
  auto face = [](R lo, R hi, R alpha, R A) {
    if constexpr (OP == OP_GRAD) return ((lo + hi) * R(0.5)) * A;
    else return ((hi - lo) * alpha) * A;
  };
  R Ax[NY], ayv[NY + 1];
  double hy[NY];
  const double hz = UNI ? 0.0 : g.hz[w.z];
#pragma unroll
  for (int r = 0; r < NY; ++r) {
    const int y = min(w.y0 + r, g.ny - 1);
    hy[r] = UNI ? 0.0 : g.hy[y];
    Ax[r] = UNI ? g.A[0] : R(hy[r] * hz);
  }
#pragma unroll
  for (int r = 0; r <= NY; ++r) ayv[r] = OP == OP_GRAD ? R(0) : UNI ? g.al[1] : g.ay[min(w.y0 + r, g.ny)];
  const R azl = OP == OP_GRAD ? R(0) : UNI ? g.al[2] : g.az[w.z], azh = OP == OP_GRAD ? R(0) : UNI ? g.al[2] : g.az[w.z + 1];
  const R* q = phi + w.x0 * pl;
  R cur[NY], nxt[NY], fx[NY];
  {
    const int64_t back = w.x0 > 0 ? pl : 0;
    const R alpha = OP == OP_GRAD ? R(0) : UNI ? g.al[0] : g.ax[w.x0];
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      cur[r] = q[w.off[1 + r]];
      fx[r] = face(q[w.off[1 + r] - back], cur[r], alpha, Ax[r]);
    }
  }
  for (int x = w.x0; x < w.x1; ++x, q += pl) {
    const R* qn = q + (x < g.nx - 1 ? pl : 0);
    const R lo = q[w.off[0]], hi = q[w.off[NY + 1]];
#pragma unroll
    for (int r = 0; r < NY; ++r) nxt[r] = qn[w.off[1 + r]];
    const double hx = UNI ? 0.0 : g.hx[x];
    const R Ay = UNI ? g.A[1] : R(hx * hz);
    const R axv = OP == OP_GRAD ? R(0) : UNI ? g.al[0] : g.ax[x + 1];
    R fy = face(lo, cur[0], ayv[0], Ay);
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      const R P = cur[r];
      const int64_t i = x * pl + w.off[1 + r];
      const R vol = UNI ? g.v : g.volume(i);
      const Volume<R> V{vol, UNI ? g.rv : R(1) / vol};
      const R Az = UNI ? g.A[2] : R(hx * hy[r]);
      R zm = __shfl_up_sync(kWarp, P, 1), zp = __shfl_down_sync(kWarp, P, 1);
      zm = w.zlo ? P : zm;
      zp = w.zhi ? P : zp;
      const R fxh = face(P, nxt[r], axv, Ax[r]);
      const R fyh = face(P, r + 1 < NY ? cur[r + 1] : hi, ayv[r + 1], Ay);
      R acc[3] = {(R(0) - fx[r]) + fxh, (R(0) - fy) + fyh, (R(0) - face(zm, P, azl, Az)) + face(P, zp, azh, Az)};
      const R all = FULL ? R(0) : (acc[0] + acc[1]) + acc[2];
      V.template divide<3>(acc);
      fx[r] = fxh;
      fy = fyh;
      R res = R(0);
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (mask & (1 << d)) res = res + acc[d];
      const bool rows = w.y0 + r < g.ny;
      if (w.out && rows) {
        if (!finite(res) || (!FULL && !finite(all)))
          res = OP == OP_GRAD ? grad_sum_full(g, phi, x, w.y0 + r, w.z, mask) : lapl_full(g, phi, x, w.y0 + r, w.z, mask);
        out[i] = OP == OP_HEAT ? dt * (k * res) + P : res;
      }
    }
#pragma unroll
    for (int r = 0; r < NY; ++r) cur[r] = nxt[r];
  }
}

// StabVar, both stages at once (stab1_k + stab2_k, whose 18 values per cell
// between the stages made 3.5 GB of traffic at 200^3 FP32).  Along a direction,
// with g the cell gradient and a cell's face values up = phi + len g on its
// upper face and um = phi - len g on its lower, a face between B (below) and
// A (above) contributes E = (0.5 (up_B - um_A)) A: ((0 - E_lower) + E_upper) / V.
// A wall cell faces itself (E from its own up and um).
// Planes x + 1 and x + 2 are in registers while plane x is finished (its x
// neighbours' gradients need them).  `fine` is kept per plane and warp: all
// values of the rows and lanes that the array form would have touched are small
// enough that no intermediate overflows; a plane within two of one that is
// not is computed by the full sums.
template <class R, int NY, bool UNI, bool FULL>
__global__ void __launch_bounds__(kThreads) box_stab_k(const __grid_constant__ Box<R> g, const R* __restrict__ phi, R* __restrict__ out, int mask_) {
  constexpr int NR = NY + 4;  // rows -2 .. NY + 1
  March<NY, 2, 2> w;
  if (!w.start(g)) return;
  const int mask = FULL ? 7 : mask_;
  const int64_t pl = g.plane;
  const double hz = UNI ? 0.0 : g.hz[w.z];
  auto plane = [&](int x) { return phi + int64_t(min(max(x, 0), g.nx - 1)) * pl; };
  unsigned fine = 0;  // bit k: plane (newest - k) is fine
  auto load = [&](int x, R v[NR]) {
    const R* q = plane(x);
    bool ok = true;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      v[r] = q[w.off[r]];
      ok = ok && fabs(v[r]) <= g.limit;
    }
    fine = fine << 1 | (__all_sync(kWarp, ok) ? 1u : 0u);
  };
  auto vol_at = [&](int x, int r) {  // row r of plane x (walls repeated)
    const R v = UNI ? g.v : g.volume(int64_t(min(max(x, 0), g.nx - 1)) * pl + w.off[r + 2]);
    return Volume<R>{v, UNI ? g.rv : R(1) / v};
  };
  auto over = [](const Volume<R>& V, R a) {
    V.template divide<1>(&a);
    return a;
  };
  auto mean = [](R a, R b, R A) { return ((a + b) * R(0.5)) * A; };
  auto edge = [](R up, R um, R A) { return (R(0.5) * (up - um)) * A; };
  auto row = [&](int r) { return min(max(w.y0 + r, 0), g.ny - 1); };
  auto len_lo = [&](int d, int i) { return UNI ? g.lm[d] : d == 0 ? g.lmx[i] : d == 1 ? g.lmy[i] : g.lmz[i]; };
  auto len_hi = [&](int d, int i) { return UNI ? g.lp[d] : d == 0 ? g.lpx[i] : d == 1 ? g.lpy[i] : g.lpz[i]; };
  R Ax[NY];
#pragma unroll
  for (int r = 0; r < NY; ++r) Ax[r] = UNI ? g.A[0] : R(g.hy[row(r)] * hz);
  R cur[NR], n1[NR], n2[NR], fx[NY], gx[NY], ex[NY];  // fx: face (x, x + 1); gx: gradient of plane x; ex: E between x - 1 and x
  {
    R b2[NR], b1[NR];
    load(w.x0 - 2, b2);
    load(w.x0 - 1, b1);
    load(w.x0, cur);
    load(w.x0 + 1, n1);
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      const R flo = mean(b1[r + 2], cur[r + 2], Ax[r]);  // at x = 0 the wall face: b1 repeats cur
      fx[r] = mean(cur[r + 2], n1[r + 2], Ax[r]);
      gx[r] = over(vol_at(w.x0, r), (R(0) - flo) + fx[r]);
      const R um = cur[r + 2] - len_lo(0, w.x0) * gx[r];
      R up;
      if (w.x0 > 0) {
        const R gB = over(vol_at(w.x0 - 1, r), (R(0) - mean(b2[r + 2], b1[r + 2], Ax[r])) + flo);
        up = b1[r + 2] + len_hi(0, w.x0 - 1) * gB;
      } else {
        up = cur[r + 2] + len_hi(0, w.x0) * gx[r];
      }
      ex[r] = edge(up, um, Ax[r]);
    }
  }
  for (int x = w.x0; x < w.x1; ++x) {
    load(x + 2, n2);
    const bool all_fine = (fine & 31u) == 31u;
    const double hx = UNI ? 0.0 : g.hx[x];
    const R Ay = UNI ? g.A[1] : R(hx * hz);
    const bool xhi = x == g.nx - 1;
    const int xn = min(x + 1, g.nx - 1);
    // y direction, rolling over the rows: gradient and face values of the row
    // below the thread's first, then of each row and the one above it
    R fy = mean(cur[1], cur[2], Ay), upB;
    {
      const R gB = over(vol_at(x, -1), (R(0) - mean(cur[0], cur[1], Ay)) + fy);
      upB = cur[1] + len_hi(1, row(-1)) * gB;
    }
    R fyh = mean(cur[2], cur[3], Ay);
    R gy = over(vol_at(x, 0), (R(0) - fy) + fyh);
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      const R P = cur[r + 2];
      const int y = w.y0 + r;
      const int64_t i = x * pl + w.off[r + 2];
      const Volume<R> V = vol_at(x, r);
      const R Az = UNI ? g.A[2] : R(hx * g.hy[row(r)]);
      R zm = __shfl_up_sync(kWarp, P, 1), zp = __shfl_down_sync(kWarp, P, 1);
      zm = w.zlo ? P : zm;
      zp = w.zhi ? P : zp;
      // the gradients this row needs next: of its x neighbour above, its y
      // neighbour above and its own along z
      const R fx2 = mean(n1[r + 2], n2[r + 2], Ax[r]), fy2 = mean(cur[r + 3], cur[r + 4], Ay);
      R gr[3] = {(R(0) - fx[r]) + fx2, (R(0) - fyh) + fy2, (R(0) - mean(zm, P, Az)) + mean(P, zp, Az)};
      if constexpr (UNI) {
        V.template divide<3>(gr);
      } else {
        gr[0] = over(vol_at(x + 1, r), gr[0]);
        gr[1] = over(vol_at(x, r + 1), gr[1]);
        gr[2] = over(V, gr[2]);
      }
      R s3[3];
      {  // x
        const R up = P + len_hi(0, x) * gx[r];
        const R um1 = xhi ? P - len_lo(0, x) * gx[r] : n1[r + 2] - len_lo(0, xn) * gr[0];
        const R e = edge(up, um1, Ax[r]);
        s3[0] = (R(0) - ex[r]) + e;
        ex[r] = e;
        fx[r] = fx2;
        gx[r] = gr[0];
      }
      {  // y
        const R um = P - len_lo(1, row(r)) * gy, up = P + len_hi(1, row(r)) * gy;
        const R umA = y >= g.ny - 1 ? um : cur[r + 3] - len_lo(1, row(r + 1)) * gr[1];
        if (y == 0) upB = up;
        s3[1] = (R(0) - edge(upB, um, Ay)) + edge(up, umA, Ay);
        upB = up;
        fyh = fy2;
        gy = gr[1];
      }
      {  // z
        const R um = P - len_lo(2, w.z) * gr[2], up = P + len_hi(2, w.z) * gr[2];
        R upb = __shfl_up_sync(kWarp, up, 1), uma = __shfl_down_sync(kWarp, um, 1);
        upb = w.zlo ? up : upb;
        uma = w.zhi ? um : uma;
        s3[2] = (R(0) - edge(upb, um, Az)) + edge(up, uma, Az);
      }
      V.template divide<3>(s3);
      R res = R(0);
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (mask & (1 << d)) res = res + s3[d];
      if (w.out && y < g.ny) {
        if (!all_fine) res = stab_full(g, phi, x, y, w.z, mask);
        out[i] = res;
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      cur[r] = n1[r];
      n1[r] = n2[r];
    }
  }
}

// ---- vertex meshes: every face's geometry once ------------------------------------
//
// The N x 6 arrays hold each interior face twice, with its normal once as it is
// (normal) and once turned outward (normal_alt): 62 values and six neighbour ids
// per cell.  Both cells of a face compute its normal, area and alpha from the same
// vertices in the same order, so the values are the same bits up to the normal's
// sign (cells are checked not to be tangled): one normal along +axis, one area and
// one alpha per face, three faces per cell, serve both.  The face enters the lower
// cell's sums with a plus and the upper cell's with a minus sign, which rounds like
// the array form from either side; sums run over the slots in the array form's
// order, no product is left out, so the results are its bits for any operand.
// What bounds these kernels is the geometry still read, 16 values per cell for the
// Laplacian (FP64 80 x 72 x 66: 49 MB, from L2).

template <class R> struct Vert {
  int nx, ny, nz;
  unsigned plane;
  int groups;
  unsigned tiles, chunks;
  const R* nrm[3][3];  // axis, component: unit normal along +axis
  const R* area[3];
  const R* alpha[3];
  const R* len[6];     // |x_f - x_P| by slot, per cell
  const R* vol;
  // the face below cell (x, y, z) along each axis; the one above is a step further
  __device__ int64_t face(int axis, int x, int y, int z) const {
    return axis == 0 ? (int64_t(x) * ny + y) * nz + z : axis == 1 ? (int64_t(x) * (ny + 1) + y) * nz + z
                                                                  : (int64_t(x) * ny + y) * (nz + 1) + z;
  }
};

// a[d] = fl(a[d] / v), any dividends
template <class R> __device__ __forceinline__ void divide_any(R a[3], R v) {
  const Volume<R> V{v, R(1) / v};
  R q[3] = {a[0], a[1], a[2]};
  V.template divide<3>(q);
  if (finite((q[0] + q[1]) + q[2])) {
#pragma unroll
    for (int d = 0; d < 3; ++d) a[d] = q[d];
  } else {
#pragma unroll
    for (int d = 0; d < 3; ++d) a[d] = a[d] / v;
  }
}

enum { OUT_SUM = 0, OUT_GRADIENT = 1 };

// Gradient (OP_GRAD) or Laplacian (OP_LAPL, OP_HEAT) of every cell; OUT_GRADIENT
// stores the three gradient components (arrays of n) instead of their masked sum.
// One cell per thread, all of its loads in flight at once: what bounds it is memory
// beyond L2 and latency below.  Asked for 8 CTAs per SM the compiler keeps the loads
// together (left alone it takes 32 registers and waits for them one face after the
// other).  us, array kernels / a march that evaluates every face once / this: FP64
// 100^3 gradient 38.4 / 32.9 / 22.0, Laplacian 78 / 35.5 / 24.7, FP32 160^3 102 / 65 / 51
// and 201 / 66 / 60, FP32 32x24x20 2.2 / 3.4 / 1.9 and 2.6 / 3.6 / 1.9.  (The FP32
// gradient of 0.2 to 0.4 million cells is the array kernels' 3.4 and 5.4 us in 3.8 and
// 5.8 us: rows of nz + 1 faces start off the 32-byte sectors.)
template <class R, int OP, int OUT>
__global__ void __launch_bounds__(kThreads, 8) vert_cell_k(const __grid_constant__ Vert<R> g, const R* __restrict__ phi,
                                                   R* __restrict__ out, int mask, R k, R dt) {
  const int64_t pl = g.plane, n = int64_t(g.nx) * pl;
  const int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x;
  if (i >= n) return;
  const unsigned x_ = unsigned(i) / g.plane, r = unsigned(i) - x_ * g.plane, y_ = r / unsigned(g.nz);
  const int x = int(x_), y = int(y_), z = int(r - y_ * unsigned(g.nz));
  const R P = phi[i], V = g.vol[i];
  // all loads before the sums: z-, z+, y-, y+, x-, x+
  R N[6], A[6], al[6], nr[6][3];
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const int axis = 2 - s / 2, up = s & 1;
    const int64_t step = axis == 0 ? pl : axis == 1 ? g.nz : 1, f = g.face(axis, x, y, z) + up * step;
    const int at = axis == 0 ? x : axis == 1 ? y : z, wall = up ? (axis == 0 ? g.nx : axis == 1 ? g.ny : g.nz) - 1 : 0;
    N[s] = phi[at == wall ? i : up ? i + step : i - step];
    A[s] = g.area[axis][f];
    al[s] = OP == OP_GRAD ? R(0) : g.alpha[axis][f];
#pragma unroll
    for (int d = 0; d < 3; ++d) nr[s][d] = g.nrm[axis][d][f];
  }
  R acc[3] = {R(0), R(0), R(0)};
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const R v = OP == OP_GRAD ? (P + N[s]) * R(0.5) : (s & 1 ? N[s] - P : P - N[s]) * al[s];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const R F = (v * nr[s][d]) * A[s];
      acc[d] = s & 1 ? acc[d] + F : acc[d] - F;
    }
  }
  divide_any(acc, V);
  if constexpr (OUT == OUT_GRADIENT) {
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d * n + i] = acc[d];
  } else {
    R res = R(0);
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (mask & (1 << d)) res = res + acc[d];
    out[i] = OP == OP_HEAT ? dt * (k * res) + P : res;
  }
}

// StabVar's second stage from the cell gradients (grad: three arrays of n): with
// up = phi + (len g) n on a face's lower side and um = phi + (len g) (-n) on its
// upper side, the face carries E = ((0.5 (up_L - um_H)) n) A.  On a wall the other
// side is the cell's own value on its opposite face (the reference's ids point
// back to the cell).
template <class R>
__global__ void __launch_bounds__(kThreads) vert_stab_k(const __grid_constant__ Vert<R> g, const R* __restrict__ phi,
                                                   const R* __restrict__ grad, R* __restrict__ out, int mask) {
  March<1, 1, 1> w;
  if (!w.start(g)) return;
  const int64_t pl = g.plane, n = int64_t(g.nx) * pl;
  const int y = w.y0, z = w.z;
  struct Side {
    R phi, g[3];
  };
  auto at = [&](int64_t i) __attribute__((always_inline)) {
    return Side{phi[i], {grad[i], grad[n + i], grad[2 * n + i]}};
  };
  struct Normal {
    R n[3], A;
  };
  auto normal = [&](int axis, int64_t f) __attribute__((always_inline)) {
    return Normal{{g.nrm[axis][0][f], g.nrm[axis][1][f], g.nrm[axis][2][f]}, g.area[axis][f]};
  };
  auto up = [](const Side& s, R len, const Normal& m, int d) { return s.phi + (len * s.g[d]) * m.n[d]; };
  auto um = [](const Side& s, R len, const Normal& m, int d) { return s.phi + (len * s.g[d]) * -m.n[d]; };
  auto edge = [](R lo, R hi, const Normal& m, int d) { return ((R(0.5) * (lo - hi)) * m.n[d]) * m.A; };
  Side P = at(w.x0 * pl + w.off[1]);
  Normal mx = normal(0, g.face(0, w.x0, y, z));  // the x face below
  R Ex[3];
  if (w.x0 > 0) {
    const int64_t j = (w.x0 - 1) * pl + w.off[1];
    const Side B = at(j);
    const R lb = g.len[5][j], la = g.len[4][j + pl];
#pragma unroll
    for (int d = 0; d < 3; ++d) Ex[d] = edge(up(B, lb, mx, d), um(P, la, mx, d), mx, d);
  }
  for (int x = w.x0; x < w.x1; ++x) {
    const int64_t i = x * pl + w.off[1];
    const bool xlo = x == 0, xhi = x == g.nx - 1, ylo = y == 0, yhi = y == g.ny - 1;
    R l[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) l[f] = g.len[f][i];
    R acc[3];
    {  // z: faces 0 and 1
      const int64_t f = g.face(2, x, y, z);
      const Normal mh = normal(2, f + 1);
      Side H;
      H.phi = __shfl_down_sync(kWarp, P.phi, 1);
#pragma unroll
      for (int d = 0; d < 3; ++d) H.g[d] = __shfl_down_sync(kWarp, P.g[d], 1);
      const R lh = __shfl_down_sync(kWarp, l[0], 1);
      const bool wall = w.zlo || w.zhi;
      Normal ml = mh;
      if (wall) ml = normal(2, f);  // the cell's lower face
      R Eh[3], El[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        Eh[d] = edge(up(P, l[1], mh, d), w.zhi ? um(P, l[0], ml, d) : um(H, lh, mh, d), mh, d);
        El[d] = __shfl_up_sync(kWarp, Eh[d], 1);
        if (w.zlo) El[d] = edge(up(P, l[1], mh, d), um(P, l[0], ml, d), ml, d);
        acc[d] = (R(0) - El[d]) + Eh[d];
      }
    }
    {  // y: faces 2 and 3
      const int64_t f = g.face(1, x, y, z);
      const Normal ml = normal(1, f), mh = normal(1, f + g.nz);
      const Side B = at(x * pl + w.off[0]), H = at(x * pl + w.off[2]);
      const R lb = g.len[3][x * pl + w.off[0]], lh = g.len[2][x * pl + w.off[2]];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const R upP = up(P, l[3], mh, d), umP = um(P, l[2], ml, d);
        const R El = edge(ylo ? upP : up(B, lb, ml, d), umP, ml, d);
        const R Eh = edge(upP, yhi ? umP : um(H, lh, mh, d), mh, d);
        acc[d] = (acc[d] - El) + Eh;
      }
    }
    {  // x: faces 4 and 5
      const Normal mh = normal(0, g.face(0, x + 1, y, z));
      const int64_t j = i + (xhi ? 0 : pl);
      const Side N = at(j);
      const R ln = g.len[4][j];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const R upP = up(P, l[5], mh, d), umP = um(P, l[4], mx, d);
        if (xlo) Ex[d] = edge(upP, umP, mx, d);
        const R Eh = edge(upP, xhi ? umP : um(N, ln, mh, d), mh, d);
        acc[d] = (acc[d] - Ex[d]) + Eh;
        Ex[d] = Eh;
      }
      P = N;
      mx = mh;
    }
    divide_any(acc, g.vol[i]);
    if (w.out) {
      R res = R(0);
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (mask & (1 << d)) res = res + acc[d];
      out[i] = res;
    }
  }
}

// ---- the acoustic step (wave_plain_k) --------------------------------------------

template <class R> struct WaveArgs {
  const R* q;
  R* qn;
  const R* c;  // sound speed field, or null: cconst
  R cconst, dt;
  int mode;
};

// The array form of one cell, every product by a normal's zero included.
template <class R> __device__ __noinline__ void wave_full(const Box<R>& g, const WaveArgs<R>& a, int x, int y, int z) {
  const Cell c{x, y, z};
  const int64_t i = id_of(g, c), n = int64_t(g.nx) * g.plane;
  const R cP = a.c ? a.c[i] : a.cconst, c2 = cP * cP;
  const R pP = a.q[i], uP = a.q[n + i], vP = a.q[2 * n + i], wP = a.q[3 * n + i];
  R ap = R(0), au = R(0), av = R(0), aw = R(0);
  for (int f = 0; f < 6; ++f) {
    const R nx = outward<R>(f, 0), ny = outward<R>(f, 1), nz = outward<R>(f, 2);
    const R A = area_of(g, c, f);
    const R unP = (uP * nx + vP * ny) + wP * nz;
    const int64_t j = id_of(g, beyond(g, c, f));
    R pN, uN, vN, wN, cN;
    if (j != i) {
      pN = a.q[j]; uN = a.q[n + j]; vN = a.q[2 * n + j]; wN = a.q[3 * n + j];
      cN = a.c ? a.c[j] : a.cconst;
    } else {
      const R two_un = R(2) * unP;
      pN = pP; uN = uP - two_un * nx; vN = vP - two_un * ny; wN = wP - two_un * nz; cN = cP;
    }
    const R unN = (uN * nx + vN * ny) + wN * nz;
    const R cfc = a.mode == 0 ? fmax(cP, cN) : R(0.5) * (cP + cN);
    const R hc = R(0.5) * cfc;
    const R pm = R(0.5) * (pP + pN);
    ap = ap + (c2 * (R(0.5) * (unP + unN)) - hc * (pN - pP)) * A;
    au = au + (pm * nx - hc * (uN - uP)) * A;
    av = av + (pm * ny - hc * (vN - vP)) * A;
    aw = aw + (pm * nz - hc * (wN - wP)) * A;
  }
  const R V = g.volume(i);
  a.qn[i] = a.dt * (-(ap / V)) + pP;
  a.qn[n + i] = a.dt * (-(au / V)) + uP;
  a.qn[2 * n + i] = a.dt * (-(av / V)) + vP;
  a.qn[3 * n + i] = a.dt * (-(aw / V)) + wP;
}

// The flux of wave_plain_k through the face with normal +e_D between L (below)
// and H (above), times the area, as it enters L's sums with a plus and H's with
// a minus sign (each rounds like the array form's own evaluation from that side).
// With a c field the two cells' c^2 differ, so the pressure flux comes as its two
// parts, fp[0] = (u_L + u_H) / 2 and fp[1] = hc (p_H - p_L).
template <int D, bool CF, class R>
__device__ __forceinline__ void wave_face(const R L[4], const R H[4], R c2, R hc, R A, R F[4], R fp[2]) {
  fp[0] = R(0.5) * (L[1 + D] + H[1 + D]);
  fp[1] = hc * (H[0] - L[0]);
  if (!CF) F[0] = (c2 * fp[0] - fp[1]) * A;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const R diff = hc * (H[1 + e] - L[1 + e]);
    F[1 + e] = (e == D ? R(0.5) * (L[0] + H[0]) - diff : -diff) * A;
  }
}
// The cell beyond a wall: the wall-normal velocity reflected, u - (2 u).
template <int D, class R> __device__ __forceinline__ void wave_ghost(const R P[4], R G[4]) {
#pragma unroll
  for (int f = 0; f < 4; ++f) G[f] = P[f];
  G[1 + D] = P[1 + D] - R(2) * P[1 + D];
}

// A value that is not finite (or overflows) reaches one of the cell's four
// results, which are then computed again by the full sums.
// 100 x 90 x 96 FP64 (55 MB): floor 9 us.
template <class R, int NY, bool UNI, bool CF>
__global__ void __launch_bounds__(kThreads) box_wave_k(const __grid_constant__ Box<R> g, const __grid_constant__ WaveArgs<R> a) {
  March<NY, 1, 1> w;
  if (!w.start(g)) return;
  const int64_t pl = g.plane, n = int64_t(g.nx) * pl;
  const double hz = UNI ? 0.0 : g.hz[w.z];
  auto load = [&](int64_t i, R v[4]) {
#pragma unroll
    for (int f = 0; f < 4; ++f) v[f] = a.q[f * n + i];
  };
  auto half = [&](R cP, R cN) { return R(0.5) * (a.mode == 0 ? fmax(cP, cN) : R(0.5) * (cP + cN)); };
  const R c0 = a.cconst, c20 = c0 * c0, hc0 = half(c0, c0);
  R Ax[NY];
#pragma unroll
  for (int r = 0; r < NY; ++r) Ax[r] = UNI ? g.A[0] : R(g.hy[min(w.y0 + r, g.ny - 1)] * hz);
  R cur[NY][4], nxt[NY][4], tx[NY][4], px[NY][2];  // tx, px: the face between planes x - 1 and x
  R cc[NY], cn[NY];
#pragma unroll
  for (int r = 0; r < NY; ++r) {
    const int64_t i = w.x0 * pl + w.off[1 + r];
    load(i, cur[r]);
    cc[r] = CF ? a.c[i] : c0;
    R B[4], cB = cc[r];
    if (w.x0 > 0) {
      load(i - pl, B);
      if (CF) cB = a.c[i - pl];
    } else {
      wave_ghost<0>(cur[r], B);
    }
    wave_face<0, CF>(B, cur[r], c20, CF ? half(cc[r], cB) : hc0, Ax[r], tx[r], px[r]);
  }
  for (int x = w.x0; x < w.x1; ++x) {
    const int64_t b = x * pl;
    const bool xhi = x == g.nx - 1;
    R lo[4], hi[4], clo = c0, chi = c0;
    load(b + w.off[0], lo);
    load(b + w.off[NY + 1], hi);
    if (CF) {
      clo = a.c[b + w.off[0]];
      chi = a.c[b + w.off[NY + 1]];
    }
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      if (!xhi) {
        load(b + pl + w.off[1 + r], nxt[r]);
        cn[r] = CF ? a.c[b + pl + w.off[1 + r]] : c0;
      } else {
        wave_ghost<0>(cur[r], nxt[r]);
        cn[r] = cc[r];
      }
    }
    const double hx = UNI ? 0.0 : g.hx[x];
    const R Ay = UNI ? g.A[1] : R(hx * hz);
    R ty[4], py[2];
    if (w.y0 == 0) wave_ghost<1>(cur[0], lo);
    wave_face<1, CF>(lo, cur[0], c20, CF ? half(cc[0], clo) : hc0, Ay, ty, py);
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      const R* P = cur[r];
      const int y = w.y0 + r;
      const int64_t i = b + w.off[1 + r];
      const R vol = UNI ? g.v : g.volume(i);
      const Volume<R> V{vol, UNI ? g.rv : R(1) / vol};
      const R Az = UNI ? g.A[2] : R(hx * g.hy[min(y, g.ny - 1)]);
      const R c2 = CF ? cc[r] * cc[r] : c20;
      // z: the face above, and the one below from the lane below
      R Z[4], tz[4], pz[2], tzl[4], pzl[2];
#pragma unroll
      for (int f = 0; f < 4; ++f) Z[f] = __shfl_down_sync(kWarp, P[f], 1);
      R cz = CF ? __shfl_down_sync(kWarp, cc[r], 1) : c0;
      if (w.zhi) {
        wave_ghost<2>(P, Z);
        cz = cc[r];
      }
      wave_face<2, CF>(P, Z, c20, CF ? half(cc[r], cz) : hc0, Az, tz, pz);
#pragma unroll
      for (int f = 0; f < 4; ++f) tzl[f] = __shfl_up_sync(kWarp, tz[f], 1);
      if (CF) {
        pzl[0] = __shfl_up_sync(kWarp, pz[0], 1);
        pzl[1] = __shfl_up_sync(kWarp, pz[1], 1);
      }
      if (w.zlo) {
        wave_ghost<2>(P, Z);
        wave_face<2, CF>(Z, P, c20, CF ? half(cc[r], cc[r]) : hc0, Az, tzl, pzl);
      }
      // y and x: the faces above
      R th[4], ph[2], tu[4], pu[2], N[4];
      R cN = cc[r];
      if (y >= g.ny - 1) {
        wave_ghost<1>(P, N);
      } else {
#pragma unroll
        for (int f = 0; f < 4; ++f) N[f] = r + 1 < NY ? cur[r + 1 < NY ? r + 1 : r][f] : hi[f];
        if (CF) cN = r + 1 < NY ? cc[r + 1 < NY ? r + 1 : r] : chi;
      }
      wave_face<1, CF>(P, N, c20, CF ? half(cc[r], cN) : hc0, Ay, th, ph);
      wave_face<0, CF>(P, nxt[r], c20, CF ? half(cc[r], cn[r]) : hc0, Ax[r], tu, pu);
      if (CF) {  // the pressure flux with this cell's c^2
        tzl[0] = (c2 * pzl[0] - pzl[1]) * Az;
        tz[0] = (c2 * pz[0] - pz[1]) * Az;
        ty[0] = (c2 * py[0] - py[1]) * Ay;
        th[0] = (c2 * ph[0] - ph[1]) * Ay;
        tx[r][0] = (c2 * px[r][0] - px[r][1]) * Ax[r];
        tu[0] = (c2 * pu[0] - pu[1]) * Ax[r];
      }
      R o[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) o[f] = (((((R(0) - tzl[f]) + tz[f]) - ty[f]) + th[f]) - tx[r][f]) + tu[f];
      V.template divide<4>(o);
      bool ok = true;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        o[f] = a.dt * (-o[f]) + P[f];
        ok = ok && finite(o[f]);
        ty[f] = th[f];
        tx[r][f] = tu[f];
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        py[j] = ph[j];
        px[r][j] = pu[j];
      }
      if (w.out && y < g.ny) {
        if (ok) {
#pragma unroll
          for (int f = 0; f < 4; ++f) a.qn[f * n + i] = o[f];
        } else {
          wave_full(g, a, x, y, w.z);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < NY; ++r) {
      cc[r] = cn[r];
#pragma unroll
      for (int f = 0; f < 4; ++f) cur[r][f] = nxt[r][f];
    }
  }
}

// ---- Euler step -----------------------------------------------------------------

// A state and what the fluxes take from it.  u, v, w carry NaN where a velocity or
// the pressure is not finite (the array form multiplies each by the zero components
// of a normal), so such a cell and its neighbours come out NaN and take the full form.
template <class R> struct Gas {
  R q[5];    // rho, momentum, E
  R vel[3];
  R p, a;
};

// zero or far enough from the ends of the range for Volume::quot
__device__ __forceinline__ bool moderate(double x) {
  const unsigned h = unsigned(__double2hiint(x)) & 0x7fffffffu;
  return h - 0x26f00000u < 0x32000000u || x == 0.0;  // 2^-400 to 2^400
}
__device__ __forceinline__ bool moderate(float x) {
  const float b = fabsf(x);
  return (b >= 0x1p-60f && b <= 0x1p60f) || b == 0.f;
}

// prim() of the array kernel: four divisions by rho, as one reciprocal and products
// corrected to the rounded quotient (Volume).
template <class R> __device__ __forceinline__ void derive(Gas<R>& s, R gamma) {
  const R rho = s.q[0], mx = s.q[1], my = s.q[2], mz = s.q[3];
  const Volume<R> V{rho, R(1) / rho};
  const bool ok = moderate(rho) && rho != R(0);
  R u, v, w;
  if (ok && moderate(mx) && moderate(my) && moderate(mz)) {
    u = V.quot(mx); v = V.quot(my); w = V.quot(mz);
  } else {
    u = mx / rho; v = my / rho; w = mz / rho;
  }
  const R ke = R(0.5) * ((mx * u + my * v) + mz * w);
  s.p = (gamma - R(1)) * (s.q[4] - ke);
  const R gp = gamma * s.p;
  s.a = sqrt(ok && moderate(gp) ? V.quot(gp) : gp / rho);
  const R taint = ((u * R(0) + v * R(0)) + w * R(0)) + s.p * R(0);
  s.vel[0] = u + taint;
  s.vel[1] = v + taint;
  s.vel[2] = w + taint;
}

// Reflection in a wall normal to D; NaN where the array form's 2 m_D overflows.
template <int D, class R> __device__ __forceinline__ void mirror(Gas<R>& s) {
  s.vel[D] = (R(2) * s.q[1 + D]) * R(0) - s.vel[D];
  s.q[1 + D] = -s.q[1 + D];
}

// Flux through a face normal to D from L to H.  The array form evaluates it once per
// side with opposite normals, which gives the same magnitudes.
template <int D, class R> __device__ __forceinline__ void rusanov(const Gas<R>& L, const Gas<R>& H, R F[5]) {
  const R ul = L.vel[D], uh = H.vel[D];
  const R lm = fmax(fabs(ul) + L.a, fabs(uh) + H.a);
  const R hl = R(0.5) * lm;
  F[0] = R(0.5) * (L.q[0] * ul + H.q[0] * uh) - hl * (H.q[0] - L.q[0]);
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    R l = L.q[1 + e] * ul, h = H.q[1 + e] * uh;
    if (e == D) {
      l = l + L.p;
      h = h + H.p;
    }
    F[1 + e] = R(0.5) * (l + h) - hl * (H.q[1 + e] - L.q[1 + e]);
  }
  F[4] = R(0.5) * ((L.q[4] + L.p) * ul + (H.q[4] + H.p) * uh) - hl * (H.q[4] - L.q[4]);
}

template <class R> struct EulerArgs {
  const R* __restrict__ U;
  R* __restrict__ Un;
  R gamma;
  double dx, dy, dz, cfl, t_end;
  const EulerClock* clock;
  long long step;
};

// One cell of euler_plain_step_k (euler_plain.cu).
template <class R> __device__ __noinline__ void euler_full(const Box<R>& g, const EulerArgs<R>& a, R dt, int x, int y, int z) {
  const int64_t n = int64_t(g.nx) * g.plane;
  const Cell c{x, y, z};
  const int64_t i = id_of(g, c);
  auto prim = [&](const R q[5], R s[5]) {
    s[0] = q[1] / q[0]; s[1] = q[2] / q[0]; s[2] = q[3] / q[0];
    const R ke = R(0.5) * ((q[1] * s[0] + q[2] * s[1]) + q[3] * s[2]);
    s[3] = (a.gamma - R(1)) * (q[4] - ke);
    s[4] = sqrt(a.gamma * s[3] / q[0]);
  };
  R P[5], sP[5], acc[5];
  for (int k = 0; k < 5; ++k) {
    P[k] = a.U[k * n + i];
    acc[k] = R(0);
  }
  prim(P, sP);
  for (int f = 0; f < 6; ++f) {
    const R nx = outward<R>(f, 0), ny = outward<R>(f, 1), nz = outward<R>(f, 2), A = area_of(g, c, f);
    const int64_t j = id_of(g, beyond(g, c, f));
    R N[5], sN[5], F[5];
    for (int k = 0; k < 5; ++k) N[k] = a.U[k * n + j];
    if (j == i && f < 4) {
      const R two_mn = R(2) * ((P[1] * nx + P[2] * ny) + P[3] * nz);
      N[1] = P[1] - two_mn * nx;
      N[2] = P[2] - two_mn * ny;
      N[3] = P[3] - two_mn * nz;
    }
    prim(N, sN);
    const R uP = (sP[0] * nx + sP[1] * ny) + sP[2] * nz, uN = (sN[0] * nx + sN[1] * ny) + sN[2] * nz;
    const R hl = R(0.5) * fmax(fabs(uP) + sP[4], fabs(uN) + sN[4]);
    const R m[3] = {nx, ny, nz};
    F[0] = R(0.5) * (P[0] * uP + N[0] * uN) - hl * (N[0] - P[0]);
    for (int e = 0; e < 3; ++e)
      F[1 + e] = R(0.5) * ((P[1 + e] * uP + sP[3] * m[e]) + (N[1 + e] * uN + sN[3] * m[e])) - hl * (N[1 + e] - P[1 + e]);
    F[4] = R(0.5) * ((P[4] + sP[3]) * uP + (N[4] + sN[3]) * uN) - hl * (N[4] - P[4]);
    for (int k = 0; k < 5; ++k) acc[k] = acc[k] + F[k] * A;
  }
  for (int k = 0; k < 5; ++k) a.Un[k * n + i] = dt * (-(acc[k] / g.volume(i))) + P[k];
}

// euler_plain_step_k without face arrays: a cell's velocities, pressure and sound
// speed are derived once for its x and z faces and once per y neighbour (three times
// instead of seven), x and z faces are evaluated once, and no geometry is read but the
// edge lengths (31 values per cell in the array form).  FP64 step with its reduction
// (12 us) at 64^3 65.7 -> 35.0 us, 128^3 330 -> 162; FP32 there 48 -> 25, 188 -> 98.
// Bound by the chains of divisions and roots at 12 warps per SM (150 registers; 16 warps
// at 128 spill: the same time).
template <class R>
__global__ void __launch_bounds__(kThreads) box_euler_k(const __grid_constant__ Box<R> g, const __grid_constant__ EulerArgs<R> a) {
  const EulerClock* ck = a.clock;
  const int ts = int(a.step & 1), ls = int(a.step % 3);
  if (ck->finished[ts]) return;
  const double lam[3] = {bits_to_double(ck->lam[ls][0]), bits_to_double(ck->lam[ls][1]), bits_to_double(ck->lam[ls][2])};
  bool last;
  const R dt = R(euler_dt(lam, a.dx, a.dy, a.dz, a.cfl, ck->t[ts], a.t_end, &last));
  March<1, 1, 1> w;
  if (!w.start(g)) return;
  const int64_t pl = g.plane, n = pl * g.nx;
  auto load = [&](int x, int row) {
    Gas<R> s;
    const R* q = a.U + x * pl + w.off[1 + row];
#pragma unroll
    for (int k = 0; k < 5; ++k) s.q[k] = q[k * n];
    derive(s, a.gamma);
    return s;
  };
  const double hy = g.hy[w.y0], hz = g.hz[w.z];
  const R Ax = R(hy * hz);
  Gas<R> P = load(w.x0, 0);
  R fx[5];
  rusanov<0>(w.x0 > 0 ? load(w.x0 - 1, 0) : P, P, fx);
  for (int x = w.x0; x < w.x1; ++x) {
    const double hx = g.hx[x];
    const R Ay = R(hx * hz), Az = R(hx * hy);
    R acc[5], F[5];
    {
      Gas<R> L;
#pragma unroll
      for (int k = 0; k < 5; ++k) L.q[k] = __shfl_up_sync(kWarp, P.q[k], 1);
#pragma unroll
      for (int k = 0; k < 3; ++k) L.vel[k] = __shfl_up_sync(kWarp, P.vel[k], 1);
      L.p = __shfl_up_sync(kWarp, P.p, 1);
      L.a = __shfl_up_sync(kWarp, P.a, 1);
      if (w.zlo) {
        L = P;
        mirror<2>(L);
      }
      rusanov<2>(L, P, F);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] = R(0) - F[k] * Az;
#pragma unroll
      for (int k = 0; k < 5; ++k) F[k] = __shfl_down_sync(kWarp, F[k], 1);
      if (w.zhi) {
        L = P;
        mirror<2>(L);
        rusanov<2>(P, L, F);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] = acc[k] + F[k] * Az;
    }
    {
      Gas<R> Y = load(x, -1);
      if (w.y0 == 0) mirror<1>(Y);
      rusanov<1>(Y, P, F);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] = acc[k] - F[k] * Ay;
    }
    {
      Gas<R> Y = load(x, 1);
      if (w.y0 == g.ny - 1) mirror<1>(Y);
      rusanov<1>(P, Y, F);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] = acc[k] + F[k] * Ay;
    }
    const Gas<R> N = x < g.nx - 1 ? load(x + 1, 0) : P;
    rusanov<0>(P, N, F);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      acc[k] = (acc[k] - fx[k] * Ax) + F[k] * Ax;
      fx[k] = F[k];
    }
    const int64_t i = x * pl + w.off[1];
    const R vol = g.volume(i);
    const Volume<R> V{vol, g.vol ? R(1) / vol : g.rv};
    V.template divide<5>(acc);
    bool fine = true;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      acc[k] = dt * (-acc[k]) + P.q[k];
      fine = fine && finite(acc[k]);
    }
    if (w.out) {
      if (fine) {
#pragma unroll
        for (int k = 0; k < 5; ++k) a.Un[k * n + i] = acc[k];
      } else {
        euler_full(g, a, dt, x, w.y0, w.z);
      }
    }
    P = N;
  }
}

// ---- tables -------------------------------------------------------------------

// Volume of a cell, the sum of cell_geometry() (geometry_cell.hpp): the face
// centres' coordinates along the normals (g, entry i of an axis: its i-th grid
// plane) times the areas, in slot order.
template <class R>
__global__ void __launch_bounds__(kThreads) box_volume_k(int nx, int ny, int nz, const double* __restrict__ hx,
                                                         const double* __restrict__ hy, const double* __restrict__ hz,
                                                         const double* __restrict__ gx, const double* __restrict__ gy,
                                                         const double* __restrict__ gz, R* __restrict__ vol,
                                                         int* __restrict__ differs) {
  auto volume = [&](int x, int y, int z) {
    const double axy = hx[x] * hy[y], axz = hx[x] * hz[z], ayz = hy[y] * hz[z];
    double v = 0.0;
    v = v + (-gz[z]) * axy;
    v = v + gz[z + 1] * axy;
    v = v + (-gy[y]) * axz;
    v = v + gy[y + 1] * axz;
    v = v + (-gx[x]) * ayz;
    v = v + gx[x + 1] * ayz;
    return R(v / 3.0);
  };
  const R first = volume(0, 0, 0);
  const int64_t n = int64_t(nx) * ny * nz;
  bool other = false;
  for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += int64_t(gridDim.x) * kThreads) {
    const int x = int(i / (int64_t(ny) * nz)), r = int(i - int64_t(x) * ny * nz), y = r / nz, z = r - y * nz;
    const R v = volume(x, y, z);
    vol[i] = v;
    other = other || v != first;
  }
  if (other) atomicOr(differs, 1);
}

// A marching kernel, the CTAs of it that one SM holds, and its place among the marches.
struct MarchPlan {
  int resident, id;
};
template <class K> struct Form {
  K kern;
  MarchPlan plan;
};
int next_march() {
  static std::atomic<int> next{0};
  return next++;
}
template <auto kern> Form<decltype(kern)> form(const cfdb_ctx* ctx) {
  static const int id = next_march();
  static std::atomic<int> held[kMaxDevices] = {};
  const bool known = ctx->device >= 0 && ctx->device < kMaxDevices;
  int r = known ? held[ctx->device].load(std::memory_order_relaxed) : 0;
  if (r == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kern, kThreads, 0) != cudaSuccess) cudaGetLastError();
    r = std::max(r, 1);
    if (known) held[ctx->device].store(r, std::memory_order_relaxed);
  }
  return {kern, {r, id}};
}

// Chunks of x.  Fewer are less work, as each starts with 2 + HZ / 2 planes' worth of
// loads and faces that its neighbour has too, but they have to fill the SMs evenly.
// With w warps on an SM a plane costs 8 + w (8 for latency); after a first wave the
// CTAs end at different times, so the last one counts for three quarters as a wave
// and for one as its share of one.  The least sum is within 2 % of the best of 1 to 50
// chunks over 10 meshes x 5 operators; 32 warps per SM whatever the kernel held had
// lost 9 % (FP64 gradient at 200^3: 123 us in 501 CTAs on 444 places, now 75).
// A mesh that does not fill the SMs once, even with a plane per chunk, is all latency:
// there a plane costs 16 + w and a chunk's start one plane, and chunks of one plane
// count too (us with at least two planes and now: FP32 gradient 16^3 2.4 and 2.1,
// 512x1x1 2.4 and 2.2, FP64 stabilisation 32x24x20 3.7 and 2.9).
unsigned march_chunks(const cfdb_ctx* ctx, const cfdb_mesh* m, int HZ, int resident, int64_t tiles) {
  constexpr int per = kThreads / 32;
  const int64_t sms = std::max(1, ctx->num_sms), places = sms * resident, nx = m->nx;
  const bool small = (tiles * nx + per - 1) / per <= places;
  const int64_t most = small ? nx : std::max<int64_t>(1, std::min<int64_t>(nx / 2, 8 * places * per / tiles));
  const double latency = small ? 16 : 8, start = (small ? 1 : 2) + 0.5 * HZ, wave = latency + resident * per;
  double least = 0;
  int64_t chunks = 1;
  for (int64_t c = 1; c <= most; c += small ? 1 : std::max<int64_t>(1, c / 32)) {
    const int64_t ctas = (tiles * c + per - 1) / per, full = ctas / places, last = ctas % places;
    double waves = double(full) * wave;
    if (last) {
      const double own = latency + double((last + sms - 1) / sms * per);
      waves += full ? 0.75 * own + 0.25 * wave * double(last) / double(places) : own;
    }
    const double planes = small ? double((nx + c - 1) / c) : double(nx) / double(c);
    const double cost = (waves + 0.05 * wave) * (planes + start);
    if (c == 1 || cost < least) {
      least = cost;
      chunks = c;
    }
  }
  return unsigned(chunks);
}

// Warps of a march over `groups` row groups: tiles of 32 - 2 HZ lanes along (group, z),
// x cut into chunks.  The chunk count stays on the mesh (finding it had cost the host
// up to 0.6 us of every call).
void march_grid(const cfdb_ctx* ctx, cfdb_mesh* m, int HZ, MarchPlan plan, unsigned* tiles, unsigned* chunks,
                unsigned* blocks, int64_t groups) {
  *tiles = unsigned((groups * m->nz + 32 - 2 * HZ - 1) / (32 - 2 * HZ));
  std::atomic<uint32_t>* kept = plan.id < kMarches ? &m->march_chunks[plan.id] : nullptr;
  *chunks = kept ? kept->load(std::memory_order_relaxed) : 0;
  if (*chunks == 0) {
    *chunks = march_chunks(ctx, m, HZ, plan.resident, *tiles);
    if (kept) kept->store(*chunks, std::memory_order_relaxed);
  }
  constexpr int per = kThreads / 32;
  *blocks = unsigned((int64_t(*tiles) * *chunks + per - 1) / per);
}

// Kernel arguments for NY rows per thread and HZ halo lanes; *blocks = the grid.
template <class R> Box<R> box_of(const cfdb_ctx* ctx, cfdb_mesh* m, int NY, int HZ, MarchPlan plan, unsigned* blocks) {
  const BoxGeomDev& b = m->box[sizeof(R) == 8 ? 1 : 0];
  Box<R> g;
  g.nx = int(m->nx); g.ny = int(m->ny); g.nz = int(m->nz);
  g.plane = unsigned(m->ny * m->nz);
  g.groups = int((m->ny + NY - 1) / NY);
  march_grid(ctx, m, HZ, plan, &g.tiles, &g.chunks, blocks, g.groups);
  g.hx = b.h[0]; g.hy = b.h[1]; g.hz = b.h[2];
  auto t = [](const void* p) { return static_cast<const R*>(p); };
  g.ax = t(b.alpha[0]); g.ay = t(b.alpha[1]); g.az = t(b.alpha[2]);
  g.lmx = t(b.len[0]); g.lpx = t(b.len[1]); g.lmy = t(b.len[2]); g.lpy = t(b.len[3]); g.lmz = t(b.len[4]); g.lpz = t(b.len[5]);
  g.vol = t(b.vol);
  g.v = R(b.v);
  g.rv = R(1) / g.v;
  g.limit = R(b.limit);
  for (int d = 0; d < 3; ++d) {
    g.A[d] = R(b.uA[d]);
    g.al[d] = R(b.ual[d]);
    g.lm[d] = R(b.ulm[d]);
    g.lp[d] = R(b.ulp[d]);
  }
  return g;
}

// Rows per thread: two share the face between them (200^3 FP32: gradient 33
// against 40 us, stabilisation 80 against 97), once the mesh gives every SM its
// warps; in double the registers of a second row cost more warps than it saves
// (100 x 90 x 96: stabilisation 33 against 37 us, acoustic step 21 against 27).
template <class R> int rows_per_thread(const cfdb_ctx* ctx, const cfdb_mesh* m) {
  return sizeof(R) == 4 && m->n >= int64_t(ctx->num_sms) * 8192 ? 2 : 1;
}

template <class R>
int build_box(cfdb_mesh* m, BoxGeomDev& b) {
  cfdb_ctx* ctx = m->ctx;
  AxisTables t[3];
  const double limit = axis_tables(m->nx, m->ny, m->nz, m->dx, m->dy, m->dz, sizeof(R) == 8, t);
  b.state = 2;
  if (!(limit >= 0)) return CFDB_OK;  // not reducible: the array kernels serve it
  // one block: the double tables (edge lengths, face coordinates), then the
  // tables in the storage type
  std::vector<char> host;
  auto put = [&](const std::vector<double>& v, bool as_double) {
    const size_t at = host.size();
    const size_t es = as_double ? sizeof(double) : sizeof(R);
    host.resize(at + (v.size() * es + 15) / 16 * 16);
    for (size_t k = 0; k < v.size(); ++k) {
      if (as_double) reinterpret_cast<double*>(host.data() + at)[k] = v[k];
      else reinterpret_cast<R*>(host.data() + at)[k] = R(v[k]);
    }
    return at;
  };
  size_t oh[3], og[3], oa[3], ol[6];
  for (int d = 0; d < 3; ++d) {
    oh[d] = put(t[d].h, true);
    og[d] = put(t[d].g, true);
    oa[d] = put(t[d].alpha, false);
    ol[2 * d] = put(t[d].len_lo, false);
    ol[2 * d + 1] = put(t[d].len_hi, false);
  }
  const size_t flag = host.size();
  host.resize(flag + 16, 0);
  void *tab = nullptr, *vol = nullptr;
  if (int rc = cfdb_dev_alloc(ctx, int64_t(host.size()), &tab)) return rc;
  if (int rc = cfdb_dev_alloc(ctx, int64_t(sizeof(R)) * m->n, &vol)) {
    cfdb_dev_free(ctx, tab);
    return rc;
  }
  char* base = static_cast<char*>(tab);
  for (int d = 0; d < 3; ++d) {
    b.h[d] = reinterpret_cast<double*>(base + oh[d]);
    b.alpha[d] = base + oa[d];
    b.len[2 * d] = base + ol[2 * d];
    b.len[2 * d + 1] = base + ol[2 * d + 1];
  }
  auto g = [&](int d) { return reinterpret_cast<double*>(base + og[d]); };
  int* differs = reinterpret_cast<int*>(base + flag);
  struct { int differs; R first; } back{1, R(0)};
  cudaError_t e = cudaMemcpyAsync(tab, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) {
    box_volume_k<R><<<grid_for(ctx, m->n, kThreads), kThreads, 0, ctx->stream>>>(
        int(m->nx), int(m->ny), int(m->nz), b.h[0], b.h[1], b.h[2], g(0), g(1), g(2), static_cast<R*>(vol), differs);
    ++ctx->launches;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&back.differs, differs, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&back.first, vol, sizeof(R), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    cfdb_dev_free(ctx, tab);
    cfdb_dev_free(ctx, vol);
    return cfdb_cuda_fail(ctx, e, "structured-mesh tables");
  }
  b.tab = tab;
  b.v = double(back.first);
  if (back.differs) {
    b.vol = vol;
  } else {
    cfdb_dev_free(ctx, vol);
  }
  b.limit = limit;
  b.state = 1;
  // one value per direction?  (products round monotonically: the extremes decide)
  auto range = [](const std::vector<double>& v, double lim[2]) {
    lim[0] = *std::min_element(v.begin(), v.end());
    lim[1] = *std::max_element(v.begin(), v.end());
  };
  double h[3][2];
  for (int d = 0; d < 3; ++d) range(t[d].h, h[d]);
  b.uni = !back.differs;
  for (int d = 0; d < 3; ++d) {
    const int e = d == 0 ? 1 : 0, f = d == 2 ? 1 : 2;
    b.uA[d] = double(R(h[e][0] * h[f][0]));
    b.uni = b.uni && R(h[e][0] * h[f][0]) == R(h[e][1] * h[f][1]);
    auto one = [&](const double* p, size_t count, double* out) {
      *out = count ? double(R(p[0])) : 1.0;
      for (size_t k = 0; k < count; ++k) b.uni = b.uni && R(p[k]) == R(p[0]);
    };
    one(t[d].alpha.data() + 1, t[d].alpha.size() - 2, &b.ual[d]);  // interior faces; a wall face multiplies zero
    one(t[d].len_lo.data(), t[d].len_lo.size(), &b.ulm[d]);
    one(t[d].len_hi.data(), t[d].len_hi.size(), &b.ulp[d]);
  }
  return CFDB_OK;
}

template <class R> Vert<R> vert_of(const cfdb_mesh* m) {
  const FaceGeomDev& b = m->faces[sizeof(R) == 8 ? 1 : 0];
  Vert<R> g;
  g.nx = int(m->nx); g.ny = int(m->ny); g.nz = int(m->nz);
  g.plane = unsigned(m->ny * m->nz);
  g.groups = g.ny;
  g.tiles = g.chunks = 0;  // of a march
  for (int a = 0; a < 3; ++a) {
    for (int d = 0; d < 3; ++d) g.nrm[a][d] = static_cast<const R*>(b.normal[a]) + d * b.count[a];
    g.area[a] = static_cast<const R*>(b.area[a]);
    g.alpha[a] = static_cast<const R*>(b.alpha[a]);
  }
  for (int f = 0; f < 6; ++f) g.len[f] = static_cast<const R*>(b.len) + f * m->n;
  g.vol = static_cast<const R*>(b.vol);
  return g;
}

}  // namespace

int cfdb_mesh_need_box(cfdb_mesh* m, int dtype, bool* usable) {
  BoxGeomDev& b = m->box[dtype == CFDB_F64 ? 1 : 0];
  *usable = false;
  if (!m->uniform) return CFDB_OK;
  if (b.state == 0) {
    CFDB_CUDA(m->ctx, cudaSetDevice(m->ctx->device));
    const int rc = dtype == CFDB_F64 ? build_box<double>(m, b) : build_box<float>(m, b);
    if (rc) {
      b = BoxGeomDev();
      return rc;
    }
  }
  *usable = b.state == 1;
  return CFDB_OK;
}

// The kernel of a mesh: one value per direction and all directions, all
// directions, or neither (the heat step takes all); NY = 2 rows per thread in FP32 only.
template <class R, int OP, int NY> auto sum_kernel(const cfdb_ctx* ctx, bool uni, int mask) {
  if constexpr (OP != OP_HEAT)
    if (mask != 7) return form<box_sum_k<R, OP, NY, false, false>>(ctx);
  return uni ? form<box_sum_k<R, OP, NY, true, true>>(ctx) : form<box_sum_k<R, OP, NY, false, true>>(ctx);
}
template <class R, int NY> auto stab_kernel(const cfdb_ctx* ctx, bool uni, int mask) {
  if (mask != 7) return form<box_stab_k<R, NY, false, false>>(ctx);
  return uni ? form<box_stab_k<R, NY, true, true>>(ctx) : form<box_stab_k<R, NY, false, true>>(ctx);
}

template <class R, int OP> int launch_sum(cfdb_ctx* ctx, cfdb_mesh* m, const void* phi, void* out, int mask, double k, double dt) {
  constexpr int NY = sizeof(R) == 4 ? 2 : 1;
  const bool uni = m->box[sizeof(R) == 8 ? 1 : 0].uni;
  const int rows = rows_per_thread<R>(ctx, m);
  unsigned blocks = 0;
  const auto f = rows == 1 ? sum_kernel<R, OP, 1>(ctx, uni, mask) : sum_kernel<R, OP, NY>(ctx, uni, mask);
  const Box<R> g = box_of<R>(ctx, m, rows, 1, f.plan, &blocks);
  f.kern<<<blocks, kThreads, 0, ctx->stream>>>(g, static_cast<const R*>(phi), static_cast<R*>(out), mask, R(k), R(dt));
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

template <class R> int launch_stab(cfdb_ctx* ctx, cfdb_mesh* m, const void* phi, void* out, int mask) {
  constexpr int NY = sizeof(R) == 4 ? 2 : 1;
  const bool uni = m->box[sizeof(R) == 8 ? 1 : 0].uni;
  const int rows = rows_per_thread<R>(ctx, m);
  unsigned blocks = 0;
  const auto f = rows == 1 ? stab_kernel<R, 1>(ctx, uni, mask) : stab_kernel<R, NY>(ctx, uni, mask);
  const Box<R> g = box_of<R>(ctx, m, rows, 2, f.plan, &blocks);
  f.kern<<<blocks, kThreads, 0, ctx->stream>>>(g, static_cast<const R*>(phi), static_cast<R*>(out), mask);
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

template <class R, int NY> auto wave_kernel(const cfdb_ctx* ctx, bool uni, bool c) {
  return uni ? (c ? form<box_wave_k<R, NY, true, true>>(ctx) : form<box_wave_k<R, NY, true, false>>(ctx))
             : (c ? form<box_wave_k<R, NY, false, true>>(ctx) : form<box_wave_k<R, NY, false, false>>(ctx));
}
template <class R>
int launch_wave(cfdb_ctx* ctx, cfdb_mesh* m, const void* q, void* qn, const void* c, double cconst, int mode, double dt) {
  constexpr int NY = sizeof(R) == 4 ? 2 : 1;
  const bool uni = m->box[sizeof(R) == 8 ? 1 : 0].uni;
  const int rows = rows_per_thread<R>(ctx, m);
  unsigned blocks = 0;
  const auto f = rows == 1 ? wave_kernel<R, 1>(ctx, uni, c != nullptr) : wave_kernel<R, NY>(ctx, uni, c != nullptr);
  const Box<R> g = box_of<R>(ctx, m, rows, 1, f.plan, &blocks);
  const WaveArgs<R> a{static_cast<const R*>(q), static_cast<R*>(qn), static_cast<const R*>(c), R(cconst), R(dt), mode};
  f.kern<<<blocks, kThreads, 0, ctx->stream>>>(g, a);
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

int box_grad(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_sum<double, OP_GRAD>(ctx, m, phi, out, mask, 0, 0)
                           : launch_sum<float, OP_GRAD>(ctx, m, phi, out, mask, 0, 0);
}

int box_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_sum<double, OP_LAPL>(ctx, m, phi, out, mask, 0, 0)
                           : launch_sum<float, OP_LAPL>(ctx, m, phi, out, mask, 0, 0);
}

int box_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt) {
  return dtype == CFDB_F64 ? launch_sum<double, OP_HEAT>(ctx, m, T, Tn, 7, k, dt) : launch_sum<float, OP_HEAT>(ctx, m, T, Tn, 7, k, dt);
}

int box_stab(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_stab<double>(ctx, m, phi, out, mask) : launch_stab<float>(ctx, m, phi, out, mask);
}

int box_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c, double cconst, int mode,
                  double dt) {
  return dtype == CFDB_F64 ? launch_wave<double>(ctx, m, q, qn, c, cconst, mode, dt)
                           : launch_wave<float>(ctx, m, q, qn, c, cconst, mode, dt);
}

template <class R> int launch_euler(cfdb_euler* e, const void* U, void* Un, int64_t step) {
  cfdb_ctx* ctx = e->ctx;
  unsigned blocks = 0;
  const auto f = form<box_euler_k<R>>(ctx);
  const Box<R> g = box_of<R>(ctx, e->mesh, 1, 1, f.plan, &blocks);
  const EulerArgs<R> a{static_cast<const R*>(U), static_cast<R*>(Un), R(e->gamma), e->mesh->dx, e->mesh->dy, e->mesh->dz,
                       e->cfl, e->t_end, e->clock, (long long)step};
  f.kern<<<blocks, kThreads, 0, ctx->stream>>>(g, a);
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

int box_euler_step(cfdb_euler* e, const void* U, void* Un, int64_t step) {
  return e->dtype == CFDB_F64 ? launch_euler<double>(e, U, Un, step) : launch_euler<float>(e, U, Un, step);
}

template <class R, int OP, int OUT>
int launch_vert_sum(cfdb_ctx* ctx, cfdb_mesh* m, const void* phi, void* out, int mask, double k, double dt) {
  vert_cell_k<R, OP, OUT><<<unsigned((m->n + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(
      vert_of<R>(m), static_cast<const R*>(phi), static_cast<R*>(out), mask, R(k), R(dt));
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

int vert_grad(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_vert_sum<double, OP_GRAD, OUT_SUM>(ctx, m, phi, out, mask, 0, 0)
                           : launch_vert_sum<float, OP_GRAD, OUT_SUM>(ctx, m, phi, out, mask, 0, 0);
}

int vert_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_vert_sum<double, OP_LAPL, OUT_SUM>(ctx, m, phi, out, mask, 0, 0)
                           : launch_vert_sum<float, OP_LAPL, OUT_SUM>(ctx, m, phi, out, mask, 0, 0);
}

int vert_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt) {
  return dtype == CFDB_F64 ? launch_vert_sum<double, OP_HEAT, OUT_SUM>(ctx, m, T, Tn, 7, k, dt)
                           : launch_vert_sum<float, OP_HEAT, OUT_SUM>(ctx, m, T, Tn, 7, k, dt);
}

template <class R> int launch_vert_stab(cfdb_ctx* ctx, cfdb_mesh* m, const void* phi, void* out, int mask) {
  const FaceGeomDev& b = m->faces[sizeof(R) == 8 ? 1 : 0];
  if (int rc = launch_vert_sum<R, OP_GRAD, OUT_GRADIENT>(ctx, m, phi, b.grad, 7, 0, 0)) return rc;
  unsigned blocks = 0;
  const auto f = form<vert_stab_k<R>>(ctx);
  Vert<R> g = vert_of<R>(m);
  march_grid(ctx, m, 1, f.plan, &g.tiles, &g.chunks, &blocks, g.groups);
  f.kern<<<blocks, kThreads, 0, ctx->stream>>>(g, static_cast<const R*>(phi), static_cast<const R*>(b.grad),
                                                  static_cast<R*>(out), mask);
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

int vert_stab(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return dtype == CFDB_F64 ? launch_vert_stab<double>(ctx, m, phi, out, mask) : launch_vert_stab<float>(ctx, m, phi, out, mask);
}
