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
// Layout: a thread owns one (y, z) column and NX consecutive x planes, all of
// whose loads are issued before the first result is needed; threads of a warp
// are consecutive in z, x neighbours come from registers and y and z
// neighbours through L1.  Compiled with --fmad=false like plain_ops.cu.
#include <cmath>
#include <limits>

#include "cfdb_internal.hpp"

CFDB_MODULE_ANCHOR

namespace {

constexpr int kThreads = 256;

template <class R> struct Box {
  int nx, ny, nz;
  unsigned plane, chunks;   // ny nz; x chunks of NX planes
  const double *hx, *hy, *hz;   // edge lengths
  const R *ax, *ay, *az;        // alpha of the face below cell i (entry i), 0 .. n
  const R *lmx, *lpx, *lmy, *lpy, *lmz, *lpz;  // |x_f - x_P| of the - and + faces
  const R* vol;                 // cell volumes, or null: v for every cell
  R v;
  R limit;                      // magnitudes up to this overflow in no intermediate
  __device__ R volume(int64_t i) const { return vol ? vol[i] : v; }
};

template <class R> __device__ __forceinline__ bool finite(R v) { return fabs(v) <= std::numeric_limits<R>::max(); }

// The column and the x chunk of a thread.
struct Where {
  int x0, y, z;
  int64_t i0;      // cell (x0, y, z)
  bool ok;
};
template <int NX, class R> __device__ __forceinline__ Where where(const Box<R>& g) {
  const unsigned t = blockIdx.x * kThreads + threadIdx.x;
  const unsigned chunk = t / g.plane, col = t - chunk * g.plane;
  Where w;
  w.ok = chunk < g.chunks;
  w.x0 = int(chunk) * NX;
  w.y = int(col / unsigned(g.nz));
  w.z = int(col) - w.y * g.nz;
  w.i0 = int64_t(w.x0) * g.plane + col;
  return w;
}

// GradVar (grad_k): sum over the masked directions of (sum_f itp n_d A) / V.
template <class R, int NX>
__global__ void __launch_bounds__(kThreads) box_grad_k(Box<R> g, const R* __restrict__ phi, R* __restrict__ out, int mask) {
  const Where w = where<NX>(g);
  if (!w.ok) return;
  const R* p = phi + w.i0;
  const int64_t pl = g.plane;
  const int dym = w.y > 0 ? -g.nz : 0, dyp = w.y < g.ny - 1 ? g.nz : 0;
  const int dzm = w.z > 0 ? -1 : 0, dzp = w.z < g.nz - 1 ? 1 : 0;
  R c[NX + 2], ym[NX], yp[NX], zm[NX], zp[NX], V[NX];
  int xs[NX];
  c[0] = w.x0 > 0 ? p[-pl] : p[0];
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    xs[j] = min(w.x0 + j, g.nx - 1);
    const R* q = p + (xs[j] - w.x0) * pl;
    c[j + 1] = q[0];
    ym[j] = q[dym];
    yp[j] = q[dyp];
    zm[j] = q[dzm];
    zp[j] = q[dzp];
    V[j] = g.volume(w.i0 + (xs[j] - w.x0) * pl);
  }
  c[NX + 1] = p[(min(w.x0 + NX, g.nx - 1) - w.x0) * pl];
  const double hy = g.hy[w.y], hz = g.hz[w.z];
  const R Ax = R(hy * hz);
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    if (w.x0 + j >= g.nx) return;
    const double hx = g.hx[xs[j]];
    const R Ay = R(hx * hz), Az = R(hx * hy);
    const R P = c[j + 1];
    const R itp[6] = {(P + zm[j]) * R(0.5), (P + zp[j]) * R(0.5), (P + ym[j]) * R(0.5),
                      (P + yp[j]) * R(0.5), (P + c[j]) * R(0.5),  (P + c[j + 2]) * R(0.5)};
    const R A[3] = {Ax, Ay, Az};
    R res = R(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!(mask & (1 << d))) continue;
      const int f = 4 - 2 * d;
      const R acc = (R(0) + (-itp[f]) * A[d]) + itp[f + 1] * A[d];
      res = res + acc / V[j];
    }
    const R sum = ((itp[0] + itp[1]) + (itp[2] + itp[3])) + (itp[4] + itp[5]);
    if (!finite(sum)) {  // a face value times the zero components of its normal, in the other directions' sums
      for (int f = 0; f < 6; ++f)
        if (!finite(itp[f]) && (mask & ~(1 << (2 - f / 2)))) res = sum - sum;  // NaN
    }
    out[w.i0 + j * pl] = res;
  }
}

// Grad2Var (lapl_k): sum over the masked directions of (sum_f (sn_f n_d) A) / V,
// sn_f = (phi_N - phi_P) alpha_f, with the unsigned normal +e_d on both faces.
// HEAT: the heat step dt (k L) + phi of heat_update_k in the same pass.
template <class R, int NX, bool HEAT = false>
__global__ void __launch_bounds__(kThreads) box_lapl_k(Box<R> g, const R* __restrict__ phi, R* __restrict__ out, int mask,
                                                       R k = R(0), R dt = R(0)) {
  const Where w = where<NX>(g);
  if (!w.ok) return;
  const R* p = phi + w.i0;
  const int64_t pl = g.plane;
  const int dym = w.y > 0 ? -g.nz : 0, dyp = w.y < g.ny - 1 ? g.nz : 0;
  const int dzm = w.z > 0 ? -1 : 0, dzp = w.z < g.nz - 1 ? 1 : 0;
  R c[NX + 2], ym[NX], yp[NX], zm[NX], zp[NX], V[NX];
  int xs[NX];
  c[0] = w.x0 > 0 ? p[-pl] : p[0];
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    xs[j] = min(w.x0 + j, g.nx - 1);
    const R* q = p + (xs[j] - w.x0) * pl;
    c[j + 1] = q[0];
    ym[j] = q[dym];
    yp[j] = q[dyp];
    zm[j] = q[dzm];
    zp[j] = q[dzp];
    V[j] = g.volume(w.i0 + (xs[j] - w.x0) * pl);
  }
  c[NX + 1] = p[(min(w.x0 + NX, g.nx - 1) - w.x0) * pl];
  const double hy = g.hy[w.y], hz = g.hz[w.z];
  const R Ax = R(hy * hz);
  const R aym = g.ay[w.y], ayp = g.ay[w.y + 1], azm = g.az[w.z], azp = g.az[w.z + 1];
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    if (w.x0 + j >= g.nx) return;
    const double hx = g.hx[xs[j]];
    const R Ay = R(hx * hz), Az = R(hx * hy);
    const R P = c[j + 1];
    const R sn[6] = {(zm[j] - P) * azm,           (zp[j] - P) * azp, (ym[j] - P) * aym,
                     (yp[j] - P) * ayp,           (c[j] - P) * g.ax[xs[j]], (c[j + 2] - P) * g.ax[xs[j] + 1]};
    const R A[3] = {Ax, Ay, Az};
    R res = R(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!(mask & (1 << d))) continue;
      const int f = 4 - 2 * d;
      const R acc = (R(0) + sn[f] * A[d]) + sn[f + 1] * A[d];
      res = res + acc / V[j];
    }
    const R sum = ((sn[0] + sn[1]) + (sn[2] + sn[3])) + (sn[4] + sn[5]);
    if (!finite(sum)) {  // a face value times the zero components of its normal, in the other directions' sums
      for (int f = 0; f < 6; ++f)
        if (!finite(sn[f]) && (mask & ~(1 << (2 - f / 2)))) res = sum - sum;  // NaN
    }
    if constexpr (HEAT) res = dt * (k * res) + P;
    out[w.i0 + j * pl] = res;
  }
}

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

// One direction of StabVar from the five values along it: b2 b1 P a1 a2 (below
// and above; beyond a wall the wall cell repeats), the face area, the volumes
// of the three cells and the face distances (own - and +, the lower
// neighbour's + and the upper neighbour's -).
template <class R>
__device__ __forceinline__ R grad1(R lo, R P, R hi, R A, R V) {
  return ((R(0) + (-((P + lo) * R(0.5))) * A) + ((P + hi) * R(0.5)) * A) / V;
}
template <class R>
__device__ __forceinline__ R stab1(R b1, R P, R a1, R gP, R gB, R gA, R A, R V, R lm, R lp, R lpB, R lmA) {
  const R um = P + -(lm * gP), up = P + lp * gP;
  const R cm = b1 + lpB * gB, cp = a1 + -(lmA * gA);
  const R sm = R(0.5) * (um - cm), sp = R(0.5) * (up - cp);
  return ((R(0) + sm * A) + sp * A) / V;
}

// StabVar, both stages at once (stab1_k + stab2_k, whose 18 values per cell
// between the stages made 3.5 GB of traffic at 200^3 FP32): along each
// direction the sum needs the gradients of the cell and of its two
// neighbours, which five values give.
template <class R, int NX>
__global__ void __launch_bounds__(kThreads) box_stab_k(Box<R> g, const R* __restrict__ phi, R* __restrict__ out, int mask) {
  const Where w = where<NX>(g);
  if (!w.ok) return;
  const R* p = phi + w.i0;
  const int64_t pl = g.plane;
  const int y = w.y, z = w.z;
  const int dym = y > 0 ? -g.nz : 0, dyp = y < g.ny - 1 ? g.nz : 0;
  const int dym2 = y > 1 ? -2 * g.nz : dym, dyp2 = y < g.ny - 2 ? 2 * g.nz : dyp;
  const int dzm = z > 0 ? -1 : 0, dzp = z < g.nz - 1 ? 1 : 0;
  const int dzm2 = z > 1 ? -2 : dzm, dzp2 = z < g.nz - 2 ? 2 : dzp;
  auto at = [&](int k) { return min(max(w.x0 + k, 0), g.nx - 1) - w.x0; };  // plane k of the chunk, walls repeated
  // values of planes -2 .. NX+1 of the column and -1 .. NX of its four
  // neighbours; `fine`: magnitudes for which no intermediate of the two stages
  // overflows, over every cell the array form touches
  R c[NX + 4], ym[NX + 2], yp[NX + 2], zm[NX + 2], zp[NX + 2];
  R ym2[NX], yp2[NX], zm2[NX], zp2[NX];
  bool fine = true;
  auto look = [&](R v) { fine = fine && fabs(v) <= g.limit; };
#pragma unroll
  for (int k = -2; k < NX + 2; ++k) look(c[k + 2] = p[at(k) * pl]);
#pragma unroll
  for (int k = -1; k < NX + 1; ++k) {
    const R* q = p + at(k) * pl;
    look(ym[k + 1] = q[dym]);
    look(yp[k + 1] = q[dyp]);
    look(zm[k + 1] = q[dzm]);
    look(zp[k + 1] = q[dzp]);
  }
#pragma unroll
  for (int k = 0; k < NX; ++k) {
    const R* q = p + at(k) * pl;
    look(ym2[k] = q[dym2]);
    look(yp2[k] = q[dyp2]);
    look(zm2[k] = q[dzm2]);
    look(zp2[k] = q[dzp2]);
    look(q[dym + dzm]);
    look(q[dym + dzp]);
    look(q[dyp + dzm]);
    look(q[dyp + dzp]);
  }
  const double hy = g.hy[y], hz = g.hz[z];
  const R A0 = R(hy * hz);
  // x gradients of planes -1 .. NX (a wall cell's neighbour is itself)
  R gx[NX + 2];
#pragma unroll
  for (int k = -1; k < NX + 1; ++k) gx[k + 1] = grad1(c[k + 1], c[k + 2], c[k + 3], A0, g.volume(w.i0 + at(k) * pl));
  const int yb = max(y - 1, 0), ya = min(y + 1, g.ny - 1), zb = max(z - 1, 0), za = min(z + 1, g.nz - 1);
  const R lmy = g.lmy[y], lpy = g.lpy[y], lpyB = g.lpy[yb], lmyA = g.lmy[ya];
  const R lmz = g.lmz[z], lpz = g.lpz[z], lpzB = g.lpz[zb], lmzA = g.lmz[za];
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    const int x = w.x0 + j;
    if (x >= g.nx) return;
    const int64_t i = w.i0 + j * pl;
    if (!fine) {
      out[i] = stab_full(g, phi, x, y, z, mask);
      continue;
    }
    const double hx = g.hx[x];
    const R V = g.volume(i);
    const R P = c[j + 2];
    R res = R(0);
    if (mask & 1) {
      const R gP = gx[j + 1];
      const R gB = x == 0 ? gP : gx[j], gA = x == g.nx - 1 ? gP : gx[j + 2];
      res = res + stab1(c[j + 1], P, c[j + 3], gP, gB, gA, A0, V, g.lmx[x], g.lpx[x], g.lpx[max(x - 1, 0)],
                        g.lmx[min(x + 1, g.nx - 1)]);
    }
    if (mask & 2) {
      const R A = R(hx * hz);
      const R gP = grad1(ym[j + 1], P, yp[j + 1], A, V);
      const R gB = y == 0 ? gP : grad1(ym2[j], ym[j + 1], P, A, g.volume(i + dym));
      const R gA = y == g.ny - 1 ? gP : grad1(P, yp[j + 1], yp2[j], A, g.volume(i + dyp));
      res = res + stab1(ym[j + 1], P, yp[j + 1], gP, gB, gA, A, V, lmy, lpy, lpyB, lmyA);
    }
    if (mask & 4) {
      const R A = R(hx * hy);
      const R gP = grad1(zm[j + 1], P, zp[j + 1], A, V);
      const R gB = z == 0 ? gP : grad1(zm2[j], zm[j + 1], P, A, g.volume(i + dzm));
      const R gA = z == g.nz - 1 ? gP : grad1(P, zp[j + 1], zp2[j], A, g.volume(i + dzp));
      res = res + stab1(zm[j + 1], P, zp[j + 1], gP, gB, gA, A, V, lmz, lpz, lpzB, lmzA);
    }
    out[i] = res;
  }
}

// ---- the acoustic step (wave_plain_k) --------------------------------------------

template <class R> struct WaveArgs {
  const R* q;
  R* qn;
  const R* c;  // sound speed field, or null: cconst
  R cconst, dt;
  int mode;
  R limit;     // magnitudes that overflow in no sum of two
};

// One face of slot F between the cell P = (p, u, v, w) and its neighbour N:
// wave_plain_k's flux with the normal S e_D, times the area, added to acc.
template <int F, class R>
__device__ __forceinline__ void wave_face(const R P[4], const R N[4], R c2, R hc, R A, R acc[4]) {
  constexpr int D = 2 - F / 2;
  constexpr bool plus = F & 1;
  const R uP = plus ? P[1 + D] : -P[1 + D], uN = plus ? N[1 + D] : -N[1 + D];
  const R fp = c2 * (R(0.5) * (uP + uN)) - hc * (N[0] - P[0]);
  const R pm = R(0.5) * (P[0] + N[0]);
  acc[0] = acc[0] + fp * A;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const R diff = hc * (N[1 + e] - P[1 + e]);
    const R fu = e == D ? (plus ? pm : -pm) - diff : -diff;
    acc[1 + e] = acc[1 + e] + fu * A;
  }
}

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

// A wall neighbour is the cell with its wall-normal velocity negated: with
// the normal S e_D, u - (2 (S u)) S = -u exactly.
template <class R, int NX, bool CF>
__global__ void __launch_bounds__(kThreads) box_wave_k(Box<R> g, WaveArgs<R> a) {
  const Where w = where<NX>(g);
  if (!w.ok) return;
  const int64_t pl = g.plane, n = int64_t(g.nx) * pl;
  const int y = w.y, z = w.z;
  const bool ylo = y == 0, yhi = y == g.ny - 1, zlo = z == 0, zhi = z == g.nz - 1;
  const int dym = ylo ? 0 : -g.nz, dyp = yhi ? 0 : g.nz, dzm = zlo ? 0 : -1, dzp = zhi ? 0 : 1;
  const R* const q = a.q + w.i0;
  const R* const cf = CF ? a.c + w.i0 : nullptr;
  const double hy = g.hy[y], hz = g.hz[z];
  const R Ax = R(hy * hz);
  R prv[4], cur[4], nxt[4];
#pragma unroll
  for (int f = 0; f < 4; ++f) cur[f] = q[f * n];
#pragma unroll
  for (int f = 0; f < 4; ++f) prv[f] = q[f * n - (w.x0 > 0 ? pl : 0)];
  if (w.x0 == 0) prv[1] = -prv[1];
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    const int x = w.x0 + j;
    if (x >= g.nx) return;
    const bool xhi = x == g.nx - 1;
    const R* const b = q + j * pl;
    const int64_t dxp = xhi ? 0 : pl;
    R ym[4], yp[4], zm[4], zp[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      nxt[f] = b[f * n + dxp];
      ym[f] = b[f * n + dym];
      yp[f] = b[f * n + dyp];
      zm[f] = b[f * n + dzm];
      zp[f] = b[f * n + dzp];
    }
    const R V = g.volume(w.i0 + j * pl);
    if (xhi) nxt[1] = -nxt[1];
    if (ylo) ym[2] = -ym[2];
    if (yhi) yp[2] = -yp[2];
    if (zlo) zm[3] = -zm[3];
    if (zhi) zp[3] = -zp[3];
    bool fine = true;
#pragma unroll
    for (int f = 0; f < 4; ++f)
      fine = fine && fabs(cur[f]) <= a.limit && fabs(prv[f]) <= a.limit && fabs(nxt[f]) <= a.limit &&
             fabs(ym[f]) <= a.limit && fabs(yp[f]) <= a.limit && fabs(zm[f]) <= a.limit && fabs(zp[f]) <= a.limit;
    if (fine) {
      const R cP = CF ? cf[j * pl] : a.cconst;
      const R c2 = cP * cP;
      auto half_speed = [&](int64_t off) {
        if (!CF) return R(0.5) * (a.mode == 0 ? cP : R(0.5) * (cP + cP));
        const R cN = cf[j * pl + off];
        return R(0.5) * (a.mode == 0 ? fmax(cP, cN) : R(0.5) * (cP + cN));
      };
      const double hx = g.hx[x];
      const R Ay = R(hx * hz), Az = R(hx * hy);
      R acc[4] = {R(0), R(0), R(0), R(0)};
      wave_face<0>(cur, zm, c2, half_speed(dzm), Az, acc);
      wave_face<1>(cur, zp, c2, half_speed(dzp), Az, acc);
      wave_face<2>(cur, ym, c2, half_speed(dym), Ay, acc);
      wave_face<3>(cur, yp, c2, half_speed(dyp), Ay, acc);
      wave_face<4>(cur, prv, c2, half_speed(x > 0 ? -pl : 0), Ax, acc);
      wave_face<5>(cur, nxt, c2, half_speed(dxp), Ax, acc);
      R* const o = a.qn + w.i0 + j * pl;
#pragma unroll
      for (int f = 0; f < 4; ++f) o[f * n] = a.dt * (-(acc[f] / V)) + cur[f];
    } else {
      wave_full(g, a, x, y, z);
    }
    // the next plane: an x wall's ghost is never carried on (xhi ends the column)
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      prv[f] = cur[f];
      cur[f] = nxt[f];
    }
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

template <class R> Box<R> box_of(const cfdb_mesh* m, int nx_per_thread) {
  const BoxGeomDev& b = m->box[sizeof(R) == 8 ? 1 : 0];
  Box<R> g;
  g.nx = int(m->nx); g.ny = int(m->ny); g.nz = int(m->nz);
  g.plane = unsigned(m->ny * m->nz);
  g.chunks = unsigned((m->nx + nx_per_thread - 1) / nx_per_thread);
  g.hx = b.h[0]; g.hy = b.h[1]; g.hz = b.h[2];
  auto t = [](const void* p) { return static_cast<const R*>(p); };
  g.ax = t(b.alpha[0]); g.ay = t(b.alpha[1]); g.az = t(b.alpha[2]);
  g.lmx = t(b.len[0]); g.lpx = t(b.len[1]); g.lmy = t(b.len[2]); g.lpy = t(b.len[3]); g.lmz = t(b.len[4]); g.lpz = t(b.len[5]);
  g.vol = t(b.vol);
  g.v = R(b.v);
  g.limit = R(b.limit);
  return g;
}

unsigned grid_of(const cfdb_mesh* m, int nx) {
  const int64_t threads = ((m->nx + nx - 1) / nx) * m->ny * m->nz;
  return unsigned((threads + kThreads - 1) / kThreads);
}

// Fields of a few hundred thousand cells fill the SMs only with one cell per
// thread; larger ones want the loads of several planes in flight.
bool one_cell(const cfdb_ctx* ctx, const cfdb_mesh* m) { return m->n < int64_t(ctx->num_sms) * 4096; }

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
  return CFDB_OK;
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

// f(R(), NX) with the precision and the planes per thread of this mesh
template <class F> int with_form(cfdb_ctx* ctx, const cfdb_mesh* m, int dtype, F f) {
  if (dtype == CFDB_F64) f(double(), one_cell(ctx, m));
  else f(float(), one_cell(ctx, m));
  CFDB_LAUNCHED(ctx);
  return CFDB_OK;
}

int box_grad(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return with_form(ctx, m, dtype, [&](auto r, bool one) {
    using R = decltype(r);
    auto kern = one ? box_grad_k<R, 1> : box_grad_k<R, 4>;
    const int nx = one ? 1 : 4;
    kern<<<grid_of(m, nx), kThreads, 0, ctx->stream>>>(box_of<R>(m, nx), static_cast<const R*>(phi), static_cast<R*>(out), mask);
  });
}

int box_lapl(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return with_form(ctx, m, dtype, [&](auto r, bool one) {
    using R = decltype(r);
    auto kern = one ? box_lapl_k<R, 1> : box_lapl_k<R, 4>;
    const int nx = one ? 1 : 4;
    kern<<<grid_of(m, nx), kThreads, 0, ctx->stream>>>(box_of<R>(m, nx), static_cast<const R*>(phi), static_cast<R*>(out), mask,
                                                       R(0), R(0));
  });
}

int box_heat_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* T, void* Tn, double k, double dt) {
  return with_form(ctx, m, dtype, [&](auto r, bool one) {
    using R = decltype(r);
    auto kern = one ? box_lapl_k<R, 1, true> : box_lapl_k<R, 4, true>;
    const int nx = one ? 1 : 4;
    kern<<<grid_of(m, nx), kThreads, 0, ctx->stream>>>(box_of<R>(m, nx), static_cast<const R*>(T), static_cast<R*>(Tn), 7, R(k), R(dt));
  });
}

int box_stab(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* phi, void* out, int mask) {
  return with_form(ctx, m, dtype, [&](auto r, bool one) {
    using R = decltype(r);
    constexpr int NX = sizeof(R) == 8 ? 2 : 4;
    auto kern = one ? box_stab_k<R, 1> : box_stab_k<R, NX>;
    const int nx = one ? 1 : NX;
    kern<<<grid_of(m, nx), kThreads, 0, ctx->stream>>>(box_of<R>(m, nx), static_cast<const R*>(phi), static_cast<R*>(out), mask);
  });
}

int box_wave_step(cfdb_ctx* ctx, cfdb_mesh* m, int dtype, const void* q, void* qn, const void* c, double cconst, int mode,
                  double dt) {
  return with_form(ctx, m, dtype, [&](auto r, bool one) {
    using R = decltype(r);
    WaveArgs<R> a{static_cast<const R*>(q), static_cast<R*>(qn), static_cast<const R*>(c), R(cconst), R(dt), mode,
                  std::numeric_limits<R>::max() / R(16)};
    auto kern = c ? (one ? box_wave_k<R, 1, true> : box_wave_k<R, 4, true>) : (one ? box_wave_k<R, 1, false> : box_wave_k<R, 4, false>);
    const int nx = one ? 1 : 4;
    kern<<<grid_of(m, nx), kThreads, 0, ctx->stream>>>(box_of<R>(m, nx), a);
  });
}
