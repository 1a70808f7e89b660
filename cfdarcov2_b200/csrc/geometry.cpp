// Host geometry of the hexahedral mesh, following the reference's
// Mesh3D::init_basic_internals / Face3D::compute / Quadrangle3D::compute /
// Mesh3D::compute (src/mesh3d.cpp:43-385).  Built in double with every
// multiply and add separately rounded (compiled with -ffp-contract=off) so the
// FP64 plain kernels see exactly the arrays the CPU oracle restates.  The
// per-cell formulas live in geometry_cell.hpp, shared with the device
// builder (geometry_dev.cu) that gives the same doubles.
//
// Differences from the reference, on purpose:
//  * computed per cell in one pass instead of through shared_ptr object graphs
//    (same formulas and operation order; a shared face is computed by both
//    cells from the same vertex order, so both see identical values);
//  * uniform lattices use the reference formulas with the norm of the two
//    half cross products as face area (the reference's component sum,
//    src/mesh3d.cpp:61, is identical on axis-aligned faces);
//  * vertex meshes default to the exact vector area of each bilinear face,
//    S = (C - A) x (D - B) / 2 (n = S/|S|, A = |S|), and a volume taken about
//    the cell centre: with one-triangle normals and absolute coordinates the
//    reference's volume formula goes negative on strongly jittered cells.
//    CFDB_MESH_COMPAT_AREA restores the reference formulas verbatim;
//  * the unused _n_min_alpha_d arrays (non-orthogonal correction, commented
//    out in include/grad_utils.hpp:117-122) are not built.
#include <algorithm>
#include <cmath>
#include <limits>
#include <new>

#include "cfdb_internal.hpp"
#include "geometry_cell.hpp"

bool cfdb_build_geometry(HostGeom& g, int64_t nx, int64_t ny, int64_t nz, double dx, double dy, double dz,
                         const double* verts, int mode) {
  using namespace cfdb_geom;
  const int64_t n = nx * ny * nz;
  g.nx = nx; g.ny = ny; g.nz = nz; g.n = n;
  try {
    g.normal.assign(18 * n, 0.0); g.normal_alt.assign(18 * n, 0.0);
    g.area.assign(6 * n, 0.0); g.alpha.assign(6 * n, 0.0); g.len.assign(6 * n, 0.0);
    g.volume.assign(n, 0.0); g.center.assign(3 * n, 0.0); g.isb.assign(n, 0.0);
    g.ids.assign(6 * n, 0); g.ibf.assign(6 * n, 0);
  } catch (const std::bad_alloc&) {
    return false;
  }
  const Lattice L{nx, ny, nz, dx, dy, dz, verts};

#pragma omp parallel for schedule(static)
  for (int64_t x = 0; x < nx; ++x)
    for (int64_t y = 0; y < ny; ++y)
      for (int64_t z = 0; z < nz; ++z) {
        const P3 c = L.center(x, y, z);
        const int64_t i = L.id(x, y, z);
        g.center[i] = c.x; g.center[n + i] = c.y; g.center[2 * n + i] = c.z;
      }
  auto center_of = [&](int64_t x, int64_t y, int64_t z) {
    const int64_t j = L.id(x, y, z);
    return P3{g.center[j], g.center[n + j], g.center[2 * n + j]};
  };

#pragma omp parallel for schedule(static)
  for (int64_t x = 0; x < nx; ++x)
    for (int64_t y = 0; y < ny; ++y)
      for (int64_t z = 0; z < nz; ++z) {
        const int64_t i = L.id(x, y, z);
        bool bnd = false;
        auto store = [&](int f, const CellFace& o) {
          const int64_t k6 = int64_t(f) * n + i;
          g.normal[k6] = o.uns.x; g.normal[6 * n + k6] = o.uns.y; g.normal[12 * n + k6] = o.uns.z;
          g.normal_alt[k6] = o.good.x; g.normal_alt[6 * n + k6] = o.good.y; g.normal_alt[12 * n + k6] = o.good.z;
          g.area[k6] = o.area;
          g.alpha[k6] = o.alpha;
          g.len[k6] = o.len;
          g.ids[k6] = o.id;
          g.ibf[k6] = o.ibf;
        };
        const double vol = cell_geometry(L, x, y, z, mode, center_of, store, &bnd);
        g.volume[i] = vol;
        g.isb[i] = bnd ? 1.0 : 0.0;
      }
  return true;
}

// ---- structured meshes as tables per axis ------------------------------------
// With grid planes at X[i] = i h along each axis, cell_geometry() (reference
// mode) sees faces whose corners differ along two axes only, so:
//   normal   the cross product has one nonzero component m = fl(h1 h2);
//            |n| = sqrt(m m) = m for any m whose square is in range, so n = +-e_d
//   area     0.5 (m + m) = m
//   alpha    centres of x neighbours differ in x only: 1 / |c[i+1] - c[i]|
//   length   |x_f - x_P|: the offset along the normal, and two offsets of
//            rounding size (the four-corner and eight-corner means of one
//            coordinate may differ in the last place), which must vanish when
//            their squares are added (checked for the largest of them)
//   volume   the face centre's coordinate along the normal (the four-corner
//            mean of one value), times m
// Means are taken in the corner order of corner(): along x the eight corners
// read 0000 1111, along y 0011 0011, along z 0101 0101.
double axis_tables(int64_t nx, int64_t ny, int64_t nz, double dx, double dy, double dz, bool f64, AxisTables t[3]) {
  const double bad = std::numeric_limits<double>::quiet_NaN();
  const int64_t n[3] = {nx, ny, nz};
  const double h[3] = {dx, dy, dz};
  auto mean4 = [](double a, double b, double c, double d) { return (((0.0 + a) + b) + c + d) / 4.0; };
  double off2[3][2] = {};  // largest square of the across-axis offset, per corner pattern of the face
  double min_len2[3] = {INFINITY, INFINITY, INFINITY}, max_len = 0, min_h[3], max_h[3], min_d = INFINITY;
  for (int d = 0; d < 3; ++d) {
    if (!(h[d] > 1e-70 && h[d] < 1e70) || !(double(n[d]) * h[d] < 1e70)) return bad;
    const size_t N = size_t(n[d]);
    AxisTables& a = t[d];
    a.h.resize(N);
    a.g.resize(N + 1);
    a.alpha.assign(N + 1, 1.0);  // a wall face multiplies phi_P - phi_P
    a.len_lo.resize(N);
    a.len_hi.resize(N);
    std::vector<double> c(N);
    for (int64_t i = 0; i <= n[d]; ++i) {
      const double X = double(i) * h[d];
      a.g[i] = mean4(X, X, X, X);
    }
    min_h[d] = INFINITY;
    max_h[d] = 0;
    for (int64_t i = 0; i < n[d]; ++i) {
      const double X0 = double(i) * h[d], X1 = double(i + 1) * h[d];
      a.h[i] = X1 - X0;
      double s = 0.0;
      for (int k = 0; k < 8; ++k) s = s + (((d == 0 ? k >> 2 : d == 1 ? k >> 1 : k) & 1) ? X1 : X0);
      c[i] = s / 8.0;
      const double lo = a.g[i] - c[i], hi = a.g[i + 1] - c[i];
      if (!(a.h[i] > 0) || !(lo < 0) || !(hi > 0)) return bad;
      a.len_lo[i] = -lo;
      a.len_hi[i] = hi;
      if (std::sqrt(lo * lo) != -lo || std::sqrt(hi * hi) != hi) return bad;
      // the two corner orders in which faces of the other axes take this coordinate
      const double e0 = (d == 0 ? mean4(X0, X0, X1, X1) : mean4(X0, X1, X1, X0)) - c[i];
      const double e1 = (d == 2 ? mean4(X1, X1, X0, X0) : d == 0 ? mean4(X0, X0, X1, X1) : mean4(X0, X1, X1, X0)) - c[i];
      off2[d][0] = std::max(off2[d][0], e0 * e0);
      off2[d][1] = std::max(off2[d][1], e1 * e1);
      min_len2[d] = std::min(min_len2[d], std::min(lo * lo, hi * hi));
      max_len = std::max(max_len, std::max(-lo, hi));
      min_h[d] = std::min(min_h[d], a.h[i]);
      max_h[d] = std::max(max_h[d], a.h[i]);
    }
    for (int64_t i = 0; i + 1 < n[d]; ++i) {
      const double D = c[i + 1] - c[i];
      if (!(D > 0) || std::sqrt(D * D) != D) return bad;
      const double cos_phi = D / (1.0 * D);
      a.alpha[i + 1] = std::fabs((1.0 / cos_phi) / D);
      min_d = std::min(min_d, D);
    }
  }
  // (x^2 + y^2) + z^2 must keep the square along the normal: rounding is
  // monotonic, so it does for every cell if it does for the smallest square
  // against the largest offsets (z faces take x and y, y faces x and z, x faces
  // y and z, each in its own corner order)
  auto keeps = [](double a, double b, double c, double want) { return (a + b) + c == want; };
  const double ex = std::max(off2[0][0], off2[0][1]), ey = std::max(off2[1][0], off2[1][1]), ez = std::max(off2[2][0], off2[2][1]);
  for (int d = 0; d < 3; ++d)
    for (const std::vector<double>* l : {&t[d].len_lo, &t[d].len_hi})
      for (double v : *l) {
        const double q = v * v;
        if (!(d == 0 ? keeps(q, ey, ez, q) : d == 1 ? keeps(ex, q, ez, q) : keeps(ex, ey, q, q))) return bad;
      }
  // every table value, converted, is finite (a product by zero stays zero)
  const double top = f64 ? std::numeric_limits<double>::max() : double(std::numeric_limits<float>::max());
  const double max_a = std::max(max_h[0] * max_h[1], std::max(max_h[0] * max_h[2], max_h[1] * max_h[2]));
  // volumes by whose reciprocal the kernels divide (box_ops.cu); the volume
  // itself is a sum of rounded terms, within a few parts in 10^3 of the product
  // on any mesh whose cells are not lost in the rounding of its coordinates
  const double min_v = min_h[0] * min_h[1] * min_h[2], max_v = max_h[0] * max_h[1] * max_h[2];
  if (!(min_v > 0x1p-79) || !(max_v < 0x1p23)) return bad;
  if (!(max_a < 0.5 * top) || !(1.0 / min_d < 0.5 * top) || !(max_len < 0.5 * top)) return bad;
  // magnitudes below `limit` overflow in no intermediate of the operators:
  // gradient 2 |phi| A / V, face value |phi| + len |gradient|, their products by A / V
  const double k1 = std::max(1.0, max_a), k2 = std::max(1.0, 2.0 * max_a / min_v);
  const double k3 = (1.0 + 2.0 * max_len * k2) * std::max(1.0, k1) * k2;
  const double limit = top / (16.0 * std::max(k3, std::max(k1, k2)));
  return std::isfinite(limit) ? limit : bad;
}
