// Ray backtrace, water-leg entry search and Frechet rows on the device, a lane
// per pick, FP64 with the reference's expression order (this file is compiled
// without FMA contraction, like the eikonal stencil).
//
//   trace_ray_from_receiver2d   src/rays2d.f90:7-153
//   trace_ray_section2d         src/rays2d.f90:157-720 (Heun steps along -grad T
//                               with step halving; interface, head-wave and
//                               diffraction handling; source snap)
//   find_interface_crossing2d   src/rays2d.f90:764-821
//   interpolate_*               src/rays2d.f90:825-1131, 1222-1350
//   find_optimal_entry_inv      src/inversion2d.f90:6344-6438
//   compute_frechet_for_ray2d   src/inversion2d.f90:4548-4787
//
// What bounds it: the latency of a ray's steps (up to 5000 a section, one
// after the other), so the longest rays' chains (9000 steps of ~3600 cycles
// alone in a warp, ~5500 in a full one) set the time.
//  * The lanes of a warp step together and a warp takes as many rays as keep
//    every warp resident (one where there are few picks), dealt strided, so
//    that the neighbours on a receiver line, which are the same length, end up
//    in warps that run at once.
//  * A step's chain is short: quotients by the grid step through its
//    reciprocal (five multiply-adds, correctly rounded, instead of a
//    division), lengths that are only compared without their root, and the
//    cell's gradients and the interface nodes around it in shared memory for
//    the dozen steps a ray spends there (each lane reads its own lines: with a
//    dozen warps on an SM the loads of every step took three times the step's
//    own chain).  The last two cells and columns are kept, and a predicted point
//    that enters a new one loads both at once: in a full warp some lane does in
//    nearly every step, and all wait (45 -> 30 ms below).
//  * The nine shorter steps of a ray at a head wave are tried by nine lanes at
//    once instead of one after the other (7000 -> 800 cycles an event).
//  * A ray caught in a cycle (a point it has been at before) is given up at
//    once: it would go round until it runs out of points.
// Times of 30276 picks on 2001 x 401 nodes: 150 -> 30 ms; 7870 picks on
// 401 x 121, a third of them caught: 153 -> 15 ms.
//
// A section's points are not stored: each segment is turned into its four
// slowness-derivative contributions as soon as both ends are final (only the
// last point of a section is ever moved after it is computed), consecutive
// segments that touch the same four parameters are merged, and the
// contributions are written as (pick, parameter) keys.  The caller sorts
// the keys and sums equal ones into CSR rows.  One pass traces and writes: a ray
// takes chunks of a pool as it goes, and a gather puts them in pick order
// (counting first cost a second trace: 57 of 130 ms on 2001 x 401 nodes).
#include "rays.cuh"
#include "model.h"
#include <algorithm>
#include <cmath>

namespace fmt2d {

namespace {

constexpr double kHugeT = 1.0e20;   // mod_fmt2d.f90:616
constexpr int kMaxPoints = 5000;    // rays2d.f90:206
constexpr int kMaxSec = 4;

// Phase tables (invert2d_main.f90:564-700): interface sequence (1-based,
// 2*n_tf entries) and time-field sequence.
__constant__ int c_ntf[6] = {0, 1, 2, 2, 4, 4};
__constant__ int c_seq[6][9] = {{0}, {0, 0, 2}, {0, 0, 3, 3, 0}, {0, 0, 4, 4, 0},
                                {0, 0, 2, 2, 1, 1, 2, 2, 2}, {0, 0, 1, 1, 2, 2, 2, 2, 2}};
__constant__ int c_tfs[6][5] = {{0}, {0, 1}, {0, 2, 3}, {0, 4, 5}, {0, 1, 6, 7, 8},
                                {0, 9, 10, 11, 12}};
__constant__ int c_tfreg[13] = {0, 5, 2, 2, 6, 6, 1, 1, 1, 1, 1, 5, 1};

// a / b for b with y = RN(1/b) by two residual corrections, the second of
// which rounds the quotient correctly (Markstein's theorem); operands near the
// ends of the exponent range are divided.
__device__ __forceinline__ double quot(double a, double b, double y) {
  const unsigned e = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  if (e - 100u < 1800u) {
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
  }
  return a == 0.0 ? a : a / b;   // (b > 0)
}

// floor(a / b): the product with y is within 2^-51 of the quotient relatively,
// so away from a whole number its floor is the quotient's.
__device__ __forceinline__ int cell_of(double a, double b, double y) {
  const double q = a * y, f = floor(q), r = q - f;
  if (fabs(q) < 1.0e6 && r > 1.0e-8 && r < 1.0 - 1.0e-8) return (int)f;
  return (int)floor(quot(a, b, y));
}

// Whether q = a * y (a quotient to within 2^-51 relatively) lies inside the
// cell that starts at the whole number c, away from its ends by more than that
// error: the quotient's floor is c, and a remainder's share of the cell is
// strictly between 0 and 1 (clamp01 leaves it).
__device__ __forceinline__ bool inside(double q, double c) {
  const double f = q - c;
  return f > 1.0e-8 && f < 1.0 - 1.0e-8;   // (cells are numbered below 1e6)
}
// a / b for an a inside a cell of width b.
__device__ __forceinline__ double share(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-q, b, a), y, q);
  return fma(fma(-q, b, a), y, q);
}

// sqrt(d2) < c (c > 0, c2 = c*c): squares away from c2 by more than the
// roundings decide without the root.
__device__ __forceinline__ bool shorter(double d2, double c, double c2) {
  if (d2 > c2 * (1.0 + 1.0e-14)) return false;
  if (d2 < c2 * (1.0 - 1.0e-14)) return true;
  return sqrt(d2) < c;
}

__device__ __forceinline__ double gxc(const TrModel& M, int ix) { return M.x0 + (ix - 1) * M.dx; }
__device__ __forceinline__ double gzc(const TrModel& M, int iz) { return 0.0 + (iz - 1) * M.dx; }
__device__ __forceinline__ double clamp01(double w) { return fmin(1.0, fmax(0.0, w)); }

// Slot of grid node (ix, iz) (1-based) if it belongs to region r, else -1.
__device__ __forceinline__ int region_node(const TrModel& M, const TrRegion& r, int ix, int iz) {
  if (ix < 1 || ix > M.nx || iz < 1 || iz > M.nz) return -1;
  const int br = iz - 1 - r.z_lo;
  if (br < 0 || br >= r.H) return -1;
  const int s = br * r.pitch + (ix - 1);
  return (r.code[s] & kInRegion) ? s : -1;
}

__device__ void node_pos(const TrModel& M, const TrRegion& r, int s, double& x, double& z) {
  const int row = s / r.pitch, col = s - row * r.pitch;
  if (row < r.H) {
    x = gxc(M, col + 1);
    z = gzc(M, r.z_lo + row + 1);
  } else {
    x = M.xpos[col];
    z = M.ifz[row == r.H ? r.itop : r.ibot][col];
  }
}

// rays2d.f90:996-1020: for a grid node outside the region, the nearest region
// node in the same column, up to five rows away.  A column's region nodes are
// one row range, so it is the range's near end.
__device__ __forceinline__ int nearby_row(int row, int a, int b) {
  if (a > b) return -1;
  const int e = row < a ? a : b;
  return abs(e - row) <= 5 ? e : -1;
}

__device__ __forceinline__ int nearby_node(const TrModel& M, const TrRegion& r, int ix, int iz) {
  if (ix < 1 || ix > M.nx) return -1;
  const int e = nearby_row(iz - 1, r.r0[ix - 1], r.r1[ix - 1]);
  return e < 0 ? -1 : (e - r.z_lo) * r.pitch + (ix - 1);
}

// The region node nearest to (px, pz), the first in the reference's node
// order among equals (grid nodes column by column, rows down each column,
// then the top and the bottom interface nodes by column): what a scan of
// every node with a strict "closer" test returns (rays2d.f90:966-972,
// 1118-1127).  The region's grid nodes are one row range per column, so the
// search widens column by column from the query and stops once a column's
// horizontal distance alone exceeds the best distance found; each column
// costs its nearest rows and its two interface nodes.
__device__ __noinline__ int nearest_node(const TrModel& M, const TrRegion& r, double px, double pz) {
  double best = 1.0e300;
  int bcls = 3, bcol = 0, brow = 0, bslot = -1;
  auto offer = [&](double d, int cls, int col, int row, int slot) {
    if (d < best || (d == best && (cls < bcls || (cls == bcls && (col < bcol ||
                                                  (col == bcol && row < brow)))))) {
      best = d; bcls = cls; bcol = col; brow = row; bslot = slot;
    }
  };
  const int nx = M.nx;
  int c0 = cell_of(px - M.x0, M.dx, M.rdx);
  c0 = max(0, min(nx - 1, c0));
  const int fr = cell_of(pz, M.dx, M.rdx);
  // columns c0, c0 - 1, c0 + 1, c0 - 2, ...: the horizontal distance grows on
  // each side, so once neither side's next column can hold a node as close as
  // the best (d >= its horizontal term), no farther column can either
  for (int k = 0;; ++k) {
    bool near = false;
    for (int side = 0; side < (k == 0 ? 1 : 2); ++side) {
      const int c = side == 0 ? c0 - k : c0 + k;
      if (c < 0 || c >= nx) continue;
      const double gx = gxc(M, c + 1), xi = M.xpos[c];
      if ((px - gx) * (px - gx) > best && (px - xi) * (px - xi) > best) continue;
      near = true;
      const int a = r.r0[c], b = r.r1[c];
      if (a <= b) {
#pragma unroll
        for (int q = -1; q <= 2; ++q) {
          const int row = min(b, max(a, fr + q));
          const double z = gzc(M, row + 1);
          offer((px - gx) * (px - gx) + (pz - z) * (pz - z), 0, c, row,
                (row - r.z_lo) * r.pitch + c);
        }
      }
      const double zt = M.ifz[r.itop][c], zb = M.ifz[r.ibot][c];
      offer((px - xi) * (px - xi) + (pz - zt) * (pz - zt), 1, c, 0, r.H * r.pitch + c);
      offer((px - xi) * (px - xi) + (pz - zb) * (pz - zb), 2, c, 0, (r.H + 1) * r.pitch + c);
    }
    if (!near && k > 0) break;
  }
  return bslot;
}

// Threads of a tracing block.
constexpr int kTraceThreads = 64;

// Per thread of a block, in shared memory: a cell of a region's grid, the cell
// between grid nodes a ray was in, with its column and row from 0, its corner
// node, the gradients at its corners (a corner outside the region takes
// nearby_node's) and which of them are in the region (bits, corner 1 first);
// and the nodes of a region's top and bottom interface around a column.
enum {
  kCqx = 0, kCqz, kCx, kCz, kCg1x, kCg2x, kCg3x, kCg4x, kCg1z, kCg2z, kCg3z, kCg4z, kCin, kCellN
};
enum { kIq = 0, kIx, kIt0, kIt1, kIb0, kIb1, kColN };
typedef double CellMem[kCellN][kTraceThreads];
typedef double ColMem[kColN][kTraceThreads];

// A cell's loads: the columns' row ranges and the corners' gradients together.
struct CellLoad {
  int c, row, la, lb, ra, rb;
  double2 a1, a2, a3, a4;
};

// (ix and ix + 1 are columns, iz and iz + 1 grid rows, from 1)
__device__ __forceinline__ CellLoad load_cell(const TrRegion& r, const double2* G, int ix, int iz) {
  CellLoad L;
  L.c = ix - 1;
  L.row = iz - 1;
  const int br = L.row - r.z_lo;
  const bool up = br >= 0 && br < r.H, dn = br + 1 >= 0 && br + 1 < r.H;
  const int s0 = up ? br * r.pitch + L.c : 0, s1 = dn ? (br + 1) * r.pitch + L.c : 0;
  L.la = r.r0[L.c];
  L.lb = r.r1[L.c];
  L.ra = r.r0[L.c + 1];
  L.rb = r.r1[L.c + 1];
  L.a1 = G[s0];
  L.a2 = G[s0 + 1];
  L.a3 = G[s1];
  L.a4 = G[s1 + 1];
  return L;
}

__device__ __forceinline__ void keep_cell(const TrRegion& r, const double2* G, CellMem& C,
                                          CellLoad& L, double x, double z) {
  const int t = threadIdx.x;
  auto in = [](int k, int a, int b) { return k >= a && k <= b; };
  const int mask = (in(L.row, L.la, L.lb) ? 1 : 0) | (in(L.row, L.ra, L.rb) ? 2 : 0) |
                   (in(L.row + 1, L.la, L.lb) ? 4 : 0) | (in(L.row + 1, L.ra, L.rb) ? 8 : 0);
  if (mask != 15) {
    // a corner outside the region takes its column's nearest region node
    auto other = [&](int bit, int k, int col, int a, int b, double2& g) {
      if (mask & bit) return;
      const int e = nearby_row(k, a, b);
      g = e >= 0 ? G[(e - r.z_lo) * r.pitch + col] : make_double2(0.0, 0.0);
    };
    other(1, L.row, L.c, L.la, L.lb, L.a1);
    other(2, L.row, L.c + 1, L.ra, L.rb, L.a2);
    other(4, L.row + 1, L.c, L.la, L.lb, L.a3);
    other(8, L.row + 1, L.c + 1, L.ra, L.rb, L.a4);
  }
  C[kCqx][t] = (double)L.c;
  C[kCqz][t] = (double)L.row;
  C[kCx][t] = x;
  C[kCz][t] = z;
  C[kCin][t] = (double)mask;
  C[kCg1x][t] = L.a1.x; C[kCg2x][t] = L.a2.x; C[kCg3x][t] = L.a3.x; C[kCg4x][t] = L.a4.x;
  C[kCg1z][t] = L.a1.y; C[kCg2z][t] = L.a2.y; C[kCg3z][t] = L.a3.y; C[kCg4z][t] = L.a4.y;
}

__device__ __noinline__ double2 enter_cell(const TrModel& M, const TrRegion& r, const double2* G,
                                           CellMem& C, double px, double pz) {
  const int t = threadIdx.x;
  int ix = cell_of(px - M.x0, M.dx, M.rdx) + 1;
  int iz = cell_of(pz - 0.0, M.dx, M.rdx) + 1;
  ix = max(1, min(M.nx - 1, ix));
  iz = max(1, min(M.nz - 1, iz));
  const double x = gxc(M, ix), z = gzc(M, iz);
  if ((double)(ix - 1) != C[kCqx][t] || (double)(iz - 1) != C[kCqz][t]) {
    CellLoad L = load_cell(r, G, ix, iz);
    keep_cell(r, G, C, L, x, z);
  }
  return make_double2(clamp01(quot(px - x, M.dx, M.rdx)), clamp01(quot(pz - z, M.dx, M.rdx)));
}

__device__ __forceinline__ bool in_cell(const TrModel& M, const CellMem& C, double px, double pz) {
  const int t = threadIdx.x;
  return inside((px - M.x0) * M.rdx, C[kCqx][t]) && inside((pz - 0.0) * M.rdx, C[kCqz][t]);
}

// rays2d.f90:825-894, in cell C with the point's shares w1, w2 of it.
__device__ __forceinline__ void grad_of_cell(const TrModel& M, const TrRegion& r,
                                             const double2* G, const CellMem& C, double px,
                                             double pz, double w1, double w2, double& dtdx,
                                             double& dtdz) {
  const int t = threadIdx.x;
  double gx = (1.0 - w1) * (1.0 - w2) * C[kCg1x][t] + w1 * (1.0 - w2) * C[kCg2x][t] +
              (1.0 - w1) * w2 * C[kCg3x][t] + w1 * w2 * C[kCg4x][t];
  double gz = (1.0 - w1) * (1.0 - w2) * C[kCg1z][t] + w1 * (1.0 - w2) * C[kCg2z][t] +
              (1.0 - w1) * w2 * C[kCg3z][t] + w1 * w2 * C[kCg4z][t];
  if (shorter(gx * gx + gz * gz, 0.01, 0.01 * 0.01)) {
    // position_in_region's node: the nearest corner in the region (column by
    // column), else the nearest of all region nodes
    const int mask = (int)C[kCin][t], ix = (int)C[kCqx][t] + 1, iz = (int)C[kCqz][t] + 1;
    const double xl = gxc(M, ix), xr = gxc(M, ix + 1), zu = gzc(M, iz), zd = gzc(M, iz + 1);
    double dmin = 1.0e100;
    int best = -1;
    auto corner = [&](int k, double x, double z) {
      const double d = (px - x) * (px - x) + (pz - z) * (pz - z);
      if (((mask >> k) & 1) && d < dmin) { best = k; dmin = d; }
    };
    corner(0, xl, zu);
    corner(2, xl, zd);
    corner(1, xr, zu);
    corner(3, xr, zd);
    gx = 0.0;
    gz = 0.0;
    if (best >= 0) {
      gx = C[kCg1x + best][t];
      gz = C[kCg1z + best][t];
    } else {
      const int nm = nearest_node(M, r, px, pz);
      if (nm >= 0) { gx = G[nm].x; gz = G[nm].y; }
    }
  }
  dtdx = gx;
  dtdz = gz;
}

// The same, the point's cell to be made C if it is not.
__device__ __forceinline__ void grad_in(const TrModel& M, const TrRegion& r, const double2* G,
                                        CellMem& C, double px, double pz, double& dtdx,
                                        double& dtdz) {
  double2 w;
  if (in_cell(M, C, px, pz))
    w = make_double2(share(px - C[kCx][threadIdx.x], M.dx, M.rdx),
                     share(pz - C[kCz][threadIdx.x], M.dx, M.rdx));
  else
    w = enter_cell(M, r, G, C, px, pz);
  grad_of_cell(M, r, G, C, px, pz, w.x, w.y, dtdx, dtdz);
}

// The same with no cell to start from (C is left as the point's cell).
__device__ __noinline__ double2 grad_at(const TrModel& M, const TrRegion& r, const double2* G,
                                        CellMem& C, double px, double pz) {
  C[kCqx][threadIdx.x] = -10.0;
  double gx, gz;
  grad_in(M, r, G, C, px, pz, gx, gz);
  return make_double2(gx, gz);
}

// rays2d.f90:898-975
__device__ double time_at(const TrModel& M, const TrRegion& r, const double* T, double px,
                          double pz) {
  int ix = cell_of(px - M.x0, M.dx, M.rdx) + 1;
  int iz = cell_of(pz - 0.0, M.dx, M.rdx) + 1;
  ix = max(1, min(M.nx - 1, ix));
  iz = max(1, min(M.nz - 1, iz));
  const double w1 = clamp01(quot(px - gxc(M, ix), M.dx, M.rdx));
  const double w2 = clamp01(quot(pz - gzc(M, iz), M.dx, M.rdx));
  auto tn = [&](int a, int b) {
    int s = region_node(M, r, a, b);
    if (s < 0) s = nearby_node(M, r, a, b);
    return s >= 0 ? T[s] : kHugeT;
  };
  const double t1 = tn(ix, iz), t2 = tn(ix + 1, iz), t3 = tn(ix, iz + 1), t4 = tn(ix + 1, iz + 1);
  const double hh = kHugeT * 0.5;
  if (t1 < hh && t2 < hh && t3 < hh && t4 < hh)
    return (1.0 - w1) * (1.0 - w2) * t1 + w1 * (1.0 - w2) * t2 + (1.0 - w1) * w2 * t3 +
           w1 * w2 * t4;
  const int s = nearest_node(M, r, px, pz);
  return s >= 0 ? T[s] : kHugeT;
}

// rays2d.f90:1222-1257
__device__ double iface_z(const TrModel& M, double px, int k) {
  const int nn = M.nx;
  const double* z = M.ifz[k];
  if (nn < 2) return z[0];
  const int ix = cell_of(px - M.xp0, M.dx, M.rdx) + 1;
  if (ix < 1) return z[0];
  if (ix >= nn) return z[nn - 1];
  const double w = clamp01(quot(px - M.xpos[ix - 1], M.dx, M.rdx));
  return (1.0 - w) * z[ix - 1] + w * z[ix];
}

// A column's loads.
struct ColLoad {
  int ix;                    // its first node, from 1; outside: 0 or nx
  double x, t0, t1, b0, b1;
};

__device__ __forceinline__ ColLoad load_col(const TrModel& M, double px, const double* zt,
                                            const double* zb) {
  const int nn = M.nx;
  ColLoad L;
  L.ix = nn < 2 ? 0 : cell_of(px - M.xp0, M.dx, M.rdx) + 1;
  L.ix = L.ix < 1 ? 0 : min(L.ix, nn);
  const int a = L.ix < 1 ? 0 : L.ix - 1, b = L.ix < 1 || L.ix >= nn ? a : L.ix;
  L.x = M.xpos[a];
  L.t0 = zt[a];
  L.t1 = zt[b];
  L.b0 = zb[a];
  L.b1 = zb[b];
  return L;
}

// The column as C, and the interfaces at px (outside the nodes: the end's).
__device__ __forceinline__ double2 keep_col(const TrModel& M, ColMem& C, const ColLoad& L,
                                            double px) {
  const int t = threadIdx.x;
  if (L.ix < 1 || L.ix >= M.nx) return make_double2(L.t0, L.b0);
  // (the share's numerator is taken from the node's own x: inside's margin
  // holds where that is the grid's up to rounding)
  const double q = (double)(L.ix - 1);
  C[kIq][t] = fabs(L.x - (M.xp0 + q * M.dx)) < 1.0e-9 * M.dx ? q : -10.0;
  C[kIx][t] = L.x;
  C[kIt0][t] = L.t0;
  C[kIt1][t] = L.t1;
  C[kIb0][t] = L.b0;
  C[kIb1][t] = L.b1;
  const double w = clamp01(quot(px - L.x, M.dx, M.rdx));
  return make_double2((1.0 - w) * L.t0 + w * L.t1, (1.0 - w) * L.b0 + w * L.b1);
}

__device__ __noinline__ double2 enter_col(const TrModel& M, double px, const double* zt,
                                          const double* zb, ColMem& C) {
  const ColLoad L = load_col(M, px, zt, zb);
  return keep_col(M, C, L, px);
}

__device__ __forceinline__ bool in_col(const TrModel& M, const ColMem& C, double px) {
  return inside((px - M.xp0) * M.rdx, C[kIq][threadIdx.x]);
}
__device__ __forceinline__ double2 pair_of_col(const TrModel& M, const ColMem& C, double px) {
  const int t = threadIdx.x;
  const double w = share(px - C[kIx][t], M.dx, M.rdx);
  return make_double2((1.0 - w) * C[kIt0][t] + w * C[kIt1][t],
                      (1.0 - w) * C[kIb0][t] + w * C[kIb1][t]);
}

// iface_z of a region's top and bottom interface at the same x.
__device__ __forceinline__ void iface_pair(const TrModel& M, double px, const double* zt,
                                           const double* zb, ColMem& C, double& top, double& bot) {
  const double2 z = in_col(M, C, px) ? pair_of_col(M, C, px) : enter_col(M, px, zt, zb, C);
  top = z.x;
  bot = z.y;
}

// rays2d.f90:1261-1306
__device__ void iface_normal(const TrModel& M, double px, int k, double& nx, double& nz) {
  const int nn = M.nx;
  const double* z = M.ifz[k];
  const double dx = M.dx;
  if (nn < 2) { nx = 0.0; nz = 1.0; return; }
  int ix = cell_of(px - M.xp0, dx, M.rdx) + 1;
  if (ix < 1) ix = 1;
  if (ix >= nn) ix = nn - 1;
  double dzdx;
  if (ix > 1 && ix < nn - 1) dzdx = (z[ix] - z[ix - 2]) / (2.0 * dx);
  else if (ix == 1 && nn >= 3) dzdx = (z[ix] - z[ix - 1]) / dx;
  else if (ix == nn - 1 && nn >= 3) dzdx = (z[ix] - z[ix - 2]) / (2.0 * dx);
  else dzdx = 0.0;
  const double l = sqrt(1.0 + dzdx * dzdx);
  nx = -dzdx / l;
  nz = 1.0 / l;
}

// rays2d.f90:1310-1350: bilinear propagation-grid velocity.
__device__ double vel_at(const TrModel& M, double px, double pz) {
  int ix = cell_of(px - M.x0, M.dx, M.rdx) + 1;
  int iz = cell_of(pz - 0.0, M.dx, M.rdx) + 1;
  ix = max(1, min(M.nx - 1, ix));
  iz = max(1, min(M.nz - 1, iz));
  const double w1 = clamp01(quot(px - gxc(M, ix), M.dx, M.rdx));
  const double w2 = clamp01(quot(pz - gzc(M, iz), M.dx, M.rdx));
  auto V = [&](int a, int b) { return M.vel[(size_t)(b - 1) * M.nx + (a - 1)]; };
  return (1.0 - w1) * (1.0 - w2) * V(ix, iz) + w1 * (1.0 - w2) * V(ix + 1, iz) +
         (1.0 - w1) * w2 * V(ix, iz + 1) + w1 * w2 * V(ix + 1, iz + 1);
}

// Frechet contributions of one pick.  They are written as the ray is traced,
// into chunks of the pool that it takes as it needs them: how many there will
// be is not known before its end.  Without a chunk left they are only counted.
// The pending entries are those of the last segment's cell, compacted (ids 0
// beyond them).
template <int MODE>
struct Sink {
  TrPool pool;
  unsigned long long chunk;  // the current chunk's first entry, ~0: none
  unsigned n;                // entries so far
  int pick;
  int cell;                  // the pending entries' cell, -1: none
  int ivx, ivz;              // its column and row, from 1
  double qx, qz;             // and from 0
  unsigned mask;             // its nodes that are parameters
  int i0, i1, i2, i3;
  double v0, v1, v2, v3;
};

template <int MODE>
__device__ __forceinline__ void sink_put(Sink<MODE>& k, int idx, double v) {
  if (idx <= 0) return;
  const unsigned at = k.n % kTrChunk;
  if (at == 0) {
    const unsigned c = atomicAdd(k.pool.used, 1u);
    k.chunk = ~0ull;
    if (c < k.pool.nchunks) {
      k.pool.owner[c] = make_uint2((unsigned)k.pick, k.n / kTrChunk);
      k.chunk = (unsigned long long)c * kTrChunk;
    }
  }
  if (k.chunk != ~0ull) {
    k.pool.ids[k.chunk + at] = idx;
    k.pool.vals[k.chunk + at] = v;
  }
  ++k.n;
}

template <int MODE>
__device__ __forceinline__ void sink_flush(Sink<MODE>& k) {
  if (MODE == kTrTimes) return;
  sink_put(k, k.i0, k.v0);
  sink_put(k, k.i1, k.v1);
  sink_put(k, k.i2, k.v2);
  sink_put(k, k.i3, k.v3);
  k.i0 = k.i1 = k.i2 = k.i3 = 0;
  k.v0 = k.v1 = k.v2 = k.v3 = 0.0;
  k.cell = -1;
  k.qx = k.qz = -10.0;
}

// Moves the entries of mask to the front (of ids or values; zeros behind).
template <class T>
__device__ __forceinline__ void compact(unsigned mask, T& a, T& b, T& c, T& d) {
  if (mask == 15u) return;
  if (!(mask & 8u)) d = T(0);
  if (!(mask & 4u)) { c = d; d = T(0); }
  if (!(mask & 2u)) { b = c; c = d; d = T(0); }
  if (!(mask & 1u)) { a = b; b = c; c = d; d = T(0); }
}

// inversion2d.f90:4581-4673: midpoint-rule bilinear splat of one segment's
// length onto the four inversion nodes around its midpoint, merged with the
// previous segment's when it touched the same parameters.
template <int MODE>
__device__ __forceinline__ void segment(const TrModel& M, Sink<MODE>& k, double x0, double z0,
                                        double x1, double z1) {
  if (MODE == kTrTimes) return;
  const double px = 0.5 * (x0 + x1), pz = 0.5 * (z0 + z1);
  const double ddx = x1 - x0, ddz = z1 - z0;
  const double d2 = ddx * ddx + ddz * ddz;
  if (shorter(d2, 1.0e-10, 1.0e-10 * 1.0e-10)) return;
  const bool same =
      inside((px - M.xp0) * M.rvdx, k.qx) && inside((pz - gzc(M, 1)) * M.rdx, k.qz);
  int ivx = k.ivx, ivz = k.ivz;
  if (!same) {
    if (pz < gzc(M, 1)) return;
    ivx = cell_of(px - M.xp0, M.vdx, M.rvdx) + 1;
    ivx = max(1, min(M.nx - 1, ivx));
    ivz = M.nz - 1;
    if (!(pz >= gzc(M, M.nz))) {
      ivz = cell_of(pz - gzc(M, 1), M.dx, M.rdx) + 1;
      ivz = max(1, min(M.nz - 1, ivz));
    }
  }
  const int cell = (ivz - 1) * M.nx + (ivx - 1);
  const double sl = sqrt(d2);
  const double wx = clamp01(quot(px - M.xpos[ivx - 1], M.vdx, M.rvdx));
  const double wz = pz >= gzc(M, M.nz) ? 1.0 : clamp01(quot(pz - gzc(M, ivz), M.dx, M.rdx));
  double a = (1.0 - wx) * (1.0 - wz) * sl;
  double b = wx * (1.0 - wz) * sl;
  double c = (1.0 - wx) * wz * sl;
  double d = wx * wz * sl;
  if (cell != k.cell) {
    int q0 = M.inv_idx[cell], q1 = M.inv_idx[cell + 1];
    int q2 = M.inv_idx[cell + M.nx], q3 = M.inv_idx[cell + M.nx + 1];
    k.mask = (q0 > 0 ? 1u : 0u) | (q1 > 0 ? 2u : 0u) | (q2 > 0 ? 4u : 0u) | (q3 > 0 ? 8u : 0u);
    compact(k.mask, q0, q1, q2, q3);
    // (another cell's parameters are the same only where some nodes are none)
    if (!(q0 == k.i0 && q1 == k.i1 && q2 == k.i2 && q3 == k.i3)) {
      sink_flush(k);
      k.i0 = q0; k.i1 = q1; k.i2 = q2; k.i3 = q3;
    }
    k.cell = cell;
    k.ivx = ivx;
    k.ivz = ivz;
    k.qx = (double)(ivx - 1);
    k.qz = (double)(ivz - 1);
  }
  compact(k.mask, a, b, c, d);
  k.v0 += a;
  k.v1 += b;
  k.v2 += c;
  k.v3 += d;
}

template <int MODE>
__device__ __forceinline__ void add_one(Sink<MODE>& k, int idx, double v) {
  sink_flush(k);
  if (MODE != kTrTimes) sink_put(k, idx, v);
}

struct Section {
  int tf, reg, istart, iend;
  int npts;
  double x1, z1;           // first point
};

// A thread's cells and columns: the last two that the ray's points and
// predicted points were in, and those of anything else.
struct TraceMem {
  CellMem cell[2], other;
  ColMem col[2], ocol;
};

__device__ __forceinline__ TraceMem& trace_mem() {
  __shared__ TraceMem m;
  return m;
}

// (the sections apart: indexed, they live in local memory, the rest in registers)
template <int MODE>
struct RayState {
  const TrModel* M;
  const TrField* F;        // this pick's source fields (indexed by tf)
  double sx, sz;           // source
  int raypath, nsec;
  Section* sec;
  bool valid, headwave, diffracted;
  Sink<MODE>* sink;
};

// find_interface_crossing2d (rays2d.f90:764-821).  On success X/Z (the
// current point) hold the crossing.
__device__ bool crossing(const TrModel& M, double Xp, double Zp, double& Xc, double& Zc,
                         double ppx, double ppz, int ie, double g0x, double g0z, double dl) {
  const double tol = 0.01 * M.tol;
  const double zi = iface_z(M, ppx, ie);
  const double x1 = 0.0, x2 = dl;
  const double f = Zp - iface_z(M, Xp, ie);
  double fmid = ppz - zi;
  if (f * fmid > tol) return false;
  if (fabs(f * fmid) <= tol) {
    Xc = Xp;
    Zc = iface_z(M, Xc, ie);
    return true;
  }
  if (f * fmid < -tol) {
    double rtbis, dxx;
    if (f < 0.0) { rtbis = x1; dxx = x2 - x1; }
    else { rtbis = x2; dxx = x1 - x2; }
    for (int k = 1; k <= 10; ++k) {
      dxx *= 0.5;
      const double xm = rtbis + dxx;
      Xc = Xp - xm * g0x;
      Zc = Zp - xm * g0z;
      fmid = Zc - iface_z(M, Xc, ie);
      if (fmid <= 0.0) rtbis = xm;
    }
    Xc = Xp - rtbis * g0x;
    Zc = Zp - rtbis * g0z;
    Zc = iface_z(M, Xc, ie);
  }
  return true;
}

// trace_ray_section2d (rays2d.f90:157-720), all sections of a ray from the
// receiver (x_in, z_in) to the source, one step (a pass of its ploop) at a
// time.  Whole warps call it, every lane with its own ray or none (active):
// the lanes take their steps together, whatever section they are in.  (Left to
// themselves, the lanes of a warp part at the first branch and most of them
// then run alone: 120 ms instead of 40 for the 30k rays of the 2001x401 model.)
template <int MODE>
__device__ __forceinline__ void trace_ray(RayState<MODE>& R, bool active, double x_in,
                                          double z_in) {
  const TrModel& M = *R.M;
  const double v_average = 5.0;
  const double dlmax = 0.1 * M.dx * v_average;
  const double p_tol = 5.0e-4 * M.dx;
  const double s_tol = 2.5 * M.dx;
  const double s_tol2 = s_tol * s_tol, p_tol2 = p_tol * p_tol;
  TraceMem& C = trace_mem();
  // the section: number, region, interfaces, fields
  int seqnum = active ? R.nsec : 0, iftop = 0, ifbot = 0, istart = 0, rid = 1;
  int ifend = 0;               // interface id the section ends on (0 none)
  int tfn = 0;                 // next section's time field
  int start_direction = 0;
  bool enter = active, refraction = false, same_internal = false, left_start = true;
  bool emit = false, on_bot = false, on_top = false;
  const double2* G = nullptr;
  const double *ztop = nullptr, *zbot = nullptr;
  // points: current (n), previous (n-1), the one before (n-2)
  int n = 1;
  double Xc = 0, Zc = 0, Xp = 0, Zp = 0, Xpp = 0, Zpp = 0, x_out = 0, z_out = 0;
  double dist_hw = 0.0;
  // From the third point on a step depends on the point and three flags alone:
  // at a point it has been at with the same flags the ray goes round until it
  // runs out of points or of head-wave length, and either makes it invalid.  The
  // points to compare with: one that moves on at powers of two (Brent), for
  // cycles of any length, and one every 32 points, which finds the common short
  // cycles soon.
  double Xs = 0, Zs = 0, Xk = 0, Zk = 0;
  int next_s = 4, flags_s = -1, flags_k = -1;
  auto near_src = [&](double x, double z) {
    const double dx = x - R.sx, dz = z - R.sz;
    return shorter(dx * dx + dz * dz, s_tol, s_tol2);
  };
  // whose the lane's other cell and column are (halve): a field and a pair of
  // interfaces
  const double2* other_g = nullptr;
  int other_if = -1;
  auto refracts = [&](double px, double zi, double& g0x, double& g0z) {
    double nx, nz;
    other_g = nullptr;
    iface_normal(M, px, ifend, nx, nz);
    const double2 g0 = grad_at(M, M.reg[rid], G, C.other, px, zi);
    const double2 g1 = grad_at(M, M.reg[c_tfreg[tfn]], R.F[tfn].G, C.other, px, zi);
    g0x = g0.x;
    g0z = g0.y;
    const double d = nx * g1.x + nz * g1.y;
    const double tx = g1.x - d * nx, tz = g1.y - d * nz;
    return sqrt(tx * tx + tz * tz) <= sqrt(g0x * g0x + g0z * g0z);
  };
  // what a step comes to: the next point (in Xc, Zc), the section's end there
  // (the ray's in the first section), the end of the loop (the exit point is
  // still to be found), an invalid ray
  enum { kNext, kEnd, kExit, kInvalid, kHalve };
  double g0x = 0, g0z = 0, ppx = 0, ppz = 0, dl = 0;
  int ci = 0, li = 0;          // the cell and the column used last
  // A point (px, pz) at or beyond interface k of the region ends the loop
  // (kExit), goes along the interface as a head wave or diffracted (kEnd: the
  // point is Xc, Zc), or may stay (kNext).  corrected: it is the corrector's
  // point, which takes the place of the predicted one at the end of the loop
  enum { kStay = kNext, kAlong = kEnd };
  auto stays = [&](int k, bool on) {
    return k != ifend && n == 2 && on && istart && istart == k;
  };
  auto beyond = [&](double px, double pz, double zi, int k, bool on, bool corrected) -> int {
    if (stays(k, on)) return kStay;
    if (k == ifend) {
      if (!refraction || (k == ifbot && R.raypath == 4 && seqnum == 2) ||
          refracts(px, zi, g0x, g0z)) {
        if (corrected) { ppx = px; ppz = pz; }
        return kExit;
      }
      R.headwave = true;
    } else {
      R.diffracted = true;
    }
    Xc = px;
    Zc = zi;
    return kAlong;
  };
  // how a step whose points are settled ends; w: beyond's answer, predicted:
  // for the predicted point
  auto settle = [&](int w, bool predicted) -> int {
    if (w == kExit) {
      if (seqnum == 1) return kInvalid;
      if (ifend && !crossing(M, Xp, Zp, Xc, Zc, ppx, ppz, ifend, g0x, g0z, dl)) return kInvalid;
      x_out = Xc;
      z_out = Zc;
      return kEnd;
    }
    // (a corrected point that goes along an interface is not tested against
    // the source until the next step)
    if (seqnum == 1 && (predicted || w == kStay) && near_src(Xc, Zc)) {
      Xc = R.sx; Zc = R.sz;
      return kEnd;
    }
    return kNext;
  };
  auto step = [&]() -> int {
    if (n >= 4) {
      const int f = (left_start ? 1 : 0) | (R.headwave ? 2 : 0) | (R.diffracted ? 4 : 0);
      if ((f == flags_s && Xp == Xs && Zp == Zs) || (f == flags_k && Xp == Xk && Zp == Zk))
        return kInvalid;
      if ((n & 31) == 0) {
        Xk = Xp;
        Zk = Zp;
        flags_k = f;
      }
      if (n == next_s) {
        Xs = Xp;
        Zs = Zp;
        flags_s = f;
        next_s *= 2;
      }
    }
    if (n > kMaxPoints) return kInvalid;
    if (seqnum == 1 && n > 2 && near_src(Xp, Zp)) {
      Xc = R.sx; Zc = R.sz;
      return kEnd;
    }
    if (R.headwave || R.diffracted) {
      if (n > 2) {
        const double ddx = Xp - Xpp, ddz = Zp - Zpp;
        dist_hw += sqrt(ddx * ddx + ddz * ddz);
      }
      if (dist_hw > 200.0) return kInvalid;
    }
    const TrRegion& reg = M.reg[rid];
    dl = dlmax;
    if (n == 2 && (on_bot || on_top)) dl = 10.0 * dlmax;
    double g1x, g1z;
    if (!in_cell(M, C.cell[ci], Xp, Zp)) ci ^= 1;
    grad_in(M, reg, G, C.cell[ci], Xp, Zp, g0x, g0z);
    ppx = Xp - dl * g0x;
    ppz = Zp - dl * g0z;
    // the corrector's gradient at the predicted point and the interfaces at its
    // x: where one of them is not at hand, both are loaded (one wait a step for
    // the warp: some lane enters a cell in nearly every step)
    double zit, zib;
    {
      bool cm = !in_cell(M, C.cell[ci], ppx, ppz), lm = !in_col(M, C.col[li], ppx);
      if (cm) {
        ci ^= 1;
        cm = !in_cell(M, C.cell[ci], ppx, ppz);
      }
      if (lm) {
        li ^= 1;
        lm = !in_col(M, C.col[li], ppx);
      }
      double2 wt, zz;
      if (cm || lm) {
        int ix = cell_of(ppx - M.x0, M.dx, M.rdx) + 1;
        int iz = cell_of(ppz - 0.0, M.dx, M.rdx) + 1;
        ix = max(1, min(M.nx - 1, ix));
        iz = max(1, min(M.nz - 1, iz));
        const double x = gxc(M, ix), z = gzc(M, iz);
        CellLoad cl = load_cell(reg, G, ix, iz);
        const ColLoad ll = load_col(M, ppx, ztop, zbot);
        if (cm) keep_cell(reg, G, C.cell[ci], cl, x, z);
        if (lm) zz = keep_col(M, C.col[li], ll, ppx);
        wt = make_double2(clamp01(quot(ppx - x, M.dx, M.rdx)),
                          clamp01(quot(ppz - z, M.dx, M.rdx)));
      }
      if (!cm)
        wt = make_double2(share(ppx - C.cell[ci][kCx][threadIdx.x], M.dx, M.rdx),
                          share(ppz - C.cell[ci][kCz][threadIdx.x], M.dx, M.rdx));
      if (!lm) zz = pair_of_col(M, C.col[li], ppx);
      zit = zz.x;
      zib = zz.y;
      grad_of_cell(M, reg, G, C.cell[ci], ppx, ppz, wt.x, wt.y, g1x, g1z);
    }
    if (on_bot && ppz > Zp) ppz = 2.0 * Zp - ppz;
    if (on_top && ppz < Zp) ppz = 2.0 * Zp - ppz;
    if (n == 2 && start_direction != 0 && !refraction && seqnum != 1) {
      double nx, nz;
      iface_normal(M, R.sec[seqnum].x1, istart, nx, nz);
      if (g0x * start_direction * nx + g0z * start_direction * nz > 0.0) return kInvalid;
    }
    if (ifend && ifend != iftop && ifend != ifbot) {
      const double fp = Zp - iface_z(M, Xp, ifend);
      const double fn = ppz - iface_z(M, ppx, ifend);
      if (same_internal && !left_start) {
        if (fabs(fn) > 0.5 * M.dx) left_start = true;
      } else if (fabs(fp) > 1.0e-3) {
        if (fp * fn <= 0.0) {
          double fr = fabs(fp - fn) > 1.0e-12 ? fp / (fp - fn) : 1.0;
          fr = fmin(1.0, fmax(0.0, fr));
          Xc = Xp + fr * (ppx - Xp);
          Zc = iface_z(M, Xc, ifend);
          if (seqnum == 1 && near_src(Xc, Zc)) { Xc = R.sx; Zc = R.sz; }
          return kEnd;   // the reference leaves the exit point unset on this branch
        }
      }
    }
    int w = kStay;
    if (ppz <= zit) w = beyond(ppx, ppz, zit, iftop, on_top, false);
    if (w == kStay && ppz >= zib) w = beyond(ppx, ppz, zib, ifbot, on_bot, false);
    if (w != kStay) return settle(w, true);
    // the Heun step; where its two points are too far apart, halved (halve)
    ppx = Xp - dl * g0x;
    ppz = Zp - dl * g0z;
    Xc = Xp - dl * (g0x + g1x) * 0.5;
    Zc = Zp - dl * (g0z + g1z) * 0.5;
    if (!in_col(M, C.col[li], Xc)) li ^= 1;
    iface_pair(M, Xc, ztop, zbot, C.col[li], zit, zib);
    if (Zc <= zit) w = beyond(Xc, Zc, zit, iftop, on_top, true);
    if (w == kStay && Zc >= zib) w = beyond(Xc, Zc, zib, ifbot, on_bot, true);
    if (w != kStay) return settle(w, false);
    const double ex = Xc - ppx, ez = Zc - ppz;
    if (!shorter(ex * ex + ez * ez, p_tol, p_tol2)) return kHalve;
    return settle(kStay, false);
  };
  // itloop's halvings for lane src's ray: the nine step lengths left are tried
  // at once, a lane each, and the first that settles the step counts.  Returns
  // (to that lane) beyond's answer, kHalve if none did.  A few rays near a
  // valley of the time field halve at every one of their 5000 steps; one by one
  // their trials took longer than all other rays of the batch.
  auto halve = [&](int src) -> int {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double bx = __shfl_sync(all, Xp, src), bz = __shfl_sync(all, Zp, src);
    const double bgx = __shfl_sync(all, g0x, src), bgz = __shfl_sync(all, g0z, src);
    const int top = __shfl_sync(all, iftop, src), bot = __shfl_sync(all, ifbot, src);
    const int br = __shfl_sync(all, rid, src);
    const double2* bG = reinterpret_cast<const double2*>(
        __shfl_sync(all, reinterpret_cast<unsigned long long>(G), src));
    const int skip =
        __shfl_sync(all, (stays(iftop, on_top) ? 1 : 0) | (stays(ifbot, on_bot) ? 2 : 0), src);
    // (exact: halving changes the exponent only)
    const double d =
        __shfl_sync(all, dl, src) * __hiloint2double((1023 - 1 - (lane < 9 ? lane : 0)) << 20, 0);
    double px = 0, pz = 0, x = 0, z = 0, zi = 0;
    int code = 0;
    if (lane < 9) {
      px = bx - d * bgx;
      pz = bz - d * bgz;
      if (bG != other_g) C.other[kCqx][threadIdx.x] = -10.0;
      if (top * 8 + bot != other_if) C.ocol[kIq][threadIdx.x] = -10.0;
      other_g = bG;
      other_if = top * 8 + bot;
      double g1x, g1z, zt, zb;
      grad_in(M, M.reg[br], bG, C.other, px, pz, g1x, g1z);
      x = bx - d * (bgx + g1x) * 0.5;
      z = bz - d * (bgz + g1z) * 0.5;
      iface_pair(M, x, M.ifz[top], M.ifz[bot], C.ocol, zt, zb);
      const double ex = x - px, ez = z - pz;
      if (z <= zt && !(skip & 1)) { code = 1; zi = zt; }
      else if (z >= zb && !(skip & 2)) { code = 2; zi = zb; }
      else if (shorter(ex * ex + ez * ez, p_tol, p_tol2)) code = 3;
    }
    const unsigned m = __ballot_sync(all, code != 0);
    const int f = m ? __ffs(m) - 1 : 0;
    const double fx = __shfl_sync(all, x, f), fz = __shfl_sync(all, z, f);
    const double fpx = __shfl_sync(all, px, f), fpz = __shfl_sync(all, pz, f);
    const double fzi = __shfl_sync(all, zi, f), fd = __shfl_sync(all, d, f);
    const int fc = __shfl_sync(all, code, f);
    if (lane != src) return kNext;
    if (!m) return kHalve;
    Xc = fx;
    Zc = fz;
    ppx = fpx;
    ppz = fpz;
    dl = fd;
    if (fc == 1) return beyond(Xc, Zc, fzi, iftop, on_top, true);
    if (fc == 2) return beyond(Xc, Zc, fzi, ifbot, on_bot, true);
    return kStay;
  };
  while (__any_sync(0xffffffffu, active)) {
    int w = kNext;
    if (active) {
      if (enter) {
        enter = false;
        Section& rs = R.sec[seqnum];
        rid = rs.reg;
        iftop = M.reg[rid].itop;
        ifbot = M.reg[rid].ibot;
        istart = rs.istart;
        G = R.F[rs.tf].G;
        ztop = M.ifz[iftop];
        zbot = M.ifz[ifbot];
        ifend = seqnum > 1 ? rs.iend : 0;
        tfn = seqnum > 1 ? R.sec[seqnum - 1].tf : 0;
        refraction = seqnum > 1 && c_tfreg[tfn] != rid;
        start_direction = seqnum < R.nsec ? rid - c_tfreg[R.sec[seqnum + 1].tf] : 0;
        same_internal =
            ifend && istart && ifend == istart && ifend != iftop && ifend != ifbot;
        left_start = !same_internal;
        emit = rid != 1;   // water sections carry no slowness derivatives
        n = 1;
        Xc = x_in;
        Zc = z_in;
        Xp = Zp = Xpp = Zpp = 0.0;
        dist_hw = 0.0;
        on_bot = fabs(z_in - iface_z(M, x_in, ifbot)) < 0.1 * M.dx;
        on_top = fabs(z_in - iface_z(M, x_in, iftop)) < 0.1 * M.dx;
        rs.x1 = x_in;
        rs.z1 = z_in;
        next_s = 4;
        flags_s = flags_k = -1;
        C.cell[0][kCqx][threadIdx.x] = C.cell[1][kCqx][threadIdx.x] = -10.0;
        C.col[0][kIq][threadIdx.x] = C.col[1][kIq][threadIdx.x] = -10.0;
      }
      ++n;
      Xpp = Xp; Zpp = Zp;
      Xp = Xc; Zp = Zc;
      if (MODE != kTrTimes && emit && n >= 3) segment(M, *R.sink, Xpp, Zpp, Xp, Zp);
      w = step();
    }
    for (unsigned m = __ballot_sync(0xffffffffu, w == kHalve); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int h = halve(src);
      if ((int)(threadIdx.x & 31) == src) w = h == kHalve ? kInvalid : settle(h, false);
    }
    if (active) {
      if (w == kInvalid) {
        R.valid = false;
        active = false;
      } else if (w == kEnd) {
        R.sec[seqnum].npts = n;
        if (MODE != kTrTimes && emit) segment(M, *R.sink, Xp, Zp, Xc, Zc);
        --seqnum;
        active = seqnum > 0;
        enter = true;
        x_in = x_out;
        z_in = z_out;
      }
    }
  }
}

// inversion2d.f90:6344-6438: best seafloor entry point of an in-water pick.
__device__ void optimal_entry(const TrModel& M, const TrRegion& r, const double* T,
                              const double* sft, double rx, double rz, double& ex, double& ez,
                              double& wt) {
  const int nsf = M.nx;
  const double* sz = M.ifz[2];
  const double* sxp = M.xpos;
  const double dxs = sxp[1] - sxp[0];
  auto sf_z = [&](double px) {
    if (nsf < 2) return sz[0];
    const int ixx = cell_of(px - M.xp0, dxs, M.rvdx) + 1;
    if (ixx < 1) return sz[0];
    if (ixx >= nsf) return sz[nsf - 1];
    const double w = clamp01(quot(px - sxp[ixx - 1], dxs, M.rvdx));
    return (1.0 - w) * sz[ixx - 1] + w * sz[ixx];
  };
  double tbest = kHugeT;
  const double z0 = sf_z(rx);
  double xb = rx, zb = z0, wb = (z0 - rz) / M.vwater;
  // the field's time at each seafloor node is the same for every pick of the
  // source: precomputed once per field (sft), else interpolated here.  A node
  // can only be better if the distance's square is within ((tbest - tf) *
  // vwater)^2, up to the roundings: most are settled without root and quotient
  for (int i = 0; i < nsf; ++i) {
    const double xt = sxp[i], zs = sz[i];
    const double tf = sft ? sft[i] : time_at(M, r, T, xt, zs);
    if (tf > kHugeT * 0.5) continue;
    const double d2 = (xt - rx) * (xt - rx) + (zs - rz) * (zs - rz);
    const double lim = (tbest - tf) * M.vwater;
    if (lim < 0.0 || d2 > lim * lim * (1.0 + 1.0e-9)) continue;
    const double tw = quot(sqrt(d2), M.vwater, M.rvwater);
    if (tf + tw < tbest) { tbest = tf + tw; xb = xt; zb = zs; wb = tw; }
  }
  if (xb <= sxp[0] || xb >= sxp[nsf - 1]) { ex = xb; ez = zb; wt = wb; return; }
  double xl = 0, xr = 0;
  for (int i = 0; i < nsf - 1; ++i)
    if (xb >= sxp[i] && xb <= sxp[i + 1]) { xl = sxp[i]; xr = sxp[i + 1]; break; }
  const int nref = 10;
  const double dr = (xr - xl) / double(nref);
  for (int k = 1; k <= nref - 1; ++k) {
    const double xt = xl + double(k) * dr;
    const double zs = sf_z(xt);
    const double tf = time_at(M, r, T, xt, zs);
    if (tf > kHugeT * 0.5) continue;
    const double tw = sqrt((xt - rx) * (xt - rx) + (zs - rz) * (zs - rz)) / M.vwater;
    if (tf + tw < tbest) { tbest = tf + tw; xb = xt; zb = zs; wb = tw; }
  }
  ex = xb; ez = zb; wt = wb;
}

// inversion2d.f90:4675-4759: interface-depth entries of a reflection or
// transmission at the inverted interface.
template <int MODE>
__device__ void iface_entries(RayState<MODE>& R) {
  const TrModel& M = *R.M;
  if (M.iface_inv <= 0) return;
  const int np = M.n_inv;
  bool done_rec = false, do_if = false;
  int prev = 0;
  for (int k = R.nsec; k >= 1; --k) {
    const Section& rs = R.sec[k];
    if (rs.npts <= 2) continue;
    if (!done_rec) { prev = k; done_rec = true; }
    else do_if = true;
    if (do_if) {
      if (rs.istart == 0) { prev = k; continue; }
      if (rs.istart == M.iface_inv) {
        const double px = rs.x1, pz = rs.z1;
        const double2 g = grad_at(M, M.reg[rs.reg], R.F[rs.tf].G, trace_mem().other, px, pz);
        double gx = g.x, gz = g.y;
        const double vin = vel_at(M, px, pz);
        const double nl = sqrt(gx * gx + gz * gz);
        if (nl > 0.0) { gx = gx / (vin * nl); gz = gz / (vin * nl); }
        double nx, nz;
        iface_normal(M, px, rs.istart, nx, nz);
        const double gin = gx * nx + gz * nz;
        double gout;
        if (rs.reg == R.sec[prev].reg) {
          gout = -gin;
        } else {
          const double tx = gx - gin * nx, tz = gz - gin * nz;
          const double par = sqrt(tx * tx + tz * tz);
          const double vout = vel_at(M, px, pz);
          double det = 1.0 / (vout * vout) - par * par;
          if (det < 0.0) det = 0.0;
          gout = copysign(sqrt(det), gin);
        }
        const double geo = (gin - gout) * nz;
        const double dxi = M.xpos[1] - M.xpos[0];
        int ivx = (int)floor((px - M.xpos[0]) / dxi) + 1;
        ivx = max(1, min(M.nx - 1, ivx));
        const double wx = clamp01((px - M.xpos[ivx - 1]) / dxi);
        int idx = M.iface_start + ivx - 1;
        if (idx >= 1 && idx + 1 <= np) add_one(*R.sink, idx + 1, (1.0 - wx) * geo);
        idx = M.iface_start + ivx;
        if (idx >= 1 && idx + 1 <= np) add_one(*R.sink, idx + 1, wx * geo);
      }
    }
    prev = k;
  }
}

__device__ double seafloor_z(const TrModel& M, double px) {
  const int n = M.nx;
  const double* z = M.ifz[2];
  if (n < 2) return z[0];
  const double dx = M.xpos[1] - M.xpos[0];
  const int ixx = (int)floor((px - M.xpos[0]) / dx) + 1;
  if (ixx < 1) return z[0];
  if (ixx >= n) return z[n - 1];
  const double w = clamp01((px - M.xpos[ixx - 1]) / dx);
  return (1.0 - w) * z[ixx - 1] + w * z[ixx];
}

// per: rays of a warp (its first lanes).
template <int MODE>
__global__ void __launch_bounds__(kTraceThreads, 4)
    k_trace(const __grid_constant__ TrModel M, const TrField* fields, const double* src_x,
            const double* src_z, const TrPick* picks, int npick, int per, double* t_calc,
            int* valid, bool again, unsigned* cnt, TrPool pool, double* entry) {
  // (lanes without a ray go along: whole warps trace)
  const int lane = threadIdx.x & 31;
  const int p0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) +
                 lane * (int)(gridDim.x * (kTraceThreads / 32));
  const bool mine = lane < per && p0 < npick && !(again && !valid[p0]);
  const int p = mine ? p0 : 0;
  const TrPick pk = picks[p];
  Section sec[kMaxSec + 1];
  RayState<MODE> R;
  R.sec = sec;
  R.M = &M;
  R.F = fields + (size_t)pk.src * 13;
  R.sx = src_x[pk.src];
  R.sz = src_z[pk.src];
  R.raypath = pk.phase;
  R.valid = true;
  R.headwave = false;
  R.diffracted = false;
  Sink<MODE> sk;
  sk.pool = pool;
  sk.chunk = ~0ull;
  sk.n = 0;
  sk.pick = p;
  sk.cell = -1;
  sk.ivx = sk.ivz = 1;
  sk.qx = sk.qz = -10.0;
  sk.mask = 0;
  sk.i0 = sk.i1 = sk.i2 = sk.i3 = 0;
  sk.v0 = sk.v1 = sk.v2 = sk.v3 = 0.0;
  R.sink = &sk;
  const int ns = c_ntf[pk.phase];
  R.nsec = ns;
  bool ok = mine && ns > 0;
  for (int n = ns; n >= 1 && ok; --n) {
    Section& rs = R.sec[n];
    rs.tf = c_tfs[pk.phase][n];
    rs.reg = c_tfreg[rs.tf];
    rs.istart = (n < ns) ? c_seq[pk.phase][2 * n] : 0;
    rs.iend = (n > 1) ? c_seq[pk.phase][2 * n - 1] : 0;
    rs.npts = 0;
    if (!R.F[rs.tf].T) ok = false;   // field not solved
  }
  double tr = kHugeT;
  double ent_x = pk.rx, ent_z = pk.rz, ent_w = 0.0;   // the ray's receiver end, water time
  double x_in = 0.0, z_in = 0.0, wt_ray = 0.0;
  if (ok) {
    // invert2d_main.f90:517-537: a receiver above the seafloor is in water
    const double zsf = seafloor_z(M, pk.rx);
    const bool in_water = pk.rz < zsf;
    double recx = pk.rx, recz = in_water ? zsf : pk.rz, wt = 0.0;
    const int last_tf = R.sec[ns].tf;
    const TrRegion& lr = M.reg[c_tfreg[last_tf]];
    if (in_water) {
      if (pk.phase == 4 || pk.phase == 5) {
        recx = pk.rx;
        recz = pk.rz;
      } else {
        optimal_entry(M, lr, R.F[last_tf].T, R.F[last_tf].sft, pk.rx, pk.rz, recx, recz, wt);
      }
    }
    ent_x = recx;
    ent_z = recz;
    ent_w = wt;
    // trace_ray_from_receiver2d
    tr = time_at(M, lr, R.F[last_tf].T, recx, recz);
    const double2 rg = grad_at(M, lr, R.F[last_tf].G, trace_mem().other, recx, recz);
    if (tr > 1.0e10) R.valid = false;
    if (rg.x == 0.0 && rg.y == 0.0) R.valid = false;
    x_in = recx;
    z_in = recz;
    wt_ray = wt;
  }
  trace_ray(R, ok && R.valid, x_in, z_in);
  if (ok) {
    if (R.valid) tr = tr + wt_ray;
    ok = R.valid;
  }
  if (MODE != kTrTimes && ok) {
    sink_flush(sk);
    iface_entries(R);
    sink_flush(sk);
  }
  if (mine && !again) {
    t_calc[p] = tr;
    valid[p] = ok ? 1 : 0;
    if (MODE == kTrRows) cnt[p] = ok ? sk.n : 0u;
    if (entry) {
      entry[3 * (size_t)p] = ent_x;
      entry[3 * (size_t)p + 1] = ent_z;
      entry[3 * (size_t)p + 2] = ent_w;
    }
  }
}

__global__ void k_sf_times(const __grid_constant__ TrModel M, const SfJob* jobs, int njobs,
                           int nx) {
  const SfJob J = jobs[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x)
    J.out[i] = time_at(M, M.reg[J.reg], J.T, M.xpos[i], M.ifz[2][i]);
}

// The slots and weights through which time_at(px, pz) reads the field:
// time_at = sum_k w[k] * T[s[k]] (k < the returned count), or 0 nodes where
// it returns huge_time.
__device__ int time_weights(const TrModel& M, const TrRegion& r, const double* T, double px,
                            double pz, int* s, double* w) {
  int ix = cell_of(px - M.x0, M.dx, M.rdx) + 1;
  int iz = cell_of(pz - 0.0, M.dx, M.rdx) + 1;
  ix = max(1, min(M.nx - 1, ix));
  iz = max(1, min(M.nz - 1, iz));
  const double w1 = clamp01(quot(px - gxc(M, ix), M.dx, M.rdx));
  const double w2 = clamp01(quot(pz - gzc(M, iz), M.dx, M.rdx));
  auto sn = [&](int a, int b) {
    int q = region_node(M, r, a, b);
    if (q < 0) q = nearby_node(M, r, a, b);
    return q;
  };
  s[0] = sn(ix, iz);
  s[1] = sn(ix + 1, iz);
  s[2] = sn(ix, iz + 1);
  s[3] = sn(ix + 1, iz + 1);
  const double hh = kHugeT * 0.5;
  bool all = true;
  for (int k = 0; k < 4; ++k) all = all && s[k] >= 0 && T[s[k]] < hh;
  if (all) {
    w[0] = (1.0 - w1) * (1.0 - w2);
    w[1] = w1 * (1.0 - w2);
    w[2] = (1.0 - w1) * w2;
    w[3] = w1 * w2;
    return 4;
  }
  s[0] = nearest_node(M, r, px, pz);
  if (s[0] < 0 || !(T[s[0]] < hh)) return 0;
  w[0] = 1.0;
  return 1;
}

// One block per target field (src*13 + tf in tgt), whose picks are
// tpk[tp[k] .. tp[k+1]) in pick order: the threads find the weights of a
// chunk of picks at once, then one thread adds coef[p] times them to d in
// pick order, so the sums do not depend on thread timing.
__global__ void __launch_bounds__(128) k_adj_picks(const __grid_constant__ TrModel M,
                                                   const TrField* fields,
                                                   const TrPick* picks, const double* entry,
                                                   const double* coef, const int* tgt,
                                                   const int* tp, const int* tpk,
                                                   double* const* d) {
  const int k = blockIdx.x;
  const int src = tgt[k] / 13, tf = tgt[k] % 13;
  const double* T = fields[(size_t)src * 13 + tf].T;
  const TrRegion& r = M.reg[c_tfreg[tf]];
  double* dk = d[k];
  __shared__ int s_n[128], s_sl[128][4];
  __shared__ double s_w[128][4];
  for (int base = tp[k]; base < tp[k + 1]; base += blockDim.x) {
    const int i = base + threadIdx.x;
    s_n[threadIdx.x] = 0;
    if (i < tp[k + 1]) {
      const int p = tpk[i];
      int sl[4];
      double w[4];
      const int n = time_weights(M, r, T, entry[3 * (size_t)p], entry[3 * (size_t)p + 1], sl, w);
      s_n[threadIdx.x] = n;
      for (int j = 0; j < n; ++j) {
        s_sl[threadIdx.x][j] = sl[j];
        s_w[threadIdx.x][j] = coef[p] * w[j];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int m = min((int)blockDim.x, tp[k + 1] - base);
      for (int t = 0; t < m; ++t)
        for (int j = 0; j < s_n[t]; ++j) dk[s_sl[t][j]] += s_w[t][j];
    }
    __syncthreads();
  }
}

}  // namespace

void tr_adj_picks(const TrModel& m, const TrField* fields, const TrPick* picks,
                  const double* entry, const double* coef, const int* tgt, const int* tp,
                  const int* tpk, double* const* d, int ntgt, cudaStream_t st) {
  if (ntgt <= 0) return;
  k_adj_picks<<<ntgt, 128, 0, st>>>(m, fields, picks, entry, coef, tgt, tp, tpk, d);
}

void tr_sf_times(const TrModel& m, const SfJob* jobs, int njobs, int nx, cudaStream_t st) {
  if (njobs <= 0) return;
  k_sf_times<<<dim3((nx + 127) / 128, njobs), 128, 0, st>>>(m, jobs, njobs, nx);
}

// One block per chunk: an entry's place is its pick's offset plus its number
// within the pick.
__global__ void __launch_bounds__(kTrChunk)
    k_gather(TrPool pool, const int* valid, const unsigned* cnt, const unsigned long long* off,
             unsigned long long* keys, double* vals) {
  const uint2 o = pool.owner[blockIdx.x];
  const unsigned i = o.y * kTrChunk + threadIdx.x;
  if (!valid[o.x] || i >= cnt[o.x]) return;
  const unsigned long long from = (unsigned long long)blockIdx.x * kTrChunk + threadIdx.x;
  keys[off[o.x] + i] = ((unsigned long long)o.x << 32) | (unsigned)pool.ids[from];
  vals[off[o.x] + i] = pool.vals[from];
}

void tr_gather(const TrPool& pool, unsigned nchunks, const int* valid, const unsigned* cnt,
               const unsigned long long* off, unsigned long long* keys, double* vals,
               cudaStream_t st) {
  if (nchunks == 0) return;
  k_gather<<<nchunks, kTrChunk, 0, st>>>(pool, valid, cnt, off, keys, vals);
}

void tr_launch(TrMode mode, const TrModel& m, const TrField* fields, const double* src_x,
               const double* src_z, const TrPick* picks, int npick, double* t_calc, int* valid,
               bool again, unsigned* cnt, const TrPool& pool, double* entry, cudaStream_t st) {
  // rays of a warp: as few as keep all warps resident at once
  int dev = 0, nsm = 148, blocks = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_trace<kTrRows>, kTraceThreads, 0);
  const int warps = std::max(1, nsm * std::max(1, blocks) * (kTraceThreads / 32));
  const int per = std::min(32, (npick + warps - 1) / warps);
  const int need = (npick + per - 1) / per;
  const int grid = (need + kTraceThreads / 32 - 1) / (kTraceThreads / 32);
  auto run = [&](auto kernel) {
    kernel<<<grid, kTraceThreads, 0, st>>>(m, fields, src_x, src_z, picks, npick, per, t_calc,
                                           valid, again, cnt, pool, entry);
  };
  if (mode == kTrTimes) run(k_trace<kTrTimes>);
  else run(k_trace<kTrRows>);
}

}  // namespace fmt2d
