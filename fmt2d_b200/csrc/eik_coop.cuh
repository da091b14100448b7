// Evaluation of an eikonal node by the solver's thread block: the same
// candidates as eik_eval.cuh's update_grid / update_iface, in the same
// expressions and with the same tie order, so the value written is the same to
// the last bit, but arranged so that a step of the solver waits for as few
// instructions as possible.
//
// * Regular quadrants: a thread per node (reg_best).  The candidates of the
//   earlier x and the earlier z neighbour are formed; of the other quadrants
//   only those whose trigger is not later than the best time found can change
//   the result (a candidate's time is at or above its trigger's), which is
//   rare, and they are formed in a loop.
// * Cells cut by an interface: sixteen lanes per node (cut_best).  They load
//   the nodes around it at once, a lane per member forms its one-sided event,
//   and the plane-front events of member pairs are formed a lane each, again
//   only where the trigger is not later than the best of the regular and
//   one-sided candidates: such a pair can neither win nor decide the suspect
//   flag.  Most nodes have none.
//
// (One node evaluated by one thread with every candidate formed took 77k of
// the 85k cycles of a step's evaluate phase at 2001x401: a cut cell's update
// is a chain of up to 60 events.)
//
// Divisions and square roots that only feed a comparison are left out where a
// product decides it beyond rounding (the comment at each bound says why);
// inside the bound the reference's expression is evaluated.
#pragma once
#include "eik_eval.cuh"

namespace fmt2d {
namespace ev {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ double shfl(double x, int lane) {
  return __shfl_sync(kFull, x, lane);
}

// Solver record of a slot, one 32-byte sector: time, velocity (negative
// unless the node is a fully regular, updated one), gradient.  A neighbour
// costs one load instead of three: a step's loads go to 32 different lines per
// warp, and the line lookups were its largest cost.
struct Rec {
  double T, v, gx, gz;
};

__device__ __forceinline__ Rec load_rec(const Fld64& F, int s) {
  Rec r;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(r.T), "=d"(r.v), "=d"(r.gx), "=d"(r.gz)
               : "l"(F.R + s));
  return r;
}

// The node being evaluated, as it stands.
struct Self {
  double T;
  double2 g;
  uint8_t fl;
};

constexpr int kNoKey = 0x7fffffff;

__device__ __forceinline__ bool before(double t, double trig, int key, double bt, double btrig,
                                       int bkey) {
  return t < bt || (t == bt && (trig < btrig || (trig == btrig && key < bkey)));
}

// a / b for b with reciprocal y = RN(1/b): two residual corrections; the
// second rounds the quotient correctly (Markstein's theorem; a and the
// quotient are far from the ends of the exponent range here).
__device__ __forceinline__ double div_by(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-q, b, a), y, q);
  return fma(fma(-q, b, a), y, q);
}

// a / b and sqrt(x) with a zero a or x set aside: those operands leave the
// compiler's short division and root for its general ones, about 500 cycles
// for the whole warp, and they are common here (a node straight above a
// member, equal times).  b is neither zero nor infinite, x not negative.
__device__ __forceinline__ double quot(double a, double b) {
  double n = a == 0.0 ? 1.0 : a;
  asm("" : "+d"(n));   // (else the select is folded away)
  const double q = n / b;
  return a == 0.0 ? (b < 0.0 ? -a : a) : q;
}
__device__ __forceinline__ double root(double x) {
  double y = x > 0.0 ? x : 1.0;
  asm("" : "+d"(y));
  const double r = sqrt(y);
  return x > 0.0 ? r : 0.0;
}

// ---------------------------------------------------------------- regular quadrants
// A direction's terms of regular_update2d's quadratic (the neighbour's time T,
// the second-order neighbour's T2, 0 at first order).
struct Dir {
  double A, B, C, T, T2, dpos;
};

// Direction k (L, R, U, D) of grid slot s = (r, c), whose first neighbour n1 is
// reached.
__device__ __forceinline__ Dir dir_of(const Fld64& F, double rdx, int s, int r, int c, double vu,
                                      int k, const Rec& n1) {
  const int sgn = (k & 1) ? 1 : -1;
  const bool dirx = k < 2;
  const int off = dirx ? sgn : sgn * F.pitch, p2 = (dirx ? c : r) + 2 * sgn;
  const bool two = p2 >= 0 && p2 < (dirx ? F.nx : F.H);
  const Rec n2 = load_rec(F, two ? s + 2 * off : s);
  const double t1 = n1.T, t2 = two ? n2.T : kHugeD;
  const double v1 = fabs(n1.v), v2 = fabs(n2.v);
  Dir d;
  const double dd = div_by(0.5 * (vu + v1), F.dx, rdx);
  const double d2 = dd * dd;
  d.dpos = dirx ? xg(F, c) - xg(F, c + sgn) : zg(F, r) - zg(F, r + sgn);
  const double p = v1 * v2;
  bool second = t2 < kReachD && t1 >= t2 && p > kTinyD;
  // dot >= 0.71/p: away from equality by far more than the rounding of the
  // product and of the quotient, dot*p against 0.71 decides
  const double dot = n1.gx * n2.gx + n1.gz * n2.gz, m = dot * p;
  if (second && !(m > 0.71 * (1.0 + 1.0e-14))) {
    if (m < 0.71 * (1.0 - 1.0e-14)) second = false;
    else second = dot >= 0.71 / p;
  }
  d.T = t1;
  d.T2 = second ? t2 : 0.0;
  d.A = second ? 2.25 * d2 : d2;
  d.B = 0.0 + (second ? -6.0 * t1 + 1.5 * t2 : -2.0 * t1) * d2;
  d.C = (second ? 4.0 * t1 * t1 - 2.0 * t1 * t2 + 0.25 * t2 * t2 : t1 * t1) * d2;
  return d;
}

// The root of reg_cand's quadratic (a, b, c without the - 1), at least tmax;
// without branches on the usual path so that a thread's candidates overlap.
__device__ __forceinline__ bool reg_root(double a, double b, double c, double tmax, double& t) {
  c = c - 1.0;
  bool valid = !(fabs(a) < kTinyD);
  const double det = b * b - 4.0 * a * c;
  // det < 0 counts as 0 when 0.5*sqrt(|det|)/|a| < 1e20, which |det| <= 1e10
  // and |a| >= 1e-10 imply
  if (det < 0.0 && !(det >= -1.0e10 && fabs(a) >= 1.0e-10))
    valid = valid && 0.5 * sqrt(fabs(det)) / fabs(a) < 1.0e20;
  const double t1 = 0.5 * (-b + root(det)) / a;
  t = t1 > tmax ? t1 : tmax;
  return valid;
}

// The best regular candidate: time, event (trigger time; key: 2 * order in the
// reference's quadrant loop + two-sided; a one-sided winner is suspect) and
// the gradient it writes.
struct RegBest {
  double t, trig, gx, gz;
  int key;
};

// act: bit j = quadrant j (X: L R L R, Z: U U D D) is part of the update;
// cut: its order is 32 * cell, cells (R,D) (R,U) (L,D) (L,U), else j (and all
// four are part of it).
template <bool cut>
__device__ __forceinline__ RegBest reg_best(const Fld64& F, double rdx, int s, int r, int c,
                                            double vu, unsigned act) {
  if (!cut) act = 15u;
  const Rec nl = load_rec(F, c > 0 ? s - 1 : s), nr = load_rec(F, c + 1 < F.nx ? s + 1 : s);
  const Rec nu = load_rec(F, r > 0 ? s - F.pitch : s);
  const Rec nd = load_rec(F, r + 1 < F.H ? s + F.pitch : s);
  // (a slot outside the region holds huge_time)
  const double T[4] = {c > 0 && nl.T < kReachD ? nl.T : kHugeD,
                       c + 1 < F.nx && nr.T < kReachD ? nr.T : kHugeD,
                       r > 0 && nu.T < kReachD ? nu.T : kHugeD,
                       r + 1 < F.H && nd.T < kReachD ? nd.T : kHugeD};
  auto time = [&](int k) { return k < 2 ? (k ? T[1] : T[0]) : (k == 3 ? T[3] : T[2]); };
  auto order = [&](int j) { return cut ? 32 * (3 - 2 * (j & 1) - (j >> 1)) : j; };
  auto frozen = [&](int k) {
    const int off = k < 2 ? (k ? 1 : -1) : (k == 3 ? F.pitch : -F.pitch);
    return s + off == F.frozen_slot;
  };
  // order of direction k's one-sided candidate: it is taken in every active
  // quadrant where k is the earlier neighbour, the first of them counts
  auto single_order = [&](int k) {
    int o = kNoKey;
    const double Tk = time(k);
    if (!cut) {
      const int j = k < 2 ? k : 2 * (k - 2);
      if (k < 2 ? Tk <= T[3] : Tk < T[1]) o = k < 2 ? j + 2 : j + 1;
      if (k < 2 ? Tk <= T[2] : Tk < T[0]) o = j;
      return Tk < kReachD && !frozen(k) ? o : kNoKey;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = k < 2 ? k + 2 * h : 2 * (k - 2) + h;
      const double To = k < 2 ? T[2 + h] : T[h];
      if (((act >> j) & 1u) && (k < 2 ? Tk <= To : Tk < To)) o = min(o, order(j));
    }
    return Tk < kReachD && !frozen(k) ? o : kNoKey;
  };
  RegBest b;
  b.t = b.trig = kHugeD;
  b.key = kNoKey;
  double x0 = 0.0, x1 = 0.0, x2 = 1.0, z0 = 0.0, z1 = 0.0, z2 = 1.0;
  bool gxi = false, gzi = false;
  auto single = [&](const Dir& d, bool dirx, int so) {
    double t;
    const bool v = reg_root(d.A, d.B, d.C, d.T, t) && so != kNoKey && t <= kHugeD;
    if (v && before(t, d.T, 2 * so, b.t, b.trig, b.key)) {
      b.t = t;
      b.trig = d.T;
      b.key = 2 * so;
      gxi = dirx;
      gzi = !dirx;
      if (dirx) { x0 = d.T; x1 = d.T2; x2 = d.dpos; }
      else { z0 = d.T; z1 = d.T2; z2 = d.dpos; }
    }
  };
  auto both = [&](const Dir& X, const Dir& Z, bool on, int ord) {
    const double tr = X.T > Z.T ? X.T : Z.T;
    double t;
    const bool v = reg_root(X.A + Z.A, X.B + Z.B, X.C + Z.C, tr, t) && on && t <= kHugeD;
    if (v && before(t, tr, 2 * ord + 1, b.t, b.trig, b.key)) {
      b.t = t;
      b.trig = tr;
      b.key = 2 * ord + 1;
      gxi = gzi = true;
      x0 = X.T; x1 = X.T2; x2 = X.dpos;
      z0 = Z.T; z1 = Z.T2; z2 = Z.dpos;
    }
  };
  // the earlier neighbour of each axis
  const int kx = T[1] < T[0] ? 1 : 0, kz = T[3] < T[2] ? 3 : 2;
  const double TX = T[1] < T[0] ? T[1] : T[0], TZ = T[3] < T[2] ? T[3] : T[2];
  const bool okx = TX < kReachD, okz = TZ < kReachD;
  {
    // (a direction without a neighbour gets the other's terms, not used)
    const int ka = okx ? kx : kz, kb = okz ? kz : kx;
    Dir X, Z;
    if (okx || okz) {
      const Rec nx = T[1] < T[0] ? nr : nl, nz = T[3] < T[2] ? nd : nu;
      X = dir_of(F, rdx, s, r, c, vu, ka, okx ? nx : nz);
      Z = dir_of(F, rdx, s, r, c, vu, kb, okz ? nz : nx);
      const int j = kx + 2 * (kz - 2);
      single(X, true, okx ? single_order(kx) : kNoKey);
      single(Z, false, okz ? single_order(kz) : kNoKey);
      both(X, Z, okx && okz && ((act >> j) & 1u), order(j));
    }
  }
  // the rest: those whose trigger is not above the best time
  const int lx = kx ^ 1, lz = kz ^ 1;
  unsigned left = 0;      // bits 0-1: one-sided lx, lz; 2-4: quadrants (lx,kz) (kx,lz) (lx,lz)
  const double TA = time(lx), TB = time(lz);
  if (TA < kReachD && TA <= b.t) left |= 1u | (okz && TZ <= b.t ? 4u : 0u);
  if (TB < kReachD && TB <= b.t) left |= 2u | (okx && TX <= b.t ? 8u : 0u);
  if ((left & 3u) == 3u) left |= 16u;
  auto again = [&](int k) {
    return dir_of(F, rdx, s, r, c, vu, k,
                  load_rec(F, s + (k < 2 ? (k ? 1 : -1) : (k == 3 ? F.pitch : -F.pitch))));
  };
  while (left) {
    const int q = __ffs(left) - 1;
    left &= left - 1;
    if (q < 2) {
      const int k = q == 0 ? lx : lz, so = single_order(k);
      if (so != kNoKey) single(again(k), k < 2, so);
    } else {
      const int a = q == 3 ? kx : lx, z = q == 2 ? kz : lz, j = a + 2 * (z - 2);
      if ((act >> j) & 1u)
        both(again(a), again(z), true, order(j));
    }
  }
  // grad_of's one-sided first or second-order differences
  const double t = b.t;
  const double nx = gxi ? (x1 == 0.0 ? t - x0 : 0.5 * (3.0 * t - 4.0 * x0 + x1)) : 0.0;
  const double nz = gzi ? (z1 == 0.0 ? t - z0 : 0.5 * (3.0 * t - 4.0 * z0 + z1)) : 0.0;
  b.gx = quot(nx, gxi ? x2 : 1.0);
  b.gz = quot(nz, gzi ? z2 : 1.0);
  return b;
}

// finish for a winner whose gradient is known.
__device__ __forceinline__ NewV settle(const Fld64& F, int s, double t, double gx, double gz,
                                       bool copy, bool sus, double sus_t, const Self& me) {
  Cand c;
  c.t = t;
  c.trig = 0.0;
  c.ord = 0;
  c.kind = kGradGiven;
  c.gxi = c.gzi = false;
  c.sus = false;
  c.copy = copy;
  c.g0 = gx;
  c.g1 = gz;
  c.g2 = c.g3 = c.g4 = c.g5 = 0.0;
  return finish(F, s, c, sus, sus_t, me.fl, me.T, me.g);
}

// ---------------------------------------------------------------- cut cells
// The nodes around a cut node, a lane each: the eight grid neighbours (rows
// above to below, left to right), and the four interface nodes of the two
// columns of cells (top left, top right, bottom left, bottom right).  An
// interface node's: the corners of its cell (column by column, downwards) in
// lanes 0-3, the other interface's node of the column in lane 8.
// Members of connected cell q = (R,D) (R,U) (L,D) (L,U) as those lanes, in the
// reference's connected-node order, four bits each; an interface node's cell
// is the last.
__device__ __forceinline__ unsigned cell_lanes(int k) {
  return k == 0 ? 0x746b9u : k == 1 ? 0x421b9u : k == 2 ? 0x653a8u : k == 3 ? 0x130a8u : 0x32108u;
}
struct CutWork {
  double T[16];
  unsigned char lane[16];    // the members a pair may have
};

// sqrt(d2) < c with c > 0: squares away from c*c by more than the roundings
// decide without the root.
__device__ __forceinline__ bool dist_below(double d2, double c, double c2) {
  if (d2 > c2 * (1.0 + 1.0e-14)) return false;
  if (d2 < c2 * (1.0 - 1.0e-14)) return true;
  return sqrt(d2) < c;
}

// from_2's side tests.  m is the normal (-rz, rx)/l of one member's direction,
// turned towards the other member: w . m <= 0.  The signs do not depend on
// the division by l unless a sum is within its terms' rounding of zero, where
// the reference's expression is evaluated.
struct Side {
  double mx, mz;   // turned, not divided
  bool sure;
  double rx, rz, ox, oz;
};

__device__ __forceinline__ Side side_of(double rx, double rz, double ox, double oz) {
  Side o;
  o.rx = rx; o.rz = rz; o.ox = ox; o.oz = oz;
  const double mx = -rz, mz = rx;
  const double a = mx * ox, b = mz * oz, d = a + b;
  o.sure = fabs(d) > 1.0e-14 * (fabs(a) + fabs(b));
  o.mx = d < 0.0 ? -mx : mx;
  o.mz = d < 0.0 ? -mz : mz;
  return o;
}

__device__ __forceinline__ bool side_in(const Side& s, double wx, double wz) {
  const double a = wx * s.mx, b = wz * s.mz, e = a + b;
  if (s.sure && fabs(e) > 1.0e-14 * (fabs(a) + fabs(b))) return e < 0.0;
  double mx = -s.rz, mz = s.rx;
  const double l = sqrt(mx * mx + mz * mz);
  mx /= l;
  mz /= l;
  if (mx * s.ox + mz * s.oz < 0.0) { mx = -mx; mz = -mz; }
  return wx * mx + wz * mz <= 0.0;
}

__device__ __forceinline__ double half_min(double x) {
#pragma unroll
  for (int o = 8; o; o >>= 1) {
    const double y = __shfl_xor_sync(kFull, x, o);
    x = y < x ? y : x;
  }
  return x;
}

// New value of a node whose candidates need cells cut by an interface (or
// whose surroundings are incomplete), sixteen lanes per node (both halves of a
// warp call it, each with its own node); valid in the lane whose `mine` is
// set.  code: the node's static code (0: nothing to evaluate); rb: its best
// regular candidate.
__device__ __forceinline__ NewV cut_best(const Fld64& F, CutWork& W, int s, int row, int c,
                                         uint32_t code, const RegBest& rb, int lane, bool& mine,
                                         Self& me) {
  const int hl = lane & 15, hb = lane & 16;
  auto half = [&](unsigned ballot) { return (ballot >> hb) & 0xffffu; };
  const bool grid = row < F.H;
  const int side = grid ? 0 : row - F.H;
  const Rec ru = load_rec(F, s);
  me.T = ru.T;
  me.g = make_double2(ru.gx, ru.gz);
  me.fl = F.fl[s];
  int izc = 0;
  if (!grid) izc = FMT_RO(F.izc + side * F.pitch + c);
  const double vu = fabs(ru.v);
  // ---- the nodes around it, all loads at once
  int mrow = -1, mcol = c;
  bool mif = false;      // an interface node (mrow: H + side)
  if (grid) {
    if (hl < 8) {
      const int k = hl < 4 ? hl : hl + 1;     // 3x3 block without its middle
      mrow = row + k / 3 - 1;
      mcol = c + k % 3 - 1;
    } else if (hl < 12) {
      mif = true;
      mrow = F.H + ((hl >> 1) & 1);
      mcol = c - 1 + (hl & 1);
    }
  } else if (hl < 4) {
    mrow = izc < 0 ? -1 : izc - F.z_lo + (hl & 1);
    mcol = c + (hl >> 1);
  } else if (hl == 8 && izc >= 0) {
    mif = true;
    mrow = F.H + (side ^ 1);
  }
  const bool have = mrow >= 0 && (mif || mrow < F.H) && mcol >= 0 && mcol < F.nx;
  double mT = kHugeD, mx = 0.0, mz = 0.0, mv = 1.0;
  double2 mg = make_double2(0.0, 0.0);
  bool copied = false, single = true;
  if (have) {
    const int ms = mrow * F.pitch + mcol;
    const Rec m = load_rec(F, ms);
    mT = m.T;
    mg = make_double2(m.gx, m.gz);
    mv = fabs(m.v);
    copied = (F.fl[ms] & kFlCopy) != 0;
    if (mif) {
      mx = FMT_RO(F.ifx + mcol);
      mz = FMT_RO(F.ifz + (mrow - F.H) * F.pitch + mcol);
    } else {
      mx = xg(F, mcol);
      mz = zg(F, mrow);
      single = ms != F.frozen_slot;
    }
  }
  const double xu = grid ? xg(F, c) : FMT_RO(F.ifx + c);
  const double zu = grid ? zg(F, row) : FMT_RO(F.ifz + side * F.pitch + c);
  // ---- which cut cells they are members of, and of which first
  const unsigned cells = grid ? (code >> 4) & (code >> 8) & 15u : 1u;   // connected, cut
  unsigned in = 0;     // cells that hold this lane's node
  if (grid) {
    if (hl < 8) in = (0x1543c2a8u >> (4 * hl)) & 15u;
    else if (hl < 12) in = (hl & 1 ? 3u : 12u) & (hl < 10 ? code >> 12 : code >> 16);
    in &= cells;
  } else if (hl < 4 || (hl == 8 && (code & (1u << (side ? 12 : 16))))) {
    in = 1u;
  }
  const int cell0 = in ? __ffs(in) - 1 : 8;
  // place of a lane's node in a cell's connected-node order
  auto place_in = [&](int cell, int l) {
    const unsigned tab = cell_lanes(grid ? cell : 4);
    int p = 0;
#pragma unroll
    for (int m = 1; m < 5; ++m)
      if (((tab >> (4 * m)) & 15u) == (unsigned)l) p = m;
    return p;
  };
  const bool member = cell0 < 8 && mT < kReachD;
  const int rord = rb.key == kNoKey ? kNoKey : rb.key >> 1;
  const bool rsus = rb.key != kNoKey && !(rb.key & 1);   // a one-sided update is suspect
  // (interface nodes have no regular update: nothing precedes, nothing is suspect)
  // ---- one-sided events, a lane per member (in its first cell: its events in
  // the others have the same value and come later).  A lane's best event:
  double ot = kHugeD, otrig = kHugeD, g0 = 0.0, g1 = 0.0, g2 = 1.0;
  int okey = kNoKey;
  uint8_t kind = kGradNone;
  bool copy = false;
  bool pre = false;      // an event ahead of the regular one at or below its time
  auto offer = [&](double t, double trig, int key, int ord) -> bool {
    if (rsus && t <= rb.t && (trig < rb.trig || (trig == rb.trig && ord < rord))) pre = true;
    if (!(t <= kHugeD) || !before(t, trig, key, ot, otrig, okey)) return false;
    ot = t;
    otrig = trig;
    okey = key;
    return true;
  };
  const double tol1 = 0.01 * F.tol, tol2 = tol1 * tol1;
  bool close = false;
  if (member) {
    const double dxu = xu - mx, dzu = zu - mz;
    const double dist = root(dxu * dxu + dzu * dzu);
    close = dist < tol1;
    const int key = (cell0 * 32 * 8 + place_in(cell0, hl)) * 2;
    const double t = close ? mT : mT + quot(dist, 0.5 * (vu + mv));
    if (single && !(close && copied) && offer(t, mT, key, cell0 * 32)) {
      kind = close ? kGradGiven : kGradRay;
      copy = close;
      g0 = close ? mg.x : dxu;
      g1 = close ? mg.y : dzu;
      g2 = dist * vu;
    }
  }
  double ct = half_min(ot);
  const double bound = rb.t < ct ? rb.t : ct;
  // ---- plane-front events.  Both members of a pair that can matter are
  // within the bound (its trigger is, and the other is earlier), or the
  // earlier one is the fixed source node on this node, which has no one-sided
  // event of its own.  Of a pair in two cells the first cell's event counts:
  // the other has the same value and comes later.
  const unsigned singlem = half(__ballot_sync(kFull, single));
  const unsigned closem = half(__ballot_sync(kFull, close));
  const unsigned okm = half(__ballot_sync(kFull, member));
  const unsigned odd = closem & okm & ~singlem;
  const unsigned within = half(__ballot_sync(kFull, member && mT <= bound));
  const unsigned due = odd ? okm : within;
  const int ndue = __popc(due), npair = ndue * (ndue - 1) / 2;
  if (__any_sync(kFull, npair > 0)) {
    W.T[hl] = member ? mT : kHugeD;
    if ((due >> hl) & 1u) W.lane[__popc(due & ((1u << hl) - 1u))] = (unsigned char)hl;
    const unsigned copym = half(__ballot_sync(kFull, copied));
    __syncwarp();
    const int np2 = __shfl_xor_sync(kFull, npair, 16), most = npair > np2 ? npair : np2;
    // (both halves go round together: the loop's end is the same for the warp,
    // and no lane leaves its body early)
    for (int b = 0; b < most; b += 16) {
      // pair k = (i, j), i < j, of the due members
      const int k = b + hl < npair ? b + hl : 0;
      const int j = (int)(0.5f * (1.0f + sqrtf(8.0f * (float)k + 1.0f))), i = k - j * (j - 1) / 2;
      int l1 = npair > 0 ? W.lane[j] : 0, l2 = npair > 0 ? W.lane[i] : 0;
      const unsigned shared = (unsigned)__shfl_sync(kFull, (int)in, hb + l1) &
                              (unsigned)__shfl_sync(kFull, (int)in, hb + l2);
      const int cell = shared ? __ffs(shared) - 1 : 0;
      int p = place_in(cell, l1), u = place_in(cell, l2);
      // the later accepted one triggers
      const double Ta = W.T[l1], Tb = W.T[l2];
      if (Ta < Tb || (Ta == Tb && p < u)) {
        int x = l1; l1 = l2; l2 = x;
        x = p; p = u; u = x;
      }
      // a trigger on the node hands its values over as its one-sided event
      // did; an earlier member on the node likewise, unless it triggers none
      const bool live = b + hl < npair && shared && ((singlem >> l1) & 1u) &&
                        !((closem >> l1) & 1u) &&
                        (((closem >> l2) & 1u) ? !((singlem >> l2) & 1u) : W.T[l1] <= bound);
      const unsigned tab = cell_lanes(grid ? cell : 4);
      const double T1 = shfl(mT, hb + l1), x1 = shfl(mx, hb + l1), z1 = shfl(mz, hb + l1);
      const double T2 = shfl(mT, hb + l2), x2 = shfl(mx, hb + l2), z2 = shfl(mz, hb + l2);
      const double v1 = shfl(mv, hb + l1), v2 = shfl(mv, hb + l2);
      const double g2x = shfl(mg.x, hb + l2), g2z = shfl(mg.y, hb + l2);
      if (live) {
        // place of the pair in the events of trigger p: the members accepted
        // by then in their order, p swapped to the front
        int pp = 0, uu = 0;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          const bool is = !grid || m > 1 || (code & (1u << ((m ? 16 : 12) + cell)));
          const double Tm = W.T[(tab >> (4 * m)) & 15];
          const bool up = is && Tm < kReachD && (Tm < T1 || (Tm == T1 && m <= p));
          pp += up && m < p;
          uu += up && m < u;
        }
        const int ord = cell * 32 + (uu == 0 ? pp : uu);
        const int key = (ord * 8 + p) * 2;
        const double ex = x2 - x1, ez = z2 - z1;
        if ((closem >> l2) & 1u) {
          if (!((copym >> l2) & 1u) && offer(T2, T1, key, ord)) {
            kind = kGradGiven;
            copy = true;
            g0 = g2x;
            g1 = g2z;
          }
        } else if (!dist_below(ex * ex + ez * ez, tol1, tol2)) {
          // (coincident members: time_from_1 of the trigger again, a later
          // event of the same value)
          const double r1x = x1 - xu, r1z = z1 - zu, r2x = x2 - xu, r2z = z2 - zu;
          const double v12 = 0.5 * (v1 + v2);
          const double dx_ = quot(x1 - x2, v12), dz_ = quot(z1 - z2, v12);
          const double dd = dx_ * dx_ + dz_ * dz_;
          const double tq = quot(T1 - T2, dd);
          const double px = tq * dx_, pz = tq * dz_;
          const double qx = -dz_, qz = dx_;
          const double ae = qx * qx + qz * qz;
          const double be = 2.0 * (px * qx + pz * qz);
          const double ce = px * px + pz * pz - 1.0;
          const double det = be * be - 4.0 * ae * ce;
          if (!(det < 0.0)) {
            const double sq = root(det);
            const Side s1 = side_of(r1x, r1z, r2x, r2z), s2 = side_of(r2x, r2z, r1x, r1z);
            const double ua = quot(0.5 * (-be + sq), ae), ub = quot(0.5 * (-be - sq), ae);
            const double wax = px + ua * qx, waz = pz + ua * qz;
            const double wbx = px + ub * qx, wbz = pz + ub * qz;
            const bool ia = side_in(s1, wax, waz) && side_in(s2, wax, waz);
            const bool ib = side_in(s1, wbx, wbz) && side_in(s2, wbx, wbz);
            const double vm = 0.5 * (vu + v1);
            const double ta = T1 - quot(wax * r1x + waz * r1z, vm);
            const double tb = T1 - quot(wbx * r1x + wbz * r1z, vm);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const double at = h == 0 ? ta : tb;
              if ((h == 0 ? ia : ib) && at >= T1 && offer(at, T1, key + h, ord)) {
                kind = kGradPlane;
                copy = false;
                g0 = h == 0 ? wax : wbx;
                g1 = h == 0 ? waz : wbz;
                g2 = v1;
              }
            }
          }
        }
      }
      __syncwarp();
    }
    __syncwarp();
    ct = half_min(ot);
  }
  // ---- the cut cells' best event, and the regular one against it
  unsigned win = half(__ballot_sync(kFull, okey != kNoKey && ot == ct));
  if (__any_sync(kFull, (win & (win - 1u)) != 0u)) {   // equal times: the earlier event
    double tr = okey != kNoKey && ot == ct ? otrig : kHugeD;
    int k = okey != kNoKey && ot == ct ? okey : kNoKey;
#pragma unroll
    for (int o = 8; o; o >>= 1) {
      const double t2 = __shfl_xor_sync(kFull, tr, o);
      const int k2 = __shfl_xor_sync(kFull, k, o);
      if (k2 != kNoKey && (k == kNoKey || t2 < tr || (t2 == tr && k2 < k))) {
        tr = t2;
        k = k2;
      }
    }
    win = half(__ballot_sync(kFull, okey != kNoKey && okey == k && ot == ct && otrig == tr));
  }
  const int wl = win ? __ffs(win) - 1 : 0;
  const double ctr = shfl(otrig, hb + wl);
  const int ckey = __shfl_sync(kFull, okey, hb + wl);
  const int cord = ckey == kNoKey ? kNoKey : ckey >> 4;
  const bool reg_wins =
      rb.t < ct || (rb.t == ct && (rb.trig < ctr || (rb.trig == ctr && rord < cord)));
  const bool anypre = half(__ballot_sync(kFull, pre)) != 0u;
  mine = hl == wl;
  NewV none;
  none.write = none.spread = false;
  if (!mine || (!grid && izc < 0) || code == 0u) return none;
  double gx = rb.gx, gz = rb.gz;
  if (!reg_wins) {
    gx = gz = 0.0;
    if (kind == kGradGiven) {   // handed over as it is (it may be a NaN)
      gx = g0;
      gz = g1;
    } else if (kind != kGradNone) {
      // time_from_1: / (dist * v); time_from_2: / (|w| * v)
      const double den = kind == kGradPlane ? sqrt(g0 * g0 + g1 * g1) * g2 : g2;
      gx = quot(g0, den);
      gz = quot(g1, den);
    }
  }
  return settle(F, s, reg_wins ? rb.t : ct, gx, gz, !reg_wins && copy,
                rsus && (reg_wins || !anypre), rb.t, me);
}

}  // namespace ev
}  // namespace fmt2d
