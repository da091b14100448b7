// FP64 eikonal solver: the reference's fast-marching stencil solved to its
// fixed point by data-parallel relaxation, one thread block per time field.
//
// The candidate arithmetic (eik_eval.cuh) gives every node the smallest of
// its seed and of the candidate times its fast-marching update events
// produce.  The solve is a fast iterative method over a field's active list:
// each step evaluates every listed node once, commits the new values and lists
// the nodes a changed node can move.  A time window
// bounds what may be committed: a node whose new time lies beyond it waits
// (it records the time and stays listed; until an input changes or the
// window reaches that time, listing it costs a compare), and the window moves
// on only after a step in which nothing inside it changed, so nodes settle in
// time slices as the heap accepts them.  When the list is empty every node is
// at the fixed point; a separate check of every node (k_verify) re-lists any
// that is not.
//
// One thread block owns a field for the whole solve: the lists, the
// "listed" bitset and the window live in shared memory, steps are separated
// by block barriers instead of kernel launches, and the field's front stays
// in the SM's L1.  A step's phases are separated by barriers: evaluate the
// regular quadrants, evaluate the cut cells (both read committed state only
// and stage new values), arbitrate and commit, spread.  Evaluations never see
// a value of the same step, so the result does not depend on thread timing or
// block size: a forward is bit-identical run to run.
//
// Arithmetic is FP64 with the reference's expression order; this file is
// compiled with --fmad=false so candidate times are bit-identical to the
// FP64 restatement's.
#include <math_constants.h>
#include <algorithm>
#include <climits>
#include <mutex>
#include "eik64.cuh"
#include "eik_coop.cuh"
#include "model.h"

namespace fmt2d {

namespace {

using namespace ev;

// ---------------------------------------------------------------- field solve
// Threads of a field's solve block: k_solve is instantiated for each size;
// the result does not depend on it (no evaluation sees a value of its own
// step), only the time does, so a context may pick the fastest for its
// workload (e64_solve_sizes, fmt2d_autotune).
constexpr int kSolveSizes[3] = {256, 384, 512};
constexpr int kSolveDefault = 384;
constexpr unsigned kLCap = 2048;          // regular nodes of each list held in shared memory
constexpr unsigned kXCap = 512;           // nodes next to an interface, likewise
constexpr unsigned kXBatch = 256;         // of those, evaluated between two barriers
constexpr unsigned kCCap = 512;           // commits held in shared memory
constexpr int kTileRows = 8;              // a tile: 8 slot rows x 32 slot columns (one bitset word per row)
constexpr int kTilesMax = 12288;          // tiles per field (tile minima live in shared memory)
constexpr size_t kSmemMax = 227 * 1024;   // dynamic shared memory of the solve block
constexpr unsigned kSpreadBit = 0x80000000u;   // commit entry: the node moved
constexpr unsigned kCutBit = 0x40000000u;      // commit entry: next to an interface
constexpr unsigned kSlotMask = 0x3fffffffu;
constexpr unsigned long long kNone = ULLONG_MAX;

struct SolveShared {
  Fld64 F;
  unsigned cnt[2][2];              // list lengths: [list][regular, next to an interface]
  unsigned nc;                     // commits
  unsigned nw[2];                  // commits that moved a node (winners): regular, others
  int changed[2];                  // a node moved, by step parity
  int any[2];                      // a node was listed, by step parity
  unsigned nready[2];              // tiles to release, by release parity
  int released[2];                 // a release listed a node, by release parity
  unsigned long long gmin[2];      // earliest waiting time (bits of a positive double)
  int err;
  long long c0;                    // thread 0: cycles per phase
  unsigned long long cyc[5], steps_cut;
};

__device__ __forceinline__ unsigned long long dbits(double d) {
  return (unsigned long long)__double_as_longlong(d);
}

__host__ __device__ inline int tiles_of(const Fld64& F) {
  return ((F.H + 2 + kTileRows - 1) / kTileRows) * (F.pitch / 32);
}

// Shared-memory plan of a solve launch.
struct SolvePlan {
  int bits;        // words of a bitset over the slots of the largest field
  int nbits;       // bitsets in shared memory: 1 listed, 2 and waiting
  int tiles;       // tiles of the largest field if a field has a window, else 0
  int mwords;      // moving bitmap: words per row (a power of two), and in all
  int mtotal;
  unsigned rmask;  // its rows: slot row & rmask
};

// Solve every field of the batch from its list_in (one block per field).
//
// A list holds its regular nodes and its nodes next to an interface apart: a
// thread evaluates one of the former or the regular quadrants of one of the
// latter, then sixteen lanes evaluate a node's cut cells (eik_coop.cuh).
//
// The nodes that move in a step mark a small bitmap (rows modulo rmask + 1,
// columns modulo 32 * mwords) and claim their new time in global memory with the
// step's stamp; a node looks up only the claims of marked neighbours, and the
// stamp tells a mark of another row, column or step.
//
// Waiting nodes: a node whose new time lies beyond the window records it in
// pend and sets its bit in the waiting bitset; each tile of 8 x 32 slots
// keeps the smallest waiting time of its nodes.  When the window moves on,
// the tiles it has reached are scanned (a warp per tile) and their nodes
// that are due are listed, so a waiting node costs nothing until then.  A
// waiting node whose input changes is listed at once (its recorded time was
// computed from the old value).
//
// What bounds it: a step's chain of instructions (a warp runs each phase once
// or twice a step, at about 8 cycles an instruction) times the steps of a
// field.  2001x401, Pg+PmP, 30 sources: 15 us a step (51 us with a thread per
// node and three arrays), 0.193 s a forward (0.72 s).  384 threads: 256 give
// 0.202 s (too few warps for a front of 300 nodes), 512 give 0.229 s (128
// registers, spills).  A cluster of blocks per field was tried and was slower
// where it was compared, with an earlier form of the evaluation (1 source:
// 0.18 s with 8 blocks per field against 0.15 s now with one): a cluster
// barrier that publishes global stores takes 1600 cycles against 45 for the
// block's own.
template <int kSolveThreads>
__global__ void __launch_bounds__(kSolveThreads, 1)
    k_solve(Fld64* fields, SolvePlan P, long long max_steps, unsigned long long* ctr) {
  constexpr int kWarps = kSolveThreads / 32;
  extern __shared__ __align__(16) unsigned char dsm_raw[];
  __shared__ SolveShared sh;
  __shared__ CutWork cutw[2 * kWarps];
  // regular candidates of the nodes next to an interface, by place in the batch
  __shared__ RegBest xrb[kXBatch];
  __shared__ uint32_t xcode[kXBatch];
  // commits: slot and flags, new and old time, gradient, flags; winners
  __shared__ unsigned ce[kCCap];
  __shared__ double cT[kCCap], co[kCCap], cgx[kCCap], cgz[kCCap];
  __shared__ uint8_t cf[kCCap];
  __shared__ unsigned short cw[kCCap];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    sh.F = fields[blockIdx.x];
    for (int k = 0; k < 2; ++k) {
      sh.cnt[k][0] = sh.cnt[k][1] = 0u;
      sh.changed[k] = sh.any[k] = sh.released[k] = 0;
      sh.nready[k] = 0u;
      sh.gmin[k] = kNone;
    }
    sh.nc = sh.nw[0] = sh.nw[1] = 0u;
    sh.err = 0;
    for (int k = 0; k < 5; ++k) sh.cyc[k] = 0;
    sh.steps_cut = 0;
  }
  __syncthreads();
  const Fld64& F = sh.F;
  const unsigned pitch = (unsigned)F.pitch;
  const double rdx = 1.0 / F.dx;
  const unsigned ns = (unsigned)F.nslots();
  const unsigned nbw = (ns + 31u) >> 5;
  const int tcols = F.pitch / 32, ntiles = tiles_of(F);
  // row of a slot: s / pitch for s < 2^30 by a multiplication (the quotient is
  // exact because the multiplier's error times 2^30 stays below one)
  const int mshift = 30 + (32 - __clz((int)pitch - 1));
  const unsigned long long mmul = ((1ull << mshift) + pitch - 1) / pitch;
  auto row_of = [&](unsigned s) { return (int)(((unsigned long long)s * mmul) >> mshift); };
  unsigned long long* tmin = reinterpret_cast<unsigned long long*>(dsm_raw);
  unsigned* sx = reinterpret_cast<unsigned*>(tmin + P.tiles);   // [2][kXCap]
  unsigned* sl = sx + 2 * kXCap;                                // [2][kLCap]
  unsigned short* ready = reinterpret_cast<unsigned short*>(sl + 2 * kLCap);
  unsigned* mbits = reinterpret_cast<unsigned*>(ready + P.tiles);
  unsigned* sbits = mbits + P.mtotal;
  unsigned* bits = P.nbits >= 1 ? sbits : F.inq;
  unsigned* wbits = P.nbits >= 2 ? sbits + P.bits : F.wait;
  const unsigned mmask = (unsigned)P.mwords - 1u;
  // lists: regular nodes overflow to the front of the list's part of over,
  // the others to its back (together at most the field's slots)
  // (the start list has been read when the first commit is made)
  unsigned* cov = F.list_in;
  // a field without a window never holds a node back: nothing waits
  const bool windowed = F.clock[1] < kReachD;
  // The collective steps below are called by whole warps: places in a list or
  // the commits for the lanes that want one (one atomic per warp).
  auto place = [&](unsigned* n, bool want) -> unsigned {
    const unsigned m = __ballot_sync(kFull, want);
    if (!m) return 0u;
    unsigned p = 0;
    const int first = __ffs(m) - 1;
    if (lane == first) p = atomicAdd(n, (unsigned)__popc(m));
    return __shfl_sync(kFull, p, first) + __popc(m & ((1u << lane) - 1u));
  };
  auto put = [&](int l, bool regular, unsigned s, unsigned p) {
    if (regular) {
      if (p < kLCap) sl[l * kLCap + p] = s;
      else F.over[l * (size_t)ns + (p - kLCap)] = s;
    } else {
      if (p < kXCap) sx[l * kXCap + p] = s;
      else F.over[l * (size_t)ns + (ns - 1 - (p - kXCap))] = s;
    }
  };
  // List the wanting lanes' slots s in list l unless they are listed already.
  auto push = [&](int l, unsigned s, bool regular, bool want) {
    if (want) {
      const unsigned bit = 1u << (s & 31);
      want = !(atomicOr(bits + (s >> 5), bit) & bit);
    }
    const unsigned p = place(&sh.cnt[l][0], want && regular);
    if (want && regular) put(l, true, s, p);
    const unsigned x = place(&sh.cnt[l][1], want && !regular);
    if (want && !regular) put(l, false, s, x);
  };
  constexpr uint32_t kPlain = kInRegion | kUpdatable | kFullyRegular;
  auto plain = [&](unsigned s) { return (FMT_RO(F.code + s) & kPlain) == kPlain; };
  auto waits = [&](unsigned w) { return P.nbits >= 2 ? wbits[w] : __ldcg(wbits + w); };
  auto xentry = [&](int l, unsigned i) {
    return i < kXCap ? sx[l * kXCap + i] : F.over[l * (size_t)ns + (ns - 1 - (i - kXCap))];
  };
  for (unsigned w = tid; w < nbw; w += kSolveThreads) {
    bits[w] = 0u;
    if (windowed) wbits[w] = 0u;
  }
  for (int w = tid; w < P.mtotal; w += kSolveThreads) mbits[w] = 0u;
  if (windowed)
    for (int t = tid; t < ntiles; t += kSolveThreads) tmin[t] = kNone;
  __syncthreads();
  const unsigned n0 = F.cnt[0];
  for (unsigned i = tid; i - lane < n0; i += kSolveThreads) {
    const bool live = i < n0;
    const unsigned s = live ? F.list_in[i] : 0u;
    push(0, s, live && plain(s), live);
  }
  double W = F.clock[0];
  const double wstep = F.clock[1];
  // claims of earlier solves of this field carry smaller steps
  const unsigned long long stamp0 = dbits(F.clock[2]) + 1;
  // this thread's counts (a warp's sum stays below 2^32: it evaluates a node
  // in microseconds)
  unsigned n_eval = 0, n_write = 0, n_rel = 0, n_cut = 0;
  __syncthreads();
  if (tid == 0) sh.c0 = clock64();
  auto lap = [&](int k) {   // (thread 0)
    const long long c1 = clock64();
    sh.cyc[k] += (unsigned long long)(c1 - sh.c0);
    sh.c0 = c1;
  };
  int cur = 0, rp = 0;
  long long it = 0;
  bool more = n0 != 0u;
  for (; more; ++it) {
    if (it >= max_steps) {
      if (tid == 0) sh.err = 1;
      break;
    }
    const int par = (int)(it & 1), nxt = cur ^ 1;
    const unsigned long long stamp = stamp0 + (unsigned long long)it;
    // evaluate: read committed state only, stage what changes (collective; on:
    // the lane holds node s's new value)
    auto stage = [&](bool on, unsigned s, unsigned cut, const NewV& nv, const Self& me) {
      bool commit = false;
      if (on) {
        atomicAnd(bits + (s >> 5), ~(1u << (s & 31)));
        ++n_eval;
        if (!nv.write) {
          if (windowed) F.pend[s] = -1.0;
        } else if (nv.T < kReachD && nv.T > W) {   // beyond the window: wait for it
          F.pend[s] = nv.T;
          atomicOr(wbits + (s >> 5), 1u << (s & 31));
          const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
          atomicMin(tmin + (row / kTileRows) * tcols + (col >> 5), dbits(nv.T));
        } else {
          if (windowed) F.pend[s] = -1.0;
          commit = true;
        }
      }
      const unsigned p = place(&sh.nc, commit);
      if (!commit) return;
      const uint8_t fl =
          (uint8_t)((me.fl & kFlSeed) | (nv.copy ? kFlCopy : 0) | (nv.sus ? kFlSusp : 0));
      const unsigned e = s | cut | (nv.spread ? kSpreadBit : 0u);
      if (p < kCCap) {
        ce[p] = e;
        cT[p] = nv.T;
        co[p] = me.T;
        cgx[p] = nv.gx;
        cgz[p] = nv.gz;
        cf[p] = fl;
      } else {
        cov[p - kCCap] = e;
        F.Tn[s] = nv.T;
        F.Gn[s] = make_double2(nv.gx, nv.gz);
        F.fln[s] = fl;
      }
      if (nv.spread) {
        sh.changed[par] = 1;
        F.claim[s] = make_ulonglong2(dbits(nv.T), stamp);
        const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
        atomicOr(mbits + ((unsigned)row & P.rmask) * P.mwords + ((col >> 5) & mmask), 1u << (col & 31));
      }
    };
    const unsigned nr = sh.cnt[cur][0], nx = sh.cnt[cur][1];
    for (unsigned x0 = 0;; x0 += kXBatch) {
      // (the nodes next to an interface first, in warps of their own)
      const unsigned xn = min(nx - x0, kXBatch), xpad = (xn + 31u) & ~31u;
      const unsigned n = xpad + (x0 == 0 ? nr : 0u);
      for (unsigned i = tid; i - lane < n; i += kSolveThreads) {
        const bool cut = i < xpad;          // (the same in a whole warp)
        const bool live = cut ? i < xn : i < n;
        const unsigned k = live ? (cut ? x0 + i : i - xpad) : 0u;
        const unsigned s = cut ? xentry(cur, k)
                               : k < kLCap ? sl[cur * kLCap + k] : F.over[cur * (size_t)ns + (k - kLCap)];
        const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
        const Rec me = load_rec(F, (int)s);
        uint32_t code = kPlain;
        unsigned act = 15u;
        uint8_t fl = 0;
        if (cut) {
          code = FMT_RO(F.code + s);
          // a node that is not updated has nothing to evaluate
          if (!(code & kInRegion) || !(code & kUpdatable) || (int)s == F.frozen_slot) code = 0u;
          // cells (R,D) (R,U) (L,D) (L,U) to quadrants (L,U) (R,U) (L,D) (R,D)
          const unsigned q = row < F.H ? (code >> 4) & ~(code >> 8) & 15u : 0u;
          act = (q >> 3) | (q & 6u) | ((q & 1u) << 3);
        } else {
          fl = F.fl[s];
          if ((int)s == F.frozen_slot) act = 0u;
        }
        RegBest rb;
        rb.t = rb.trig = kHugeD;
        rb.gx = rb.gz = 0.0;
        rb.key = kNoKey;
        if (cut) {
          if (act && live) rb = reg_best<true>(F, rdx, (int)s, row, col, fabs(me.v), act);
          if (live) {
            xrb[i] = rb;
            xcode[i] = code;
          }
        } else {
          Self self;
          self.T = me.T;
          self.g = make_double2(me.gx, me.gz);
          self.fl = fl;
          NewV nv;
          nv.write = nv.spread = false;
          if (act && live) {
            rb = reg_best<false>(F, rdx, (int)s, row, col, fabs(me.v), act);
            nv = settle(F, (int)s, rb.t, rb.gx, rb.gz, false, rb.key != kNoKey && !(rb.key & 1),
                        rb.t, self);
          }
          stage(live, s, 0u, nv, self);
        }
      }
      __syncthreads();
      for (unsigned b = 2u * warp; b < xn; b += 2u * kWarps) {
        const unsigned i = b + (lane >> 4), ii = i < xn ? i : b;
        const unsigned s = xentry(cur, x0 + ii);
        const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
        bool mine;
        Self me;
        const NewV nv = cut_best(F, cutw[2 * warp + (lane >> 4)], (int)s, row, col, xcode[ii],
                                 xrb[ii], lane, mine, me);
        const bool on = mine && i < xn;
        n_cut += on;
        stage(on, s, kCutBit, nv, me);
      }
      __syncthreads();
      if (x0 + kXBatch >= nx) break;
    }
    if (tid == 0) {
      const unsigned long long e0 = sh.cyc[0];
      lap(0);
      if (nx) {
        sh.cyc[2] += sh.cyc[0] - e0;
        ++sh.steps_cut;
      }
    }
    // arbitrate: a moving node commits only if no node that reads it (the
    // nodes it reads are among them) moves to a smaller (time, slot) in the
    // same step; the others are listed again.  Of two nodes that feed each
    // other the earlier goes first, as the heap accepts them, so a pair that
    // hands a time back and forth (a zero-increment update) cannot swap
    // values forever.
    const unsigned nc = sh.nc;
    if (tid == 0) {
      sh.cnt[cur][0] = sh.cnt[cur][1] = 0u;
      sh.changed[par ^ 1] = 0;
      sh.any[par ^ 1] = 0;
    }
    // (a thread per moved node: it reads the marks around it, then the claims
    // of the marked ones; a winner commits at once, nothing reads committed
    // times in this phase; its old time is kept for the spread threshold)
    for (unsigned j = tid; j - lane < nc; j += kSolveThreads) {
      const bool in_sh = j < kCCap, live = j < nc;
      const unsigned e = live ? (in_sh ? ce[j] : cov[j - kCCap]) : 0u;
      const unsigned s = e & kSlotMask;
      const double Tn = live ? (in_sh ? cT[j] : F.Tn[s]) : 0.0;
      bool lose = false;
      if (e & kSpreadBit) {
        const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
        const unsigned long long ks = dbits(Tn);
        // marks of columns c0 .. c0 + 4 of a slot row
        auto marks = [&](int r, unsigned which) -> unsigned long long {
          if (r < 0 || r >= F.H + 2) return 0ull;
          const unsigned* m = mbits + ((unsigned)r & P.rmask) * P.mwords;
          const int c0 = col - 2, w = c0 >> 5;
          return __funnelshift_r(m[w & mmask], m[(w + 1) & mmask], c0 & 31) & which;
        };
        // the marked ones: five columns each of up to seven rows ra .. ra + 4, rb, rb + 1
        unsigned long long mask;
        int ra, rb;
        if (row < F.H) {
          // second neighbours along the axes, the 3x3 block, and the interface
          // nodes of the columns of cells on both sides
          ra = row - 2;
          rb = F.H;
          mask = marks(row, 27u) << 10 | marks(row - 1, 14u) << 5 | marks(row - 2, 4u);
          if (row + 1 < F.H) mask |= marks(row + 1, 14u) << 15;
          if (row + 2 < F.H) mask |= marks(row + 2, 4u) << 20;
          mask |= marks(rb, 6u) << 25 | marks(rb + 1, 6u) << 30;
        } else {
          const int side = row - F.H;
          const int izc = FMT_RO(F.izc + side * F.pitch + col);
          ra = F.H + (side ^ 1);
          rb = izc - F.z_lo;
          mask = marks(ra, 4u);
          if (izc >= 0 && rb < F.H) mask |= marks(rb, 12u) << 25;
          if (izc >= 0 && rb + 1 < F.H) mask |= marks(rb + 1, 12u) << 30;
        }
        while (mask && !lose) {
          const int b = __ffsll((long long)mask) - 1;
          mask &= mask - 1;
          const int i = (b * 205) >> 10, c = col - 2 + b - 5 * i;
          if (c < 0 || c >= F.nx) continue;
          const unsigned t = (unsigned)(i < 5 ? ra + i : rb + i - 5) * pitch + (unsigned)c;
          const ulonglong2 k = F.claim[t];
          lose = k.y == stamp && (k.x < ks || (k.x == ks && t < s));
        }
      }
      if (lose) sh.any[par] = 1;
      push(nxt, s, !(e & kCutBit), lose);
      const bool win = live && !lose && (e & kSpreadBit);
      const bool wreg = win && in_sh && !(e & kCutBit), wcut = win && in_sh && (e & kCutBit);
      const unsigned w = place(&sh.nw[0], wreg), wx = place(&sh.nw[1], wcut);
      if (live && !lose) {
        double* const rec = reinterpret_cast<double*>(F.R + s);
        const double old = in_sh ? co[j] : rec[0];
        rec[0] = Tn;
        *reinterpret_cast<double2*>(rec + 2) = in_sh ? make_double2(cgx[j], cgz[j]) : F.Gn[s];
        F.fl[s] = in_sh ? cf[j] : F.fln[s];
        if (win) {
          ++n_write;
          if (in_sh) {
            co[j] = fmin(old, Tn);
            cw[wreg ? w : kCCap - 1 - wx] = (unsigned short)j;
          } else {
            F.Tn[s] = fmin(old, Tn);
          }
        }
      }
      // (beyond shared memory the entry itself tells the winners: their only flag
      // is kSpreadBit)
      if (live && !in_sh) cov[j - kCCap] = lose ? s | kCutBit : e & ~kCutBit;
    }
    __syncthreads();
    if (tid == 0) {
      // (all have read it before this barrier; the next commits come after the
      // one that ends the step)
      sh.nc = 0;
      lap(1);
    }
    // spread: every candidate of a node u that involves node v is at or above
    // v's time, so a change of v from a to b can only move nodes at or above
    // min(a, b); those below are not listed unless they wait with a time
    // computed from the old value, which is dropped.  A node that passes this
    // test without reading s counts for the window (any), but is not listed:
    // its evaluation would change nothing
    // A regular winner is a corner of no cut cell, so only grid nodes read it:
    // four lanes each take its neighbour along an axis, the one behind that and
    // a diagonal one
    const unsigned nw = sh.nw[0], nwx = sh.nw[1], no = nc > kCCap ? nc - kCCap : 0u;
    for (unsigned k = tid; k - lane < 4u * nw; k += kSolveThreads) {
      const bool live = (k >> 2) < nw;
      const unsigned j = cw[live ? k >> 2 : 0u];
      const int d = (int)(k & 3u), sgn = (d & 1) ? 1 : -1;
      const unsigned s = ce[j] & kSlotMask;
      const double thr = co[j];
      const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
      const int dr = d < 2 ? 0 : sgn, dc = d < 2 ? sgn : 0;
      // (diagonal: (-1,-1) (-1,1) (1,-1) (1,1))
      const int rr[3] = {row + dr, row + 2 * dr, row + (d < 2 ? -1 : 1)};
      const int cc[3] = {col + dc, col + 2 * dc, col + sgn};
      unsigned t[3];
      double2 tv[3];
      bool want[3];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        want[h] = live && rr[h] >= 0 && rr[h] < F.H && cc[h] >= 0 && cc[h] < F.nx;
        t[h] = want[h] ? (unsigned)(rr[h] * (int)pitch + cc[h]) : s;
        tv[h] = *reinterpret_cast<const double2*>(F.R + t[h]);
      }
      bool any = false;
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        // (a velocity of zero: outside the region, unless the code says otherwise)
        if (want[h] && tv[h].y == 0.0) want[h] = (FMT_RO(F.code + t[h]) & kInRegion) != 0u;
        // a waiting target (its bit may be stale) drops the time it waits with
        const bool waiting = want[h] && windowed && ((waits(t[h] >> 5) >> (t[h] & 31)) & 1u);
        want[h] = want[h] && (waiting || !(tv[h].x < thr));
        any |= want[h];
        // of those, the nodes whose update reads s: a second neighbour only
        // behind a reached neighbour that is not earlier than s (T2 <= T1, at
        // its old or new time), a diagonal one only through a cut cell
        if (h == 1) want[h] = want[h] && tv[0].x < kReachD && tv[0].x >= thr;
        if (h == 2) want[h] = want[h] && !(tv[h].y > 0.0);
        if (want[h] && waiting) F.pend[t[h]] = -1.0;
        if (want[h]) {
          const unsigned bit = 1u << (t[h] & 31);
          want[h] = !(atomicOr(bits + (t[h] >> 5), bit) & bit);
        }
      }
      if (any) sh.any[par] = 1;
      // places for the up to three nodes of each lane
      const unsigned below = (1u << lane) - 1u;
      const bool plain0 = tv[0].y > 0.0, plain1 = tv[1].y > 0.0;
      const unsigned r0 = __ballot_sync(kFull, want[0] && plain0);
      const unsigned r1 = __ballot_sync(kFull, want[1] && plain1);
      const unsigned x0 = __ballot_sync(kFull, want[0] && !plain0);
      const unsigned x1 = __ballot_sync(kFull, want[1] && !plain1);
      const unsigned x2 = __ballot_sync(kFull, want[2]);
      unsigned base = 0;
      if (lane == 0 && (r0 | r1)) base = atomicAdd(&sh.cnt[nxt][0], (unsigned)(__popc(r0) + __popc(r1)));
      if (lane == 1 && (x0 | x1 | x2))
        base = atomicAdd(&sh.cnt[nxt][1], (unsigned)(__popc(x0) + __popc(x1) + __popc(x2)));
      const unsigned rbase = __shfl_sync(kFull, base, 0), xbase = __shfl_sync(kFull, base, 1);
      if (want[0])
        put(nxt, plain0, t[0], plain0 ? rbase + __popc(r0 & below) : xbase + __popc(x0 & below));
      if (want[1])
        put(nxt, plain1, t[1], plain1 ? rbase + __popc(r0) + __popc(r1 & below)
                                      : xbase + __popc(x0) + __popc(x1 & below));
      if (want[2]) put(nxt, false, t[2], xbase + __popc(x0) + __popc(x1) + __popc(x2 & below));
    }
    // the others and those beyond shared memory: eight lanes per winner, two of
    // the nodes that read it each (from the last warp down: the first ones have
    // the regular winners)
    for (unsigned k = (kWarps - 1 - warp) * 32 + lane; k - lane < 8u * (nwx + no);
         k += kSolveThreads) {
      const unsigned w = k >> 3;
      const int sub = (int)(k & 7u);
      bool live = w < nwx + no;
      unsigned s = 0u;
      double thr = 0.0;
      if (w < nwx) {
        const unsigned j = cw[kCCap - 1 - w];
        s = ce[j] & kSlotMask;
        thr = co[j];
      } else if (live) {
        const unsigned e = cov[w - nwx];
        live = (e & kSpreadBit) != 0u;
        s = e & kSlotMask;
        thr = F.Tn[s];
      }
      const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
      int t[2];
      double2 tv[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // spread_target_at's nodes, its positions q
        const int q = sub + 8 * h;
        int r = -1, c = col;
        if (row < F.H) {
          if (q < 12) {
            // rows and columns -2..2 of the second neighbours and the 3x3 block
            r = row + (int)((0x333221112240ull >> (4 * q)) & 15) - 2;
            c = col + (int)((0x321313214022ull >> (4 * q)) & 15) - 2;
            if (r >= F.H) r = -1;
          } else {
            // the interface nodes of the cut cells it is a corner of
            const int side = (q - 12) >> 1;
            c = col - 1 + (q & 1);
            if (c >= 0 && c < F.nx) {
              const int izc = FMT_RO(F.izc + side * F.pitch + c), ar = F.z_lo + row;
              if (izc >= 0 && (izc == ar || izc + 1 == ar)) r = F.H + side;
            }
          }
        } else {
          const int side = row - F.H;
          if (q == 4) {
            r = F.H + (side ^ 1);
          } else if (q < 4) {
            const int izc = FMT_RO(F.izc + side * F.pitch + col);
            r = izc < 0 ? -1 : izc - F.z_lo + (q & 1);
            c = col + (q >> 1);
            if (r >= F.H) r = -1;
          }
        }
        t[h] = live && r >= 0 && c >= 0 && c < F.nx ? r * (int)pitch + c : -1;
        tv[h] = t[h] >= 0 ? *reinterpret_cast<const double2*>(F.R + t[h]) : make_double2(0.0, 0.0);
      }
      // time of the node between s and a second neighbour (sub < 4)
      double Tw = 0.0;
      if (row < F.H && sub < 4 && t[0] >= 0) Tw = F.R[((int)s + t[0]) / 2].x;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        bool want = t[h] >= 0;
        // (a velocity of zero: outside the region, unless the code says otherwise)
        if (want && tv[h].y == 0.0 && t[h] < F.H * (int)pitch)
          want = (FMT_RO(F.code + t[h]) & kInRegion) != 0u;
        // a waiting target (its bit may be stale) drops the time it waits with
        const bool waiting = want && windowed && ((waits((unsigned)t[h] >> 5) >> (t[h] & 31)) & 1u);
        want = want && (waiting || !(tv[h].x < thr));
        if (want) sh.any[par] = 1;
        // of those, the nodes whose update reads s: a regular node reads along
        // the axes only, and a second neighbour only behind a reached neighbour
        // that is not earlier than it (T2 <= T1, at s's old or new time)
        if (row < F.H) {
          const int q = sub + 8 * h;
          want = want && (q < 4 ? Tw < kReachD && Tw >= thr
                                : !((q == 4 || q == 6 || q == 9 || q == 11) && tv[h].y > 0.0));
        }
        if (want && waiting) F.pend[t[h]] = -1.0;
        push(nxt, (unsigned)t[h], tv[h].y > 0.0, want);
      }
    }
    // (readers are done with the marks)
    for (unsigned j = tid; j < nc; j += kSolveThreads) {
      const unsigned e = j < kCCap ? ce[j] : cov[j - kCCap];
      const unsigned s = e & kSlotMask;
      const int row = row_of(s), col = (int)(s - (unsigned)row * pitch);
      mbits[((unsigned)row & P.rmask) * P.mwords + ((col >> 5) & mmask)] = 0u;
    }
    __syncthreads();
    if (tid == 0) {
      sh.nw[0] = sh.nw[1] = 0u;
      lap(3);
    }
    // the window moves on after a step that changed nothing inside it (or
    // listed nothing); the tiles it reaches release their due nodes, and when
    // none is due it jumps to the earliest waiting time
    const bool chg = sh.changed[par] != 0;
    more = sh.any[par] != 0;
    if (!chg) W += wstep;
    if (!chg || !more) {
      for (; windowed;) {
        const int q = rp & 1;
        ++rp;
        for (int t = tid; t < ntiles; t += kSolveThreads)
          if (tmin[t] != kNone && __longlong_as_double((long long)tmin[t]) <= W)
            ready[atomicAdd(&sh.nready[q], 1u)] = (unsigned short)t;
        __syncthreads();
        const unsigned nready = sh.nready[q];
        if (tid == 0) {
          sh.nready[q ^ 1] = 0u;
          sh.gmin[q ^ 1] = kNone;
          sh.released[q ^ 1] = 0;
        }
        for (unsigned k = warp; k < nready; k += kWarps) {
          const int t = ready[k];
          const int r0 = (t / tcols) * kTileRows, c0 = (t % tcols) * 32;
          // lane l takes column c0 + l of the tile's rows; the rows' loads
          // are issued together
          unsigned word[kTileRows];
          double pd[kTileRows];
#pragma unroll
          for (int rr = 0; rr < kTileRows; ++rr)
            word[rr] = r0 + rr < F.H + 2 ? waits((unsigned)((r0 + rr) * F.pitch + c0) >> 5) : 0u;
#pragma unroll
          for (int rr = 0; rr < kTileRows; ++rr)
            pd[rr] = (word[rr] >> lane) & 1u ? F.pend[(r0 + rr) * F.pitch + c0 + lane] : 0.0;
          unsigned long long m = kNone;
#pragma unroll
          for (int rr = 0; rr < kTileRows; ++rr) {
            const bool set = (word[rr] >> lane) & 1u;
            bool clear = false, due = false;
            const unsigned s = (unsigned)((r0 + rr) * F.pitch + c0 + lane);
            if (set) {
              if (pd[rr] < 0.0) {
                clear = true;                 // listed since (an input changed)
              } else if (pd[rr] <= W) {
                clear = due = true;
                sh.released[q] = 1;
                ++n_rel;
              } else {
                m = min(m, dbits(pd[rr]));
              }
            }
            push(nxt, s, due && plain(s), due);
            const unsigned cm = __ballot_sync(0xffffffffu, clear);
            if (lane == 0 && cm) wbits[(unsigned)((r0 + rr) * F.pitch + c0) >> 5] = word[rr] & ~cm;
          }
#pragma unroll
          for (int o = 16; o; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
          if (lane == 0) tmin[t] = m;
        }
        __syncthreads();
        if (more || sh.released[q]) {
          more = true;
          break;
        }
        // nothing due: the earliest waiting time, if any
        unsigned long long m = kNone;
        for (int t = tid; t < ntiles; t += kSolveThreads) m = min(m, tmin[t]);
        if (m != kNone) atomicMin(&sh.gmin[q], m);
        __syncthreads();
        const unsigned long long g = sh.gmin[q];
        if (g == kNone) break;
        W = fmax(W, __longlong_as_double((long long)g));
      }
      if (tid == 0) lap(4);
    }
    cur = nxt;
  }
  n_eval = __reduce_add_sync(kFull, n_eval);
  n_write = __reduce_add_sync(kFull, n_write);
  n_rel = __reduce_add_sync(kFull, n_rel);
  n_cut = __reduce_add_sync(kFull, n_cut);
  if (lane == 0 && ctr) {
    atomicAdd(ctr + kCtrCut, (unsigned long long)n_cut);
    atomicAdd(ctr + kCtrEval, (unsigned long long)n_eval);
    atomicAdd(ctr + kCtrWrite, (unsigned long long)n_write);
    atomicAdd(ctr + kCtrPass, (unsigned long long)n_rel);
  }
  __syncthreads();
  if (tid == 0) {
    F.clock[0] = W;
    F.clock[2] = __longlong_as_double((long long)(stamp0 + (unsigned long long)it));
    F.cnt[0] = 0u;   // start list consumed; the check refills it
    F.cnt[1] = 0u;
    F.cnt[3] = (unsigned)(it < 0xffffffffll ? it : 0xffffffffll);
    if (sh.err) F.cnt[2] = 1u;
    if (ctr) {
      for (int k = 0; k < 5; ++k) atomicAdd(ctr + kCtrCycEval + k, sh.cyc[k]);
      atomicAdd(ctr + kCtrStepsCut, sh.steps_cut);
      atomicAdd(ctr + kCtrSteps, (unsigned long long)it);
      atomicMax(ctr + kCtrMaxSteps, (unsigned long long)it);
    }
  }
}

// Append slot s to the field's start list unless it is there already
// (F.inq zeroed before the kernel that appends).
__device__ __forceinline__ void list_start(const Fld64& F, unsigned s) {
  const unsigned bit = 1u << (s & 31);
  if (atomicOr(F.inq + (s >> 5), bit) & bit) return;
  F.list_in[atomicAdd(F.cnt, 1u)] = s;
}

// Fixed-point check of every node (window ignored): a node whose update
// would change it is listed and counted.  The regular nodes, which are nearly
// all and cost evaluate() a dozen roots and quotients each, are evaluated by
// reg_best on the records the state came from: the solver's own function, so
// this finds nodes that were not evaluated again, not an error of reg_best.
// k_verify_cut<true> evaluates every node with evaluate() instead.
__device__ __forceinline__ bool regular_slot(const Fld64& F, int s) {
  constexpr uint32_t kPlain = kInRegion | kUpdatable | kFullyRegular;
  return (F.code[s] & kPlain) == kPlain && s < F.H * F.pitch;
}

__global__ void __launch_bounds__(256) k_verify(Fld64* fields, int nf) {
  const Fld64& F = fields[blockIdx.y];
  const int ns = F.nslots();
  const double rdx = 1.0 / F.dx;
  unsigned nbad = 0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
    const int row = s / F.pitch, col = s - row * F.pitch;
    if (col >= F.nx || !regular_slot(F, s) || s == F.frozen_slot) continue;
    const Rec me = load_rec(F, s);
    Self self;
    self.T = me.T;
    self.g = make_double2(me.gx, me.gz);
    self.fl = F.fl[s];
    const RegBest rb = reg_best<false>(F, rdx, s, row, col, fabs(me.v), 15u);
    const NewV nv =
        settle(F, s, rb.t, rb.gx, rb.gz, false, rb.key != kNoKey && !(rb.key & 1), rb.t, self);
    if (nv.write) {
      ++nbad;
      list_start(F, (unsigned)s);
    }
  }
  if (nbad) atomicAdd(F.cnt + 1, nbad);
}

// The nodes at an interface (kAll: every node), by evaluate() on the state as it
// was unpacked.
// A block gathers those of its slots first: one is a chain of 57,000 cycles, and
// left where they are each holds a warp of others.  (60 fields of 800,000 nodes:
// both kernels 1.9 ms, one kernel for all nodes 3.0, evaluate() alone 4.8.  A
// longer span gathers better, 1.7 ms at 4096, but leaves a small field's nodes to a
// few blocks: 121 x 66 nodes, five fields, 7% slower.)
constexpr int kCheckSpan = 512;
template <bool kAll>
__global__ void __launch_bounds__(128) k_verify_cut(Fld64* fields, int nf) {
  const Fld64& F = fields[blockIdx.y];
  const int ns = F.nslots();
  __shared__ unsigned list[kCheckSpan];
  __shared__ unsigned n;
  unsigned nbad = 0;
  for (int b = blockIdx.x * kCheckSpan; b < ns; b += gridDim.x * kCheckSpan) {
    if (threadIdx.x == 0) n = 0;
    __syncthreads();
    for (int s = b + threadIdx.x; s < min(b + kCheckSpan, ns); s += blockDim.x)
      if ((s % F.pitch) < F.nx && (F.code[s] & kInRegion) &&
          (kAll || !regular_slot(F, s)))
        list[atomicAdd(&n, 1u)] = (unsigned)s;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
      const NewV nv = evaluate(F, (int)list[i]);
      if (nv.write) {
        ++nbad;
        list_start(F, list[i]);
      }
    }
    __syncthreads();
  }
  if (nbad) atomicAdd(F.cnt + 1, nbad);
}

// List every seeded node and the nodes around it.
__global__ void k_queue_seeds(Fld64* fields, int nf) {
  const Fld64& F = fields[blockIdx.y];
  const int ns = F.nslots();
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
    if ((s % F.pitch) >= F.nx || !(F.fl[s] & kFlSeed)) continue;
    list_start(F, (unsigned)s);
    int t[16];
    const int k = spread_targets(F, s, t);
    for (int q = 0; q < k; ++q) list_start(F, (unsigned)t[q]);
  }
}

// Solver records of a field from its state, and the state from the records.
__global__ void k_pack(Fld64* fields, int nf) {
  const Fld64& F = fields[blockIdx.y];
  const int ns = F.nslots();
  constexpr uint32_t kPlain = kInRegion | kUpdatable | kFullyRegular;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
    const uint32_t code = F.code[s];
    const double v = F.vel[s];
    const double2 g = F.G[s];
    F.R[s] = make_double4(
        F.T[s], !(code & kInRegion) ? 0.0 : (code & kPlain) == kPlain ? v : -v, g.x, g.y);
  }
}

__global__ void k_unpack(Fld64* fields, int nf) {
  const Fld64& F = fields[blockIdx.y];
  const int ns = F.nslots();
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
    const double4 r = F.R[s];
    F.T[s] = r.x;
    F.G[s] = make_double2(r.z, r.w);
  }
}

// ---------------------------------------------------------------- seeding
__global__ void k_fill(Fld64* fields, int nf) {
  Fld64& F = fields[blockIdx.y];
  const size_t ns = (size_t)(F.H + 2) * F.pitch;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < ns;
       i += (size_t)gridDim.x * blockDim.x) {
    F.T[i] = kHugeD;
    F.G[i] = make_double2(0.0, 0.0);
    F.claim[i] = make_ulonglong2(0, 0);   // of no step (the bits of Gout's zeros)
    F.seed[i] = make_double4(kHugeD, 0.0, 0.0, 0.0);
    F.fl[i] = 0;
    F.pend[i] = -1.0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    F.frozen_slot = -1;
    F.clock[2] = 0.0;
  }
}

__device__ void put_seed(Fld64& F, int s, double t, double gx, double gz) {
  F.T[s] = t;
  F.G[s] = make_double2(gx, gz);
  F.seed[s] = make_double4(t, gx, gz, 0.0);
  F.fl[s] = kFlSeed;
}

// initialize_region_from_source2d (:2307-2411): the corners of the source
// cell get dist/v and the straight-ray gradient; a corner within
// 0.01*tolerance takes t0 = 0 and stays fixed.
__global__ void k_init_source(Fld64* fields, const double* sx, const double* sz, int nf) {
  const int fi = blockIdx.x * blockDim.x + threadIdx.x;
  if (fi >= nf) return;
  Fld64& F = fields[fi];
  const double h = F.dx;
  int ix0 = (int)floor((sx[fi] - F.x0) / h);
  int iz0 = (int)floor((sz[fi] - 0.0) / h);
  ix0 = max(0, min(F.nx - 2, ix0));
  iz0 = max(0, min(F.nz - 2, iz0));
  for (int ix = ix0; ix <= ix0 + 1; ++ix)
    for (int iz = iz0; iz <= iz0 + 1; ++iz) {
      const int br = iz - F.z_lo;
      if (br < 0 || br >= F.H) continue;
      const int s = br * F.pitch + ix;
      if (!(F.code[s] & kInRegion)) continue;
      const double ddx = (F.x0 + ix * h) - sx[fi], ddz = iz * h - sz[fi];
      const double dist = sqrt(ddx * ddx + ddz * ddz);
      double v = F.vel[s];
      if (v < 0.01) v = 0.01;
      if (dist < 0.01 * F.tol) {
        put_seed(F, s, 0.0, 0.0, 0.0);
        F.frozen_slot = s;
      } else {
        const double t = dist / v;
        put_seed(F, s, t, ddx / (dist * v), ddz / (dist * v));
      }
    }
}

// Interface hand-off of a stage (transfer_times_to_intersection :2414-2554,
// reflect_gradient_at_interface :2632-2741, sweep_region_from_interface2d
// :1982-2304): the target region's interface nodes take the parent's
// boundary time and gradient (normal slowness rebuilt on the target side when
// reflecting), grid nodes up to three rows into the region take
// T_if + dist/v from the first interface node whose box holds them.
__global__ void k_seed_iface(Fld64* fields, const Seed64* descs, int nd, int nx) {
  const Seed64& D = descs[blockIdx.y];
  Fld64& F = fields[D.dst];
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= F.nx) return;
  const double h = F.dx;
  auto iface_val = [&](int k, double& T, double& gx, double& gz) {
    const int ss = D.src_row * D.src_pitch + k;
    T = D.src_T[ss];
    const double2 g = D.src_G[ss];
    gx = g.x;
    gz = g.y;
    if (T >= kReachD) { T = kHugeD; }
    if (!D.reflect) return;
    if (T >= kReachD) { gx = 0.0; gz = 0.0; return; }
    const double nx_ = D.ifc.nrm_x[k], nz_ = D.ifc.nrm_z[k];
    const double gp = gx * nx_ + gz * nz_;
    const double px = gx - gp * nx_, pz = gz - gp * nz_;
    const int side = D.target_side;
    double v = side > 0 ? D.ifc.vel_bot[k] : D.ifc.vel_top[k];
    if (!(v > 0.01)) v = F.vel[(F.H + D.dst_side) * F.pitch + k];
    if (v <= 0.01) { T = kHugeD; gx = 0.0; gz = 0.0; return; }
    const double pn2 = 1.0 / (v * v) - (px * px + pz * pz);
    if (pn2 < -1.0e-10) { T = kHugeD; gx = 0.0; gz = 0.0; return; }
    const double pn = sqrt(pn2 < 0.0 ? 0.0 : pn2);
    gx = px + side * pn * nx_;
    gz = pz + side * pn * nz_;
  };
  double T, gx, gz;
  iface_val(c, T, gx, gz);
  {
    const int s = (F.H + D.dst_side) * F.pitch + c;
    put_seed(F, s, T, gx, gz);
  }
  int done[9], ndone = 0;
  for (int n = c - 1; n <= c + 1; ++n) {
    if (n < 0 || n >= nx) continue;
    const int izf = D.ifc.izc[n];
    if (izf < 0) continue;
    int r_a, r_b, st;
    if (D.dst_side == 1) { r_a = izf; r_b = max(0, izf - 2); st = -1; }
    else { r_a = izf + 1; r_b = min(F.nz - 1, izf + 3); st = 1; }
    double Tn, gxn, gzn;
    iface_val(n, Tn, gxn, gzn);
    const double xm = F.ifx[n], zm = D.ifc.z[n];
    for (int r = r_a; st > 0 ? r <= r_b : r >= r_b; r += st) {
      if (r < D.r0[c] || r > D.r1[c]) continue;
      bool seen = false;
      for (int q = 0; q < ndone; ++q) seen = seen || (done[q] == r);
      if (seen) continue;
      done[ndone++] = r;
      const int br = r - F.z_lo;
      const int s = br * F.pitch + c;
      const double ddx = (F.x0 + c * h) - xm, ddz = r * h - zm;
      const double dist = sqrt(ddx * ddx + ddz * ddz);
      double v = F.vel[s];
      if (v < 0.01) v = 0.01;
      const double tn = Tn >= kReachD ? kHugeD : Tn + dist / v;
      put_seed(F, s, tn, ddx / (dist * v), ddz / (dist * v));
    }
  }
}

// Window of each field: from its earliest seed, advancing by step[f].
__global__ void k_clock(Fld64* fields, int nf, const double* step) {
  Fld64& F = fields[blockIdx.x];
  const int ns = (F.H + 2) * F.pitch;
  // the flags, sixteen slots a load (one block reads a field: a slot a load
  // took 1.2 ms for 60 fields of 800,000)
  double mn = kHugeD;
  const int nv = ns / 16;
  const uint4* fl = reinterpret_cast<const uint4*>(F.fl);
  constexpr unsigned kAny = kFlSeed * 0x01010101u;
#pragma unroll 4
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 w = fl[i];
    if (!((w.x | w.y | w.z | w.w) & kAny)) continue;
    for (int s = 16 * i; s < 16 * i + 16; ++s)
      if (F.fl[s] & kFlSeed) mn = fmin(mn, F.T[s]);
  }
  for (int s = 16 * nv + threadIdx.x; s < ns; s += blockDim.x)
    if (F.fl[s] & kFlSeed) mn = fmin(mn, F.T[s]);
  __shared__ double sm[32];
#pragma unroll
  for (int o = 16; o; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mn;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mn = fmin(mn, sm[w]);
    const double t0 = mn < kReachD ? mn : 0.0;
    F.clock[1] = step[blockIdx.x];
    F.clock[0] = t0 + step[blockIdx.x];
  }
}

// Final gradients: the winning candidate's, suspect nodes refitted
// (propagate2d.f90:119-123).
__global__ void k_final_grad(Fld64* fields, int nf) {
  Fld64& F = fields[blockIdx.y];
  const size_t ns = (size_t)(F.H + 2) * F.pitch;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < ns;
       i += (size_t)gridDim.x * blockDim.x) {
    if (!(F.code[i] & kInRegion)) continue;
    if ((F.fl[i] & kFlSusp) && F.T[i] < kReachD) {
      double gx, gz;
      fit_grad(F, (int)i, gx, gz);
      F.Gout[i] = make_double2(gx, gz);
    } else {
      F.Gout[i] = F.G[i];
    }
  }
}

// Top-row gradient fix of the water-layer fields (inversion2d.f90:4264-4292):
// upward = 1 requires dT/dz < 0 at the sea surface, upward = 0 requires > 0.
__global__ void k_water_fix(Fld64* fields, const int* upward, int nf) {
  const int fi = blockIdx.y;
  Fld64& F = fields[fi];
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= F.nx || upward[fi] < 0) return;
  const int bt = 0 - F.z_lo, bb = 1 - F.z_lo;
  if (bt < 0 || bb >= F.H) return;
  const int st = bt * F.pitch + c, sb = bb * F.pitch + c;
  if (!(F.code[st] & kInRegion) || !(F.code[sb] & kInRegion)) return;
  const double gz = F.Gout[st].y;
  const bool bad = upward[fi] ? (gz > 0.0 || fabs(gz) < 0.01) : (gz < 0.0 || fabs(gz) < 0.01);
  if (bad) F.Gout[st] = F.Gout[sb];
}

// PmP head-wave min-plus sweep along the Moho (inversion2d.f90:4294-4409), a
// block per field; node table and velocities are precomputed per model.  The
// two sweeps are chains over the nodes (their sums round in that order): one
// thread runs them from shared memory, a batch of nodes at a time, and all
// else is spread over the block (30 fields of 2001 nodes: 0.2 ms; a thread per
// field, its loads one after the other, took 7.5 ms).
// The solved times the sweep replaces are saved first (pre, nx per field:
// the adjoint re-derives each node's winning update from them).
constexpr int kHwBatch = 1024;
__global__ void __launch_bounds__(256)
    k_headwave(Fld64* fields, const int* hw_slot, const double* hw_v, double dx_if, int nx,
               double* scratch, const int* which, double* const* pre) {
  const int q = blockIdx.x, tid = threadIdx.x;
  Fld64& F = fields[which[q]];
  double* th = scratch + (size_t)q * nx;
  double* keep = pre ? pre[q] : nullptr;
  __shared__ double s_t[kHwBatch], s_d[kHwBatch];
  __shared__ double s_last;
  // dir 1: left to right, the nodes' times from the field; -1: back, from th
  auto sweep = [&](int dir) {
    for (int b = 0; b < nx; b += kHwBatch) {
      const int m = min(kHwBatch, nx - b);
      for (int i = tid; i < m; i += blockDim.x) {
        const int n = dir > 0 ? b + i : nx - 1 - (b + i);
        double t;
        if (dir > 0) {
          t = hw_slot[n] >= 0 ? F.T[hw_slot[n]] : kHugeD;
          if (keep) keep[n] = t;
        } else {
          t = th[n];
        }
        s_t[i] = t;
        // (a node without a velocity keeps its time)
        s_d[i] = hw_v[n] > 0.0 ? dx_if / hw_v[n] : CUDART_INF;
      }
      __syncthreads();
      if (tid == 0) {
        double t = b ? s_last : s_t[0];
#pragma unroll 8
        for (int i = b ? 0 : 1; i < m; ++i) {
          t = fmin(s_t[i], t + s_d[i]);
          s_t[i] = t;
        }
        s_last = t;
      }
      __syncthreads();
      for (int i = tid; i < m; i += blockDim.x) th[dir > 0 ? b + i : nx - 1 - (b + i)] = s_t[i];
      __syncthreads();
    }
  };
  sweep(1);
  sweep(-1);
  for (int n = tid; n < nx; n += blockDim.x) {
    const int s = hw_slot[n];
    if (s >= 0 && th[n] < F.T[s] - 1.0e-10) F.T[s] = th[n];
  }
  __syncthreads();
  for (int n = tid; n < nx; n += blockDim.x) {
    const int s = hw_slot[n];
    if (s < 0 || F.T[s] >= kReachD) continue;
    if (!(F.code[s] & kIfaceNode)) {
      double gx, gz;
      fit_grad(F, s, gx, gz);
      F.Gout[s] = make_double2(gx, gz);
    } else {
      double dtdx;
      if (n > 0 && n < nx - 1) dtdx = (th[n + 1] - th[n - 1]) / (2.0 * dx_if);
      else if (n == 0 && nx > 1) dtdx = (th[1] - th[0]) / dx_if;
      else if (n == nx - 1 && nx > 1) dtdx = (th[nx - 1] - th[nx - 2]) / dx_if;
      else dtdx = 0.0;
      double dtdz = 0.0;
      if (hw_v[n] > 0.0) {
        const double s2 = 1.0 / (hw_v[n] * hw_v[n]) - dtdx * dtdx;
        dtdz = s2 > 0.0 ? sqrt(s2) : 0.0;
      }
      F.Gout[s] = make_double2(dtdx, dtdz);
    }
  }
}

__global__ void k_export(const double* T, const double2* G, const int* slot_of_node, int nnode,
                         double* oT, double* ogx, double* ogz) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nnode; n += gridDim.x * blockDim.x) {
    const int s = slot_of_node[n];
    if (oT) oT[n] = T[s];
    const double2 g = G[s];
    if (ogx) ogx[n] = g.x;
    if (ogz) ogz[n] = g.y;
  }
}


}  // namespace

// ---------------------------------------------------------------- launchers
void e64_fill(Fld64* f, int nf, size_t max_slots, cudaStream_t st) {
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 1024);
  k_fill<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
}
void e64_init_source(Fld64* f, const double* sx, const double* sz, int nf, cudaStream_t st) {
  k_init_source<<<(nf + 63) / 64, 64, 0, st>>>(f, sx, sz, nf);
}
void e64_seed_iface(Fld64* f, const Seed64* d, int nd, int nx, cudaStream_t st) {
  k_seed_iface<<<dim3((nx + 127) / 128, nd), 128, 0, st>>>(f, d, nd, nx);
}
void e64_start(Fld64* f, int nf, size_t max_slots, const double* step, cudaStream_t st) {
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 256);
  k_queue_seeds<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
  k_clock<<<nf, 1024, 0, st>>>(f, nf, step);
}
int e64_tiles(const Fld64& f) { return tiles_of(f); }
int e64_tiles_max() { return kTilesMax; }

// Dynamic shared memory of k_solve under plan P.
static size_t solve_smem(const SolvePlan& P) {
  return (size_t)P.tiles * (sizeof(unsigned long long) + sizeof(unsigned short)) +
         2 * (kXCap + kLCap) * sizeof(unsigned) +
         ((size_t)P.mtotal + (size_t)P.nbits * P.bits) * sizeof(unsigned);
}

// Largest dynamic shared memory of an instantiation; its attribute is set
// once per device: changing a kernel's attributes while it runs (a solve of
// another stage chain on another stream) waits for that kernel to finish,
// which would serialise the chains.
template <int NT>
static size_t solve_room() {
  static std::mutex mu;
  static int room[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (room[dev]) return (size_t)room[dev];
  // the opt-in limit covers static and dynamic shared memory together
  int optin = 0;
  cudaFuncAttributes fa;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k_solve<NT>) != cudaSuccess)
    return 0;
  const int dyn = std::min<int>((int)kSmemMax, optin - (int)fa.sharedSizeBytes);
  if (cudaFuncSetAttribute(k_solve<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) ==
      cudaSuccess)
    room[dev] = dyn;
  return (size_t)room[dev];
}

template <int NT>
static void solve_launch(Fld64* f, const Fld64* fh, int nf, bool windowed, long long max_steps,
                         unsigned long long* ctr, cudaStream_t st) {
  int rows = 0, tiles = 0, slots = 0;
  for (int i = 0; i < nf; ++i) {
    rows = std::max(rows, fh[i].H + 2);
    tiles = std::max(tiles, tiles_of(fh[i]));
    slots = std::max(slots, fh[i].nslots());
  }
  SolvePlan P;
  P.bits = (slots + 31) / 32;
  P.tiles = windowed ? (tiles + 7) / 8 * 8 : 0;
  // what fits of: the listed bitset (an atomic on every push), the waiting
  // bitset; the moving bitmap needs a word per row at least and takes up to
  // eight (256 columns: marks of other columns are then rare)
  const size_t room = solve_room<NT>();
  P.nbits = windowed ? 2 : 1;
  P.rmask = ~0u;
  for (;; --P.nbits) {
    for (P.mwords = 8; P.mwords > 1; P.mwords /= 2) {
      P.mtotal = rows * P.mwords;
      if (solve_smem(P) <= room) break;
    }
    P.mtotal = rows * P.mwords;
    if (P.nbits == 0 || solve_smem(P) <= room) break;
  }
  // more rows than words of shared memory (regions of tens of thousands of rows,
  // which only a narrow model has): rows that lie 2^k apart share a word
  for (unsigned r = 1u << 30; solve_smem(P) > room && r >= 64u; r >>= 1) {
    P.rmask = r - 1;
    P.mtotal = std::min(rows, (int)r);
  }
  k_solve<NT><<<nf, NT, solve_smem(P), st>>>(f, P, max_steps, ctr);
}

const int* e64_solve_sizes(int* n) {
  *n = 3;
  return kSolveSizes;
}

void e64_pack(Fld64* f, int nf, size_t max_slots, cudaStream_t st) {
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 1024);
  k_pack<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
}

void e64_solve(Fld64* f, const Fld64* fh, int nf, size_t max_slots, bool windowed,
               long long max_steps, unsigned long long* ctr, int threads, cudaStream_t st) {
  if (threads == 256) solve_launch<256>(f, fh, nf, windowed, max_steps, ctr, st);
  else if (threads == 512) solve_launch<512>(f, fh, nf, windowed, max_steps, ctr, st);
  else solve_launch<kSolveDefault>(f, fh, nf, windowed, max_steps, ctr, st);
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 1024);
  k_unpack<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
}
void e64_verify(Fld64* f, int nf, size_t max_slots, bool all, cudaStream_t st) {
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 512);
  const int bc = (int)std::min<size_t>((max_slots + kCheckSpan - 1) / kCheckSpan, 2048);
  if (all) {
    k_verify_cut<true><<<dim3(bc, nf), 128, 0, st>>>(f, nf);
    return;
  }
  k_verify<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
  k_verify_cut<false><<<dim3(bc, nf), 128, 0, st>>>(f, nf);
}
void e64_finish(Fld64* f, int nf, size_t max_slots, const int* water_up, cudaStream_t st) {
  const int bx = (int)std::min<size_t>((max_slots + 255) / 256, 512);
  k_final_grad<<<dim3(bx, nf), 256, 0, st>>>(f, nf);
  k_water_fix<<<dim3(64, nf), 128, 0, st>>>(f, water_up, nf);
}
void e64_headwave(Fld64* f, const int* hw_slot, const double* hw_v, double dx_if, int nx,
                  double* scratch, const int* which, int nsel, double* const* pre,
                  cudaStream_t st) {
  k_headwave<<<nsel, 256, 0, st>>>(f, hw_slot, hw_v, dx_if, nx, scratch, which, pre);
}
void e64_export(const double* T, const double2* G, const int* slot_of_node, int nnode, double* oT,
                double* ogx, double* ogz, cudaStream_t st) {
  k_export<<<(nnode + 255) / 256, 256, 0, st>>>(T, G, slot_of_node, nnode, oT, ogx, ogz);
}

}  // namespace fmt2d
