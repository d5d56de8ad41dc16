// Fronts above the shared-memory limit, factored in blocked panels with
// a-posteriori threshold tests.
//
// The reference tests one candidate at a time (SparseLDL::
// factor_front_matrix_block, include/sparse_ldl.h:1316-1553): it forms the
// candidate's column, compares the pivot with the largest entry of the
// column over every remaining row of the front, and accepts a 1x1 pivot, the
// alternative 1x1 at imax or a Duff 2x2, or delays the candidate to the
// parent. Once the candidates are arranged so that nearly every one passes
// where it stands (pivot-order reuse), that sequence of column-wide tests is
// what costs time, not arithmetic. Here a panel of up to 32 candidates of
// every front of a tree level is decided in data-parallel phases:
//
//   D. Delays left by the previous panel are applied with the reference's
//      symmetric interchange (symm_swap, sparse_ldl.h:1270-1292), by the
//      whole CTA when the level has no more fronts than CTAs, else by one
//      warp per front; the next block's column maxima below follow the
//      interchanges. Then one warp factors the 32 x 32 diagonal block with
//      the reference's tests (lane r owns block row r), left-looking: a
//      column is formed from the loaded block and the pivots taken when a
//      test reads it. A test's column maximum joins the block's rows with,
//      for the panel's first pivot, the column's exact maximum below the
//      block that the previous panel's trailing update left behind. A pair
//      that formed a 2x2 pivot in the pivot record is tried as that 2x2
//      first. A candidate that fails is rotated behind the block's
//      candidates.
//   R. (row chunks) Every row below the block forms its entries of the
//      pivot columns, W = F21 L11^-T (the values the reference's tests see),
//      stores them for the trailing update, and the column maxima over all
//      rows below are reduced. The front's last chunk to finish runs the
//      reference's tests exactly, with the column maxima over the whole
//      front, and records how many leading pivots pass.
//   A+U. The row chunks write L for the passing pivots (D on the diagonal,
//      2x2 blocks with d21 below it, as the reference stores them) and the
//      first of them commits the panel; beside them, 64 x 64 tiles give the
//      trailing matrix the rank-kw update, forming L from W as the commit
//      does. The first rejected pivot, and the candidates that failed in
//      the block while only accepted pivots preceded them, are delayed at
//      the next phase D. (In the mixed-precision mode the commit and the
//      update are separate phases: the tensor-core tiles read L from the
//      front.)
//
// Every accepted pivot therefore satisfies the reference's threshold test
// against its whole column, so the factorization has the reference's
// stability bound (|L| <= 1/ustab for 1x1 pivots) and, by Sylvester's law,
// its inertia; only the order in which candidates are tried differs (a
// candidate's 2x2 partner is searched within its panel's block). A root
// cannot delay: the candidates its tests leave are finished by the chained
// panels (Bunch-Kaufman) after the level's launch.
//
// What a panel step costs is mostly fixed: three grid barriers, one warp's
// work on the block, and chains of global loads. So each phase loads before
// it computes, an item's front is described in shared memory (Info), the
// one-warp phase counts its instructions (a panel's block 79,000 -> 48,000
// cycles), delays exchange in phase D only what the block needs (30,000 ->
// 11,000-23,000 cycles on a one-front level), and the trailing tiles use
// mma.m8n8k4.f64 with the next tile's loads in flight. Plane stress 256 x
// 256, record of a neighbouring iterate: 291 -> 248 ms of panel levels a
// factorization; hex elasticity 11^3 with a dense row: 133 -> 112 ms.
//
// The phases run in one cooperative launch per level, separated by grid-wide
// barriers: three per panel step. Every CTA runs the same phases and
// barriers; the loop ends for all of them on a count that the barrier makes
// visible to all, or at a cap that the progress of every step guarantees
// not to reach (each step of an active front accepts a pivot or delays a
// candidate).
//
// The front stays in HBM in logical order between steps (column-major,
// lower triangle, the layout big_chain.cu and big_update_kernel use). A
// panel's state lives in a per-front scratch area (xoff) stamped with the
// step number, so a front that finished earlier takes no part.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>

#include "ldl_internal.h"
#include "umma.cuh"

namespace cg = cooperative_groups;

namespace b200ldl {

namespace {

constexpr int kBlk = 32;  // candidates per panel
constexpr int kLd = kBlk + 2;  // even: two entries of a row per shared-memory load
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileU = 64;          // trailing-update tile
constexpr int kChunkFronts = 1024;  // fronts per work-item prefix
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;

// per-front scratch (doubles at xoff)
constexpr int kXNext = kAppNextColmax;      // [32] next panel's column maxima below (bits)
constexpr int kXL = kXNext + kBlk;          // Lb[32][33]: block rows' L entries
constexpr int kXD = kXL + kBlk * kLd;       // dd[32][3]: d | d11, d21, d22 per pivot
constexpr int kXCin = kXD + 3 * kBlk;       // block part of the column maximum
constexpr int kXRin = kXCin + kBlk;         // block part of a 2x2 partner's column maximum
constexpr int kXBelow = kXRin + kBlk;       // column maxima over the rows below (bits)
constexpr int kXInt = kXBelow + kBlk;       // ints from here
// int offsets (from kXInt as int*)
constexpr int kIPerm = 0;    // [32] block position -> block position before the panel
constexpr int kIKind = 32;   // [32] 1: 1x1, 2: first of a 2x2, 3: second of a 2x2
constexpr int kIDlt = 64;    // [32] candidates failed in the block: pivots accepted before
constexpr int kIAcc = 96;    // pivots accepted inside the block
constexpr int kINbk = 97;    // candidates in the block
constexpr int kIK = 98;      // first position of the panel
constexpr int kIStep = 99;   // step number of the panel
constexpr int kINcand = 100;
constexpr int kIMoved = 101;  // 1 if the block permutation is not the identity
constexpr int kIDcnt = 102;   // candidates to delay at the next step
constexpr int kIDpos = 103;   // [32] their positions, decreasing
constexpr int kINp = kIDpos + kBlk;  // pivots that pass the exact tests (set by phase R)
constexpr int kIRdone = kINp + 1;    // phase-R items of the panel finished
constexpr int kISwaps = kIRdone + 1;   // interchanges that phase R carries out
constexpr int kISwapB = kISwaps + 1;   // candidates before them (b = that - 1 - q)
constexpr int kINint = kISwapB + 1;
static_assert(kXInt + (kINint + 1) / 2 <= kAppScratch, "a-posteriori scratch size");

__device__ __forceinline__ double fsym(const double* F, int f, int a, int b) {
  return (a >= b) ? F[a + (size_t)f * b] : F[b + (size_t)f * a];
}

__device__ __forceinline__ int* xint(double* X) { return reinterpret_cast<int*>(X + kXInt); }

// Non-negative doubles order as their bit patterns, so the warp reductions
// below are exact integer reductions (redux.sync) on the high and then the
// low 32 bits, instead of FP64 shuffle butterflies.

// Largest of the non-negative values v of the lanes with `on`, and the
// lowest lane holding it (idamax); -1 and lane 0 when no lane is on.
__device__ __forceinline__ void warp_argmax(bool on, double v, double& best, int& idx) {
  const unsigned long long b = on ? (unsigned long long)__double_as_longlong(v) : 0ull;
  // +1 keeps an active 0.0 above the inactive lanes
  const unsigned hi = on ? (unsigned)(b >> 32) + 1u : 0u;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const bool cand = on && hi == mhi;
  const unsigned lo = cand ? (unsigned)b : 0u;
  const unsigned mlo = __reduce_max_sync(0xffffffffu, lo);
  const unsigned win = __ballot_sync(0xffffffffu, cand && lo == mlo);
  idx = win ? __ffs(win) - 1 : 0;
  best = mhi ? __longlong_as_double((long long)(((unsigned long long)(mhi - 1u) << 32) | mlo))
             : -1.0;
}

// largest of the lanes' non-negative values
__device__ __forceinline__ double warp_max(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned mhi = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32));
  const unsigned mlo = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32) == mhi ? (unsigned)b : 0u);
  return __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
}

// The L entries (l0, l1) of a row whose W entries are (a, b) under the 2x2
// pivot d = (d11, d21, d22): (a, b) D^-1, with explicit fused multiply-adds so
// that every kernel that forms them gets the same values.
__device__ __forceinline__ void inv_2x2(const double* d, double* inv) {
  const double d11 = d[0], d21 = d[1], d22 = d[2];
  const double di = 1.0 / (d11 * d22 - d21 * d21);
  inv[0] = d22 * di;
  inv[1] = -d21 * di;
  inv[2] = d11 * di;
}
__device__ __forceinline__ double l_first(const double* inv, double a, double b) {
  return fma(a, inv[0], __dmul_rn(b, inv[1]));
}
__device__ __forceinline__ double l_second(const double* inv, double a, double b) {
  return fma(a, inv[1], __dmul_rn(b, inv[2]));
}
__device__ __forceinline__ void l_2x2(const double* d, double a, double b, double& l0,
                                      double& l1) {
  double inv[3];
  inv_2x2(d, inv);
  l0 = l_first(inv, a, b);
  l1 = l_second(inv, a, b);
}

// ------------------------------------------------------------- shared memory

struct WarpDiag {  // phase D, one per warp
  double A[kBlk][kLd];  // the block, symmetric, factored in place
  double Lb[kBlk][kLd];
  double below0[kBlk];
  int perm[kBlk], dlt[kBlk];
  int var[kBlk], part[kBlk];  // block candidates' variables and recorded 2x2 partners
};

struct RowsSm {  // phases R and A
  alignas(16) double Ls[kBlk][kLd];
  double red[kWarps][kBlk];
  double sd[3 * kBlk], sinv[kBlk];
  double inv[kBlk][3];  // phase A: inverses of the 2x2 pivots
  double scm[kBlk], srm[kBlk];  // phase A: column maxima over the front, 2x2 partner's block part
  int sperm[kBlk], skind[kBlk];
  int np;
};

// The reference's tests for the accepted pivots of a panel, with the column
// maxima over the whole front (staged in shared memory), by one warp, a lane
// per pivot: number of leading pivots that pass.
__device__ int passing_prefix(const RowsSm& sm, int acc, double ustab, double tol) {
  const int p = threadIdx.x & 31;
  bool ok = true;
  if (p < acc) {
    const double cm = sm.scm[p];
    if (sm.skind[p] == 1) {
      const double d = sm.sd[3 * p];
      ok = fabs(d) >= tol && fabs(d) >= ustab * cm;
    } else if (sm.skind[p] == 2) {
      const double d11 = sm.sd[3 * p], d21 = sm.sd[3 * p + 1], d22 = sm.sd[3 * p + 2];
      const double det = fabs(d11 * d22 - d21 * d21);
      const double ad21 = fabs(d21);
      const double delta = det / fmax(fabs(d22) + ad21, fabs(d11) + ad21);
      // the partner's maximum: its block part (srm) and its maximum below
      // (scm of the second position, whose block part phase D leaves at 0)
      const double rm = fmax(sm.srm[p], sm.scm[p + 1]);
      ok = det >= tol && delta >= ustab * cm && delta >= ustab * rm;
    }
  }
  const unsigned bad = __ballot_sync(0xffffffffu, !ok);
  return bad ? __ffs(bad) - 1 : acc;
}

// row stride of the panels in shared memory: the four pivots that a warp's
// lanes read at once start 8 banks apart
constexpr int kTileLdU = kTileU + 4;
struct UpdSm {  // phase U
  double As[kBigPanelMax][kTileLdU];
  double Bs[kBigPanelMax][kTileLdU];
  double ud[3 * kBlk], usinv[kBlk];  // the panel's D^-1, when L is formed from W
  int ukind[kBlk];
};

struct Prefix {  // work items of up to kChunkFronts fronts
  long long ptr[kChunkFronts + 1];
  long long wsum[kWarps];
};

// What a work item needs of its front, gathered by front_prefix so that an
// item does not start with a chain of global loads.
struct Info {
  double *F, *W, *X;
  int f, k, nbk, np;  // np: pivots accepted in the block (phase R) or passing
  int rows;           // row chunks (phases R and A); 0: not in this step
  int moved;
  int swaps, swap_b;  // interchanges left to phase R
};

constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
// the mixed-precision tile places the tensor-core operands after the FP64
// tiles' panels, 1 KB aligned
constexpr size_t kOpsOffset = (sizeof(UpdSm) + 1023) / 1024 * 1024;
// the work items' fronts come first, then what the phase uses
constexpr size_t kInfoBytes = (sizeof(Info) * kChunkFronts + 1023) / 1024 * 1024;
constexpr size_t kDynSmem =
    kInfoBytes + cmax(sizeof(WarpDiag) * kWarps,
                      cmax(sizeof(RowsSm), kOpsOffset + umma::kSmemFloats * sizeof(float)));

// Exclusive prefix of cnt(i) over i in [0, nl) into P.ptr (CTA-wide; nl <=
// kChunkFronts). Returns the total. A thread counts one front per round, so
// that the chains of loads of cnt run side by side.
template <typename Count>
__device__ long long front_prefix(Prefix& P, int nl, Count cnt) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int w = tid >> 5;
  long long base = 0;
  if (tid == 0) P.ptr[0] = 0;
  for (int i0 = 0; i0 < nl; i0 += kThreads) {
    const int i = i0 + tid;
    long long incl = (i < nl) ? cnt(i) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) P.wsum[w] = incl;
    __syncthreads();
    long long before = base, all = base;
#pragma unroll
    for (int q = 0; q < kWarps; q++) {
      const long long v = P.wsum[q];
      if (q < w) before += v;
      all += v;
    }
    if (i < nl) P.ptr[i + 1] = before + incl;
    base = all;
    __syncthreads();
  }
  return base;
}

// front of work item t: the last i with ptr[i] <= t
__device__ __forceinline__ int item_front(const Prefix& P, int nl, long long t) {
  int lo = 0, hi = nl;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (P.ptr[mid] <= t)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// ---------------------------------------------------------------- phase D

// A front whose candidates are all decided is done, except a root with
// candidates left (delayed by the tests; a root has no parent to take them):
// they become candidates again and the root waits in `done` for the chained
// panels (Bunch-Kaufman) that run after this launch.
__device__ void finish_front(const DevState& s, BigFront* B, int* done, int* meta) {
  if (B->nc == 0 && B->k < B->fs) {
    B->ncand = B->fs;
    B->state = 3;
    done[atomicAdd(meta + 19, 1)] = (int)(B - s.big);
    atomicMax(meta + 20, B->fs - B->k);
  } else {
    B->state = 2;
  }
}

template <int NT>
__device__ __forceinline__ void group_sync() {
  if constexpr (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}

// Close the previous step of front B (trailing-update work counters, a
// finished front becomes done) and apply the delays it left, by a group of
// NT threads (a warp, or the CTA when the level has no more fronts than
// CTAs); g is the thread's index in the group. Returns 1 if the front takes
// part in this step.
template <int NT>
__device__ int phase_d_prepare(const DevState& s, BigFront* B, int* done, int* meta, int g,
                               WarpDiag& w) {
  const int f = B->f;
  double* F = s.dpool + B->doff;
  double* X = s.dpool + B->xoff;
  int* xi = xint(X);
  int* fv = s.ivars + B->ioff;
  int* orig = fv + f;
  if (g == 0 && B->kw > 0) {
    const double r = (double)(f - B->k);
    const double fl = r * (r + 1.0) * B->kw;
    B->flops += fl;
    atomicAdd(s.flops + 2, fl);
    atomicAdd(s.flops + 3, 8.0 * (r * (r + 1.0) + 2.0 * r * B->kw));
  }
  group_sync<NT>();
  if (g == 0) {
    B->kw = 0;
    if (B->state == 1) finish_front(s, B, done, meta);
  }
  group_sync<NT>();
  int swaps = 0;
  if (B->pending > 0 && B->state == 0) {
    // The candidates to delay move behind the remaining candidates, largest
    // position first so that no interchange moves another one still to go.
    // Only the entries between the next block's rows and the rows behind the
    // candidates are exchanged here (what the block and the maxima need):
    // one CTA would take 15,000 cycles and more for a 3,600-row front's rows,
    // an 8-byte access per column, so every other row is left to phase R,
    // whose items own the rows. A front that is done with its candidates has
    // no phase R: all its rows are exchanged at once.
    const int nd = xi[kIDcnt];
    const int k = B->k;
    const int n0 = B->ncand;
    const int n1 = n0 - nd;
    const bool all = k >= n1;
    const int blk1 = min(k + kBlk, f);  // rows of the block
    const int far = max(n1, blk1);      // and of [n1, n0) beyond it
    const int near = blk1 - k;
    const int few = near + max(0, n0 - far);
    if (!all && g < kBlk) {
      // what stands at the block's positions, and at [n1, n0)
      w.perm[g] = k + g;
      w.part[g] = n0 - 1 - g;
    }
    // The next panel's first test needs the exact maximum below the block
    // (rows from k + kBlk on) of every block column. An interchange of rows
    // a (in the block) and b (below it) takes row b's entry out of a
    // column's rows below and puts the entry of row a in: thread g < kBlk
    // follows column k + g, which is formed again afterwards only if the
    // entry taken out may have been its maximum, or if it is a or b.
    const int ct = k + g;
    const bool trk = g < kBlk && ct < f;
    bool stale = false;
    double mx = trk ? X[kXNext + g] : 0.0;
    group_sync<NT>();
    for (int q = 0; q < nd; q++) {
      const int a = xi[kIDpos + q];
      const int b = n0 - 1 - q;
      if (a < b) {
        if (trk) {
          if (ct == a || ct == b) {
            stale = true;
          } else if (b >= k + kBlk) {
            const double out = fabs(fsym(F, f, b, ct)), in = fabs(fsym(F, f, a, ct));
            if (out >= mx) stale = true;
            mx = fmax(mx, in);
          }
        }
        group_sync<NT>();  // those reads before the interchange
        // the pairs of a symmetric interchange are distinct entries: eight
        // passes of the group load theirs before any is stored back
        constexpr int kU = 8;
        const int nj = all ? f : few;
        for (int j0 = 0; j0 < nj; j0 += NT * kU) {
          double* p[kU];
          double* r[kU];
          double vp[kU], vr[kU];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int jj = j0 + NT * u + g;
            p[u] = nullptr;
            r[u] = nullptr;
            const int j = all ? jj : jj < near ? k + jj : far + jj - near;
            if (jj >= nj || j == b) continue;
            if (j < a) {
              p[u] = F + a + (size_t)f * j;
              r[u] = F + b + (size_t)f * j;
            } else if (j == a) {
              p[u] = F + a + (size_t)f * a;
              r[u] = F + b + (size_t)f * b;
            } else if (j < b) {
              p[u] = F + j + (size_t)f * a;
              r[u] = F + b + (size_t)f * j;
            } else {
              p[u] = F + j + (size_t)f * a;
              r[u] = F + j + (size_t)f * b;
            }
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            vp[u] = p[u] ? *p[u] : 0.0;
            vr[u] = p[u] ? *r[u] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            if (p[u]) {
              *p[u] = vr[u];
              *r[u] = vp[u];
            }
          }
        }
        if (g == 0) {
          int t = fv[a];
          fv[a] = fv[b];
          fv[b] = t;
          t = orig[a];
          orig[a] = orig[b];
          orig[b] = t;
          if (!all) {
            int* pa = w.perm + (a - k);
            int* pb = b < blk1 ? w.perm + (b - k) : w.part + q;
            t = *pa;
            *pa = *pb;
            *pb = t;
          }
        }
      }
      group_sync<NT>();
    }
    // the block columns whose maximum below may have changed, formed again
    unsigned redo;
    if constexpr (NT == 32) {
      redo = __ballot_sync(0xffffffffu, trk && stale);
    } else {
      __shared__ unsigned redo_sh;
      if (g < 32) {
        const unsigned m = __ballot_sync(0xffffffffu, trk && stale);
        if (g == 0) redo_sh = m;
      }
      group_sync<NT>();
      redo = redo_sh;
    }
    if (trk && !stale) X[kXNext + g] = mx;
    const int lane = g & 31;
    // a column is read by the whole group, eight entries of a thread in
    // flight; non-negative doubles order as their bits
    for (unsigned left = all ? 0u : redo; left; left &= left - 1) {
      const int i = __ffs(left) - 1;
      if (g == 0) X[kXNext + i] = 0.0;
      group_sync<NT>();
      // rows not yet exchanged have the column where it stood
      const int was = w.perm[i];
      unsigned long long m = 0;
      for (int r0 = k + kBlk; r0 < f; r0 += 8 * NT) {
        unsigned long long e[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int r = r0 + NT * u + g;
          const int c = (r >= n1 && r < n0) ? k + i : was;
          e[u] = r < f ? (unsigned long long)__double_as_longlong(fabs(fsym(F, f, r, c))) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (e[u] <= kInfBits && e[u] > m) m = e[u];  // NaN entries do not take part
      }
      const double wm = warp_max(__longlong_as_double((long long)m));
      if (lane == 0 && wm > 0.0)
        atomicMax(reinterpret_cast<unsigned long long*>(X + kXNext) + i,
                  (unsigned long long)__double_as_longlong(wm));
    }
    group_sync<NT>();
    if (g == 0) {
      B->ncand = n1;
      B->pending = 0;
      xi[kISwapB] = n0;
      if (all) finish_front(s, B, done, meta);
    }
    swaps = all ? 0 : nd;
    group_sync<NT>();
  }
  if (g == 0) xi[kISwaps] = swaps;
  return B->state == 0 ? 1 : 0;
}

// Factor the next diagonal block of front B (one warp). Returns 1.
__device__ int phase_d_block(const DevState& s, const FactorParams& prm, BigFront* B, int step,
                             WarpDiag& w) {
  const int lane = threadIdx.x & 31;
  const int f = B->f;
  double* F = s.dpool + B->doff;
  double* Wg = s.dpool + B->woff;
  double* X = s.dpool + B->xoff;
  int* xi = xint(X);
  int* fv = s.ivars + B->ioff;
  int* orig = fv + f;

  const int k = B->k;
  const int ncand = B->ncand;
  const int nbk = max(0, min(kBlk, ncand - k));
  bool finite;     // every entry of the block is finite
  unsigned hints;  // positions whose candidate was in a 2x2 with the next one
  {
    // the block's lower triangle, one coalesced column per load (all loads
    // in flight before the shared-memory stores), mirrored above
    double v[kBlk];
#pragma unroll
    for (int j = 0; j < kBlk; j++)
      v[j] = (j <= lane && lane < nbk) ? F[(k + lane) + (size_t)f * (k + j)] : 0.0;
    // the candidates' variables and the partners they had in the record
    const int var = (lane < nbk) ? fv[k + lane] : -1;
    const int part = (var >= 0 && s.partner) ? s.partner[var] : -1;
    // entry (i, j) and its mirror are written by lane max(i, j) only
#pragma unroll
    for (int j = 0; j < kBlk; j++) {
      if (j <= lane) {
        w.A[lane][j] = v[j];
        w.A[j][lane] = v[j];
      }
      w.Lb[lane][j] = 0.0;
    }
    w.var[lane] = var;
    w.part[lane] = part;
    int top = 0;
#pragma unroll
    for (int j = 0; j < kBlk; j++) top = max(top, __double2hiint(v[j]) & 0x7fffffff);
    finite = __all_sync(0xffffffffu, top < 0x7ff00000);
    const int vnext = __shfl_down_sync(0xffffffffu, var, 1);
    hints = __ballot_sync(0xffffffffu, lane < 31 && var >= 0 && vnext >= 0 && part == vnext);
  }
  w.perm[lane] = lane;
  w.dlt[lane] = -1;
  // of the pivot at position `lane`: its kind, D, and the block's part of its
  // column maximum and of its 2x2 partner's (left at 0 for a 1x1 that passed
  // where it stood: it passed against those entries already)
  int kind = 0;
  double dd0 = 0.0, dd1 = 0.0, dd2 = 0.0, cin = 0.0, rin = 0.0;
  // (partly the result of atomics: read from L2)
  w.below0[lane] = __ldcg(X + kXNext + lane);
  // read: the trailing update of this panel fills them again for the next
  X[kXNext + lane] = 0.0;
  __syncwarp();

  // The reference's tests on the block's candidates in order. For the
  // panel's first pivot the column maximum below the block is exact
  // (below0); after it nothing is known below, so the maximum used is a
  // lower bound: a candidate that fails on a lower bound fails on the true
  // maximum as well, so it is delayed, unless the a-posteriori tests reject
  // a pivot accepted before it. Accepted pivots are checked with the exact
  // maxima in phase A.
  const double u = prm.ustab, tol = prm.pivot_tol;
  constexpr unsigned kFull = 0xffffffffu;
  int t = 0, nr = nbk;
  // Left-looking: the block keeps its entries as loaded in the columns not
  // pivoted yet, next to the pivot columns (W) and the L rows of the pivots
  // taken. A column that a test reads is formed when it is read: entry
  // (i, j) minus L(max(i, j), q) W(min(i, j), q) for each earlier pivot q in
  // order, the products and the order of the reference's lower-triangle
  // update. Lane i forms row i.
  // One warp runs this alone, so what counts is its number of instructions:
  // two entries of a row per load, eight pivots' products at a time, and no
  // test of q against t: beyond t the L entries are still zero, and zero
  // times a finite entry as loaded leaves the sum as it is (a block with an
  // infinity or NaN goes pivot by pivot).
  auto form = [&](int j) -> double {
    const int hi = max(lane, j), lo = min(lane, j);
    double v = w.A[lane][j];
    if (finite) {
      const double2* lr = reinterpret_cast<const double2*>(w.Lb[hi]);
      const double2* wr = reinterpret_cast<const double2*>(w.A[lo]);
      for (int q0 = 0; q0 < t; q0 += 8) {
        double2 a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          a[q] = lr[q0 / 2 + q];
          b[q] = wr[q0 / 2 + q];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          v = fma(-a[q].x, b[q].x, v);
          v = fma(-a[q].y, b[q].y, v);
        }
      }
    } else {
      for (int q = 0; q < t; q++) v = fma(-w.Lb[hi][q], w.A[lo][q], v);
    }
    return (lane >= t && lane < nbk) ? v : 0.0;
  };
  while (t < nr) {
    const bool has = t + 1 < nr;
    const bool hinted = has && ((hints >> t) & 1u);
    const double ct = form(t);  // the candidate's column
    double c2 = 0.0;            // and its recorded partner's, or imax's
    if (hinted) c2 = form(t + 1);
    const double wkk = __shfl_sync(kFull, ct, t);
    const double at = fabs(ct);
    if (!hinted) {
      // the common pivot, a 1x1 that passes where it stands: every lane tests
      // its entry (rounded products are monotone, so that is the test against
      // the largest one), while the reciprocal is formed
      const double rd = 1.0 / wkk;
      bool ok = fabs(wkk) >= tol;
      if (lane > t && lane < nbk) ok = ok && fabs(wkk) >= u * at;
      if (t == 0) ok = ok && fabs(wkk) >= u * w.below0[w.perm[0]];
      if (__all_sync(kFull, ok)) {
        if (lane >= t && lane < nbk) w.A[lane][t] = ct;
        if (lane > t && lane < nbk) w.Lb[lane][t] = ct * rd;
        if (lane == t) {
          kind = 1;
          dd0 = wkk;
        }
        __syncwarp();
        t++;
        continue;
      }
    }
    double bv;
    int bi;
    warp_argmax(lane > t && lane < nr, at, bv, bi);
    const double abswik = has ? bv : 0.0;
    const int imax = has ? bi : t;
    // block rows that are not candidates any more (rotated behind)
    const double cnc = (nr < nbk) ? warp_max((lane >= nr && lane < nbk) ? at : 0.0) : 0.0;
    const double col_in = fmax(abswik, cnc);
    const double colmax = fmax(col_in, t == 0 ? w.below0[w.perm[t]] : 0.0);
    int stp = 0, kpiv = t;
    double row_in = 0.0;
    // a pair that formed a 2x2 pivot in the pivot record is tried as that
    // 2x2 first (the Duff test), since a 1x1 test that sees only the block's
    // rows would accept the first of them alone and the a-posteriori test
    // would then reject it
    if (hinted) {
      const double r2 = warp_max((lane >= t && lane < nbk && lane != t + 1) ? fabs(c2) : 0.0);
      const double rm2 = fmax(r2, t == 0 ? w.below0[w.perm[t + 1]] : 0.0);
      const double w21 = __shfl_sync(kFull, ct, t + 1), w22 = __shfl_sync(kFull, c2, t + 1);
      const double det = fabs(wkk * w22 - w21 * w21);
      if (det >= tol) {
        const double delta = det / fmax(fabs(w22) + fabs(w21), fabs(wkk) + fabs(w21));
        if (delta >= u * colmax && delta >= u * rm2) {
          stp = 2;
          kpiv = t + 1;
          row_in = r2;
        }
      }
    }
    if (stp != 0) {
      // taken as recorded
    } else if (fabs(wkk) >= tol && fabs(wkk) >= u * colmax) {
      stp = 1;
    } else if (has) {
      c2 = form(imax);
      row_in = warp_max((lane >= t && lane < nbk && lane != imax) ? fabs(c2) : 0.0);
      const double rowmax = fmax(row_in, t == 0 ? w.below0[w.perm[imax]] : 0.0);
      const double wii = __shfl_sync(kFull, c2, imax), wik = __shfl_sync(kFull, ct, imax);
      if (fabs(wii) >= tol && fabs(wii) >= u * rowmax) {
        stp = 1;
        kpiv = imax;
      } else {
        const double det = fabs(wkk * wii - wik * wik);
        if (det >= tol) {
          const double delta = det / fmax(fabs(wii) + abswik, fabs(wkk) + abswik);
          if (delta >= u * colmax && delta >= u * rowmax) {
            stp = 2;
            kpiv = imax;
          }
        }
      }
    }
    // interchange: the accepted pivot to position t (+1), or the failing
    // candidate behind the block's candidates
    const int ksrc = (stp == 0) ? t : t + stp - 1;
    const int kdst = (stp == 0) ? nr - 1 : kpiv;
    if (ksrc != kdst) {
      {
        const double x = w.A[ksrc][lane];
        w.A[ksrc][lane] = w.A[kdst][lane];
        w.A[kdst][lane] = x;
        const double y = w.Lb[ksrc][lane];
        w.Lb[ksrc][lane] = w.Lb[kdst][lane];
        w.Lb[kdst][lane] = y;
      }
      __syncwarp();
      {
        const double x = w.A[lane][ksrc];
        w.A[lane][ksrc] = w.A[lane][kdst];
        w.A[lane][kdst] = x;
      }
      if (lane == 0) {
        int q = w.perm[ksrc];
        w.perm[ksrc] = w.perm[kdst];
        w.perm[kdst] = q;
        q = w.dlt[ksrc];
        w.dlt[ksrc] = w.dlt[kdst];
        w.dlt[kdst] = q;
      }
      __syncwarp();
      const int pl = w.perm[lane];
      const int vn = lane < 31 ? w.var[w.perm[lane + 1]] : -1;
      hints = __ballot_sync(kFull, w.var[pl] >= 0 && vn >= 0 && w.part[pl] == vn);
    }
    if (stp == 0) {
      if (lane == 0) w.dlt[nr - 1] = t;
      __syncwarp();
      nr--;
      continue;
    }
    // the pivot columns at their positions after the interchange (rows
    // ksrc and kdst exchanged), stored as W for the later columns
    const int src = (lane == ksrc) ? kdst : (lane == kdst) ? ksrc : lane;
    const double p1 = __shfl_sync(kFull, (stp == 1 && kpiv != t) ? c2 : ct, src);
    const double p2 = __shfl_sync(kFull, c2, src);
    if (lane >= t && lane < nbk) {
      w.A[lane][t] = p1;
      if (stp == 2) w.A[lane][t + 1] = p2;
    }
    if (stp == 1) {
      const double d = __shfl_sync(kFull, p1, t);
      const double li = p1 * (1.0 / d);
      if (lane > t && lane < nbk) w.Lb[lane][t] = li;
      if (lane == t) {
        kind = 1;
        dd0 = d;
        cin = (kpiv == t) ? col_in : row_in;
      }
    } else {
      const double d11 = __shfl_sync(kFull, p1, t), d21 = __shfl_sync(kFull, p1, t + 1),
                   d22 = __shfl_sync(kFull, p2, t + 1);
      // the expressions of the commit and of the update tiles (l_2x2)
      const double dv[3] = {d11, d21, d22};
      double l0, l1;
      l_2x2(dv, p1, p2, l0, l1);
      if (lane > t + 1 && lane < nbk) {
        w.Lb[lane][t] = l0;
        w.Lb[lane][t + 1] = l1;
      }
      if (lane == t) {
        kind = 2;
        dd0 = d11;
        dd1 = d21;
        dd2 = d22;
        cin = col_in;
        rin = row_in;
      }
      if (lane == t + 1) kind = 3;
    }
    __syncwarp();
    t += stp;
  }
  const int acc = t;
  const bool moved = __ballot_sync(0xffffffffu, lane < nbk && w.perm[lane] != lane) != 0u;

  // panel state for phases R and A
#pragma unroll 8
  for (int q = lane; q < kBlk * kLd; q += 32) X[kXL + q] = (&w.Lb[0][0])[q];
  X[kXD + 3 * lane] = dd0;
  X[kXD + 3 * lane + 1] = dd1;
  X[kXD + 3 * lane + 2] = dd2;
  X[kXCin + lane] = cin;
  X[kXRin + lane] = rin;
  X[kXBelow + lane] = 0.0;
  xi[kIPerm + lane] = w.perm[lane];
  xi[kIKind + lane] = kind;
  xi[kIDlt + lane] = w.dlt[lane];
  if (lane == 0) {
    xi[kIRdone] = 0;
    xi[kIAcc] = acc;
    xi[kINbk] = nbk;
    xi[kIK] = k;
    xi[kIStep] = step;
    xi[kINcand] = ncand;
    xi[kIMoved] = moved ? 1 : 0;
  }
  // the W values of the block rows for the trailing update
  for (int p = 0; p < acc; p++)
    if (lane > p && lane < nbk) Wg[(size_t)p * f + k + lane] = w.A[lane][p];
  if (moved) {
    // the block itself and the variables follow the interchanges (the factor
    // rows of earlier panels move in phase R): lane i gathers its row
    // before any lane writes
    double v[kBlk];
#pragma unroll
    for (int j = 0; j < kBlk; j++)
      v[j] = (j <= lane && lane < nbk) ? fsym(F, f, k + w.perm[lane], k + w.perm[j]) : 0.0;
    const int a = (lane < nbk) ? fv[k + w.perm[lane]] : 0;
    const int b = (lane < nbk) ? orig[k + w.perm[lane]] : 0;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kBlk; j++)
      if (j <= lane && lane < nbk) F[(k + lane) + (size_t)f * (k + j)] = v[j];
    if (lane < nbk) {
      fv[k + lane] = a;
      orig[k + lane] = b;
    }
  }
  __syncwarp();
  return 1;
}

// ---------------------------------------------------------------- phase R

__device__ __forceinline__ bool active(const DevState& s, const BigFront& B, int step) {
  return xint(s.dpool + B.xoff)[kIStep] == step;
}

// The part of a front's Info that does not change during the launch.
__device__ __forceinline__ void front_place(const DevState& s, const BigFront& B, Info& o) {
  o.F = s.dpool + B.doff;
  o.W = s.dpool + B.woff;
  o.X = s.dpool + B.xoff;
  o.f = B.f;
}

// The rest for this step: row chunks of the front, 0 if it takes no part.
__device__ __forceinline__ int front_step(int step, Info& o) {
  const int* xi = xint(o.X);
  const int st = xi[kIStep], k = xi[kIK], nbk = xi[kINbk], acc = xi[kIAcc];
  const int moved = xi[kIMoved], swaps = xi[kISwaps], swap_b = xi[kISwapB];
  o.k = k;
  o.nbk = nbk;
  o.np = acc;
  o.moved = moved;
  o.swaps = swaps;
  o.swap_b = swap_b;
  o.rows = st == step ? max(1, (o.f - (k + nbk) + kThreads - 1) / kThreads) : 0;
  return o.rows;
}

__device__ void phase_r_item(const FactorParams& prm, const Info& o, int chunk, RowsSm& sm) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  double* X = o.X;
  int* xi = xint(X);
  const int f = o.f;
  const int k = o.k;
  const int nbk = o.nbk;
  const int acc = o.np;
  const int nchunk = o.rows;
  double* F = o.F;
  double* Wg = o.W;
  const int r = k + nbk + chunk * kThreads + tid;
  {
    // the block's L, and where the block's rows come from
    constexpr int kPer = (kBlk * kLd + kThreads - 1) / kThreads;
    double t[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const int q = tid + kThreads * u;
      t[u] = q < kBlk * kLd ? X[kXL + q] : 0.0;
    }
    if (tid < kBlk) sm.sperm[tid] = xi[kIPerm + tid];
    // transposed: phase R takes L column by column, two entries per load
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const int q = tid + kThreads * u;
      if (q < kBlk * kLd && q % kLd < kBlk) sm.Ls[q % kLd][q / kLd] = t[u];
    }
  }
  // the delays' interchanges on the rows that phase D left: this thread's
  // row, and the warp's share of the earlier panels' factor columns
  if (o.swaps > 0) {
    const int* dpos = xi + kIDpos;
    if (r >= k + kBlk && r < f && (r < o.swap_b - o.swaps || r >= o.swap_b)) {
      for (int q = 0; q < o.swaps; q++) {
        const int x = dpos[q], y = o.swap_b - 1 - q;
        if (x >= y) continue;
        double* p = F + r + (size_t)f * x;
        double* z = r > y ? F + r + (size_t)f * y : F + y + (size_t)f * r;
        const double vp = *p, vz = *z;
        *p = vz;
        *z = vp;
      }
    }
    for (int j = (chunk * kWarps + warp) + lane * nchunk * kWarps; j < k;
         j += 32 * nchunk * kWarps) {
      for (int q = 0; q < o.swaps; q++) {
        const int x = dpos[q], y = o.swap_b - 1 - q;
        if (x >= y) continue;
        double* p = F + x + (size_t)f * j;
        double* z = F + y + (size_t)f * j;
        const double vp = *p, vz = *z;
        *p = vz;
        *z = vp;
      }
    }
  }
  __syncthreads();
  double a[kBlk];
#pragma unroll
  for (int j = 0; j < kBlk; j++)
    a[j] = (r < f && j < nbk) ? F[r + (size_t)f * (k + sm.sperm[j])] : 0.0;
  if (o.moved) {
    // the block's rows in the factor columns of earlier panels: a warp takes
    // eight columns at a time, lane i moves row k + perm[i] to row k + i
    const bool mv = lane < nbk && sm.sperm[lane] != lane;
    const int from = mv ? k + sm.sperm[lane] : 0;
    for (int j0 = chunk * kWarps + warp; j0 < k; j0 += 8 * nchunk * kWarps) {
      double t[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int j = j0 + u * nchunk * kWarps;
        t[u] = (mv && j < k) ? F[from + (size_t)f * j] : 0.0;
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int j = j0 + u * nchunk * kWarps;
        if (mv && j < k) F[(k + lane) + (size_t)f * j] = t[u];
      }
    }
    if (r < f) {
#pragma unroll
      for (int j = 0; j < kBlk; j++)
        if (j < nbk) F[r + (size_t)f * (k + j)] = a[j];
    }
  }
  // W = F21 L11^-T: forward substitution with the block's unit lower L,
  // column by column (the later entries' chains run side by side)
#pragma unroll
  for (int q = 0; q < kBlk; q++) {
    if (q < acc) {
      if (r < f) Wg[(size_t)q * f + r] = a[q];
      const double2* l = reinterpret_cast<const double2*>(sm.Ls[q]);
#pragma unroll
      for (int p2 = (q + 1) / 2; p2 < kBlk / 2; p2++) {
        const double2 lp = l[p2];
        if (2 * p2 > q) a[2 * p2] = fma(-a[q], lp.x, a[2 * p2]);
        a[2 * p2 + 1] = fma(-a[q], lp.y, a[2 * p2 + 1]);
      }
    }
  }
  // Column maxima (non-negative doubles order as their bits; NaN entries do
  // not take part): with every halving of the warp a lane keeps half of the
  // columns, then the CTA's and the front's maxima.
  {
    unsigned long long m[kBlk];
#pragma unroll
    for (int p = 0; p < kBlk; p++) {
      const unsigned long long e =
          (unsigned long long)__double_as_longlong(a[p]) & 0x7fffffffffffffffull;
      m[p] = (p < acc && r < f && e <= kInfBits) ? e : 0ull;
    }
#pragma unroll
    for (int n = kBlk / 2; n >= 1; n >>= 1) {
      const bool up = lane & n;
#pragma unroll
      for (int i = 0; i < n; i++) {
        const unsigned long long keep = up ? m[i + n] : m[i];
        const unsigned long long send = up ? m[i] : m[i + n];
        const unsigned long long got = __shfl_xor_sync(0xffffffffu, send, n);
        m[i] = keep > got ? keep : got;
      }
    }
    sm.red[warp][lane] = __longlong_as_double((long long)m[0]);  // column `lane`
  }
  __syncthreads();
  if (tid < acc) {
    double v = 0.0;
    for (int q = 0; q < kWarps; q++) v = fmax(v, sm.red[q][tid]);
    if (v > 0.0)
      atomicMax(reinterpret_cast<unsigned long long*>(X + kXBelow) + tid,
                (unsigned long long)__double_as_longlong(v));
  }
  // the front's last item to finish has the column maxima over the whole
  // front: it runs the reference's tests on the block's pivots and records
  // how many pass (kINp), for the commit and the trailing update
  __threadfence();
  __syncthreads();
  if (tid == 0) sm.np = (atomicAdd(xi + kIRdone, 1) == nchunk - 1) ? 1 : 0;
  __syncthreads();
  if (sm.np) {
    __threadfence();
    if (tid < kBlk) {
      sm.skind[tid] = xi[kIKind + tid];
      sm.sd[3 * tid] = X[kXD + 3 * tid];
      sm.sd[3 * tid + 1] = X[kXD + 3 * tid + 1];
      sm.sd[3 * tid + 2] = X[kXD + 3 * tid + 2];
      const unsigned long long bl =
          *(reinterpret_cast<volatile unsigned long long*>(X + kXBelow) + tid);
      sm.scm[tid] = fmax(X[kXCin + tid], __longlong_as_double((long long)bl));
      sm.srm[tid] = X[kXRin + tid];
      __syncwarp();
      const int np = passing_prefix(sm, acc, prm.ustab, prm.pivot_tol);
      if (tid == 0) xi[kINp] = np;
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- phase A


__device__ void phase_a_item(const DevState& s, BigFront* B, const Info& o, int chunk,
                             RowsSm& sm) {
  const int tid = threadIdx.x;
  double* X = o.X;
  int* xi = xint(X);
  const int f = o.f;
  const int k = o.k;
  const int nbk = o.nbk;
  const int np = o.np;
  double* F = o.F;
  const double* Wg = o.W;
  const int r = k + nbk + chunk * kThreads + tid;
  // the row's W entries, all loads in flight
  double w[kBlk];
#pragma unroll
  for (int p = 0; p < kBlk; p++) w[p] = (r < f && p < np) ? Wg[(size_t)p * f + r] : 0.0;
  if (chunk == 0)
    for (int t = tid; t < kBlk * kLd; t += kThreads) (&sm.Ls[0][0])[t] = X[kXL + t];
  if (tid < kBlk) {
    const int kd = xi[kIKind + tid];
    const double d[3] = {X[kXD + 3 * tid], X[kXD + 3 * tid + 1], X[kXD + 3 * tid + 2]};
    sm.skind[tid] = kd;
    sm.sd[3 * tid] = d[0];
    sm.sd[3 * tid + 1] = d[1];
    sm.sd[3 * tid + 2] = d[2];
    // 1x1 pivots scale their column by 1/d, as the reference does
    sm.sinv[tid] = (kd == 1) ? 1.0 / d[0] : 0.0;
    if (kd == 2) inv_2x2(d, sm.inv[tid]);
  }
  __syncthreads();
  // L of the accepted pivots on the rows below the block
  if (r < f) {
    double* Fr = F + r + (size_t)f * k;
#pragma unroll
    for (int p = 0; p < kBlk; p++) {
      if (p < np) {
        const int kd = sm.skind[p];
        double l = 0.0;
        if (kd == 1) l = w[p] * sm.sinv[p];
        if (p + 1 < kBlk && kd == 2) l = l_first(sm.inv[p], w[p], w[p + 1]);
        if (p > 0 && kd == 3) l = l_second(sm.inv[p - 1], w[p - 1], w[p]);
        Fr[(size_t)f * p] = l;
      }
    }
  }
  if (chunk == 0) {
    // the block's rows: D on the diagonal (d21 below a 2x2's first column), L
    for (int t = tid; t < kBlk * kBlk; t += kThreads) {
      const int i = t % kBlk, p = t / kBlk;
      if (p >= np || i < p || i >= nbk) continue;
      double v;
      if (i == p)
        v = (sm.skind[p] == 3) ? sm.sd[3 * (p - 1) + 2] : sm.sd[3 * p];
      else if (i == p + 1 && sm.skind[p] == 2)
        v = sm.sd[3 * p + 1];
      else
        v = sm.Ls[i][p];
      F[(k + i) + (size_t)f * (k + p)] = v;
    }
    if (tid < 32) {
      // commit the panel (the other items of this front read only the
      // scratch, never the descriptor), a lane per pivot
      int* fv = s.ivars + B->ioff;
      const int p = tid;
      const int kd = p < np ? sm.skind[p] : 0;
      int npos = 0, nneg = 0;
      double fl = 0.0;
      if (kd == 1) {
        if (sm.sd[3 * p] >= 0.0)
          npos = 1;
        else
          nneg = 1;
        fl = 2.0 * (double)(f - k - p) * (p + 1);
      } else if (kd == 2) {
        const double d11 = sm.sd[3 * p], d21 = sm.sd[3 * p + 1], d22 = sm.sd[3 * p + 2];
        const double det = d11 * d22 - d21 * d21;
        if (det >= 0.0) {
          if (d11 >= 0.0)
            npos = 2;
          else
            nneg = 2;
        } else {
          npos = 1;
          nneg = 1;
        }
        fl = 4.0 * (double)(f - k - p) * (p + 2);
      }
      if (kd >= 2) fv[k + p] = -(fv[k + p] + 1);
      // candidates to delay: those that failed in the block while only
      // pivots that are now accepted preceded them, and the first pivot the
      // a-posteriori tests reject (positions decreasing); candidates that
      // failed after a rejected pivot are tried again
      const int acc = xi[kIAcc];
      const int ncand = xi[kINcand];
      const int dlt = (p >= acc && p < nbk) ? xi[kIDlt + p] : -1;
      const unsigned late = __ballot_sync(0xffffffffu, dlt >= 0 && dlt <= np);
      if ((late >> p) & 1u) xi[kIDpos + __popc(late >> p) - 1] = k + p;
      const int nlate = __popc(late);
      if (p == 0 && np < acc) xi[kIDpos + nlate] = k + np;
      const int nd = nlate + (np < acc ? 1 : 0);
      npos = __reduce_add_sync(0xffffffffu, npos);
      nneg = __reduce_add_sync(0xffffffffu, nneg);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) fl += __shfl_xor_sync(0xffffffffu, fl, d);
      if (p == 0) {
        xi[kIDcnt] = nd;
        B->kstart = k;
        B->kw = np;
        B->k = k + np;
        B->pending = nd;
        B->npos += npos;
        B->nneg += nneg;
        B->flops += fl;
        atomicAdd(s.flops + 1, fl);
        atomicAdd(s.flops + 5, 1.0);
        if (np < acc) atomicAdd(s.flops + 6, 1.0);
        atomicAdd(s.flops + 7, (double)nlate);
        B->state = (nd == 0 && k + np >= ncand) ? 1 : 0;
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- phase U

// One 64 x 64 lower tile of a front's trailing matrix at rows i0, columns j0:
// the rank-kw update with the panel's L (columns ks..ks+kw) and W, in FP64;
// k = ks + kw is the trailing matrix's first position. L is read from the
// front's columns once committed, or (from_w) formed from W and the panel's D
// as the commit forms it.
//
// The products run as mma.m8n8k4.f64, which adds its four products to the
// accumulator one after another in the order of k, each with one rounding:
// the sums are those of a loop of fused multiply-adds, at an eighth of the
// instructions (the FP64 rate is the same, but a tile was bound by issuing
// multiply-adds, operand loads and addresses). The next tile's loads are in
// flight while one is computed.
struct Tile {
  double *F, *W, *X;
  int f, i0, j0, k, kw, ks;
};

struct TileRegs {
  static constexpr int kPer = kBigPanelMax * kTileU / kThreads;
  double cur[4][2][2];  // this thread's entries: blocks of 8 rows, of 8 columns
  // W (or L) at row i0 + tid % 64 of the columns 8 (tid / 64) - 1 .. + 8, and
  // W at row j0 + tid % 64 of the columns 8 (tid / 64) ..
  double pa[kPer + 2], pb[kPer];
  double d0, d1, d2;  // of thread c < 32: pivot column c's D
  int kd;
};

// warp w owns the tile's rows 32 (w % 2).. and columns 16 (w / 2)..; in a
// block of 8 x 8 lane l holds row l / 4 and columns 2 (l % 4), + 1
struct TileThread {
  int row, col;
  __device__ __forceinline__ TileThread() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    row = 32 * (warp & 1) + (lane >> 2);
    col = 16 * (warp >> 1) + 2 * (lane & 3);
  }
};

__device__ __forceinline__ void load_tile(const Tile& t, bool from_w, TileRegs& g) {
  const int tid = threadIdx.x;
  const int f = t.f;
  {
    const int rr = tid % kTileU, c0 = (tid / kTileU) * TileRegs::kPer;
    const int i = t.i0 + rr, j = t.j0 + rr;
    const double* pw = from_w ? t.W + i : t.F + i + (size_t)f * t.ks;
#pragma unroll
    for (int q = 0; q < TileRegs::kPer + 2; q++) {
      const int c = c0 + q - 1;
      const bool edge = q == 0 || q == TileRegs::kPer + 1;
      g.pa[q] = (i < f && c >= 0 && c < t.kw && (!edge || from_w)) ? pw[(size_t)f * c] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < TileRegs::kPer; q++)
      g.pb[q] = (j < f && c0 + q < t.kw) ? t.W[j + (size_t)f * (c0 + q)] : 0.0;
  }
  g.kd = 0;
  g.d0 = g.d1 = g.d2 = 0.0;
  if (from_w && tid < kBlk) {
    g.kd = xint(t.X)[kIKind + tid];
    g.d0 = t.X[kXD + 3 * tid];
    g.d1 = t.X[kXD + 3 * tid + 1];
    g.d2 = t.X[kXD + 3 * tid + 2];
  }
  const TileThread me;
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int j = t.j0 + me.col + 8 * b + e;
      const double* col = t.F + (size_t)f * j;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int i = t.i0 + me.row + 8 * a;
        g.cur[a][b][e] = (j < f && i < f && i >= j) ? col[i] : 0.0;
      }
    }
}

// the panel parts of g into shared memory, L formed (all threads; ends with a
// barrier). same: the tile is of the same front as the one before, whose D^-1
// is in place.
__device__ __forceinline__ void stage_tile(const Tile& t, bool from_w, bool same,
                                           const TileRegs& g, UpdSm& sm) {
  const int tid = threadIdx.x;
  if (from_w && !same) {
    if (tid < kBlk) {
      const double d[3] = {g.d0, g.d1, g.d2};
      sm.ukind[tid] = g.kd;
      sm.usinv[tid] = (g.kd == 1) ? 1.0 / g.d0 : 0.0;
      if (g.kd == 2) inv_2x2(d, sm.ud + 3 * tid);
    }
    __syncthreads();
  }
  const int rr = tid % kTileU, c0 = (tid / kTileU) * TileRegs::kPer;
#pragma unroll
  for (int q = 0; q < TileRegs::kPer; q++) {
    const int c = c0 + q;
    double l = g.pa[q + 1];
    if (from_w) {
      // L = W D^-1 on the tile's rows, the commit's expressions
      const int kd = c < t.kw ? sm.ukind[c] : 0;
      if (kd == 1)
        l = g.pa[q + 1] * sm.usinv[c];
      else if (kd == 2)
        l = l_first(sm.ud + 3 * c, g.pa[q + 1], g.pa[q + 2]);
      else if (kd == 3)
        l = l_second(sm.ud + 3 * (c - 1), g.pa[q], g.pa[q + 1]);
    }
    sm.As[c][rr] = l;
    sm.Bs[c][rr] = g.pb[q];
  }
  __syncthreads();
}

__device__ __forceinline__ void finish_tile(const Tile& t, const double (&cur)[4][2][2],
                                            const UpdSm& sm) {
  const int lane = threadIdx.x & 31;
  const int f = t.f, k = t.k;
  const TileThread me;
  const int row0 = me.row, c16 = me.col - 2 * (lane & 3) + (lane >> 2);
  double acc[4][2][2];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 2; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
  const double* ap = &sm.As[lane & 3][row0];
  const double* bp = &sm.Bs[lane & 3][c16];
  // columns at and beyond kw are zeros
  for (int c = 0; c < t.kw; c += 4) {
    double av[4], bv[2];
#pragma unroll
    for (int a = 0; a < 4; a++) av[a] = ap[c * kTileLdU + 8 * a];
#pragma unroll
    for (int b = 0; b < 2; b++) bv[b] = bp[c * kTileLdU + 8 * b];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 2; b++)
        asm volatile(
            "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(acc[a][b][0]), "+d"(acc[a][b][1])
            : "d"(av[a]), "d"(bv[b]));
  }
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int j = t.j0 + me.col + 8 * b + e;
      double* col = t.F + (size_t)f * j;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int i = t.i0 + me.row + 8 * a;
        if (j < f && i < f && i >= j) col[i] = cur[a][b][e] - acc[a][b][e];
      }
    }
  if (t.j0 == k && me.col < kBigPanelMax) {
    // the next panel's columns [k, k + 32): their largest magnitude over the
    // rows below the next block, for its first test (as bits; NaN entries do
    // not take part)
    unsigned long long* nxt =
        reinterpret_cast<unsigned long long*>(t.X + kAppNextColmax);
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        unsigned long long m = 0;
#pragma unroll
        for (int a = 0; a < 4; a++) {
          const int i = t.i0 + me.row + 8 * a;
          const unsigned long long x =
              (unsigned long long)__double_as_longlong(fabs(cur[a][b][e] - acc[a][b][e]));
          if (i < f && i >= k + kBigPanelMax && x <= kInfBits && x > m) m = x;
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
          if (x > m) m = x;
        }
        const int jj = me.col + 8 * b + e;
        if ((lane >> 2) == 0 && k + jj < f && m > 0) atomicMax(nxt + jj, m);
      }
  }
  __syncthreads();
}

__device__ __forceinline__ long long tri_tiles_rows(int rows, int tile) {
  const long long t = (rows + tile - 1) / tile;
  return t * (t + 1) / 2;
}

__device__ __forceinline__ long long tri_tiles(const BigFront& B, int tile) {
  return tri_tiles_rows(B.f - B.k, tile);
}

// tile lt of a lower triangle of T x T tiles, column by column: the CTAs that
// run at the same time then cover long stretches of the same columns (DRAM
// pages), and the tiles of the next panel's columns come first
__device__ __forceinline__ void tri_decode(long long lt, int T, int& I, int& J) {
  const int r = (int)((long long)T * (T + 1) / 2 - 1 - lt);  // row by row from the end
  int a = (int)((sqrtf(8.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
  while ((long long)(a + 1) * (a + 2) / 2 <= r) a++;
  while ((long long)a * (a + 1) / 2 > r) a--;
  J = T - 1 - a;
  I = T - 1 - (int)(r - (long long)a * (a + 1) / 2);
}

// Mixed precision: a 128 x 128 tile (I, J) of the trailing matrix. Tiles of
// the contribution block (columns from fs on: rows that the parent
// assembles, never pivoted in this front) take the update on the tensor
// cores (umma.cuh, 3xTF32 products accumulated in FP32); the others, which
// hold the fully summed columns whose pivots are still to be decided, stay
// in FP64 as four 64 x 64 tiles. Returns 1 if a tensor-core operation did
// not complete in time.
__device__ int phase_u_tile_mixed(const DevState& s, const BigFront& B, int I, int J, UpdSm& sm,
                                  float* ops, uint64_t* mbar, uint32_t* phase, uint32_t tmem) {
  const int f = B.f, k = B.k;
  const int i0 = k + I * umma::kTileM;
  const int j0 = k + J * umma::kTileN;
  if (j0 >= B.fs) {
    double* F = s.dpool + B.doff;
    const double* W = s.dpool + B.woff;
    return umma::tile_update(F, f, F + (size_t)f * B.kstart, f, W, f, i0, j0,
                             min(umma::kTileM, f - i0), min(umma::kTileN, f - j0), B.kw, I == J,
                             ops, mbar, phase, tmem);
  }
  for (int a = 0; a < 2; a++)
    for (int b = 0; b < 2; b++) {
      const int si = i0 + a * kTileU, sj = j0 + b * kTileU;
      if (si < f && sj < f && si + kTileU - 1 >= sj) {
        const Tile t = {s.dpool + B.doff, s.dpool + B.woff, s.dpool + B.xoff, f, si, sj,
                        B.k,             B.kw,             B.kstart};
        TileRegs g;
        load_tile(t, false, g);
        stage_tile(t, false, false, g, sm);
        finish_tile(t, g.cur, sm);
      }
    }
  return 0;
}

// ---------------------------------------------------------------- the level

__global__ void __launch_bounds__(kThreads, 1)
    app_level_kernel(DevState s, FactorParams prm, const int* __restrict__ list, int nl,
                     int max_steps, int* done, int* meta) {
  int* counters = meta + 21;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(1024) unsigned char dsm0[];
  Info* info = reinterpret_cast<Info*>(dsm0);
  unsigned char* dsm = dsm0 + kInfoBytes;
  __shared__ Prefix P;
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int gwarp = blockIdx.x * kWarps + warp;
  const int nwarp = gridDim.x * kWarps;
  // mixed precision: 128 tensor-memory columns per CTA for the accumulator
  uint32_t tmem = 0, phase = 0;
  int tc_fail = 0;
  if (prm.mixed) {
    if (warp == 0) umma::tmem_alloc_128(&tmem_slot);
    if (tid == 0) umma::mbar_init(&mbar);
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::);
    tmem = tmem_slot;
  }
  // where the fronts are (more of them than fit are looked up in every step)
  if (nl <= kChunkFronts)
    for (int i = tid; i < nl; i += kThreads) front_place(s, s.big[list[i]], info[i]);
  int step = 1;
  for (; step <= max_steps; step++) {
    // ---- D: a warp factors the front's block; its CTA applies the delays
    // where the level has no more fronts than CTAs, else the warp
    {
      WarpDiag& w = reinterpret_cast<WarpDiag*>(dsm)[warp];
      WarpDiag& w0 = reinterpret_cast<WarpDiag*>(dsm)[0];
      if (blockIdx.x == 0 && tid == 0) counters[(step + 1) & 1] = 0;
      if (nl <= (int)gridDim.x) {
        // a CTA per front: its threads apply the delays, warp 0 the block
        if ((int)blockIdx.x < nl) {
          BigFront* B = s.big + list[blockIdx.x];
          if (phase_d_prepare<kThreads>(s, B, done, meta, tid, w0) && warp == 0) {
            phase_d_block(s, prm, B, step, w);
            if (tid == 0) atomicAdd(counters + (step & 1), 1);
          }
        }
      } else {
        for (int i = gwarp; i < nl; i += nwarp) {
          BigFront* B = s.big + list[i];
          if (phase_d_prepare<32>(s, B, done, meta, tid & 31, w)) {
            phase_d_block(s, prm, B, step, w);
            if ((tid & 31) == 0) atomicAdd(counters + (step & 1), 1);
          }
        }
      }
    }
    grid.sync();
    if (*((volatile int*)(counters + (step & 1))) == 0) break;  // the same in every CTA
    // ---- R: row chunks of the active fronts
    for (int c0 = 0; c0 < nl; c0 += kChunkFronts) {
      const int n = min(kChunkFronts, nl - c0);
      const long long total = front_prefix(P, n, [&](int i) {
        if (nl > kChunkFronts) front_place(s, s.big[list[c0 + i]], info[i]);
        return (long long)front_step(step, info[i]);
      });
      RowsSm& sm = *reinterpret_cast<RowsSm*>(dsm);
      for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        const int fi = item_front(P, n, t);
        phase_r_item(prm, info[fi], (int)(t - P.ptr[fi]), sm);
      }
      __syncthreads();
    }
    grid.sync();
    if (!prm.mixed) {
      // ---- A and U together: the row chunks that write L and commit the
      // panel, then the trailing-update tiles, which form L from W and take
      // the panel's position from the scratch, not from the descriptor that
      // the commit changes meanwhile
      for (int c0 = 0; c0 < nl; c0 += kChunkFronts) {
        const int n = min(kChunkFronts, nl - c0);
        const long long total = front_prefix(P, n, [&](int i) {
          Info& o = info[i];
          if (nl > kChunkFronts) {
            front_place(s, s.big[list[c0 + i]], o);
            front_step(step, o);
          }
          if (o.rows == 0) return 0ll;
          o.np = xint(o.X)[kINp];
          return o.rows + (o.np > 0 ? tri_tiles_rows(o.f - (o.k + o.np), kTileU) : 0ll);
        });
        UpdSm& sm = *reinterpret_cast<UpdSm*>(dsm);
        // the CTA's items in turn; a tile's loads are issued before the tile
        // before it is computed
        auto tile_of = [&](long long t, Tile& o) {  // false: a row chunk
          const int fi = item_front(P, n, t);
          const Info& q = info[fi];
          const long long it = t - P.ptr[fi];
          if (it < q.rows) return false;
          int I, J;
          const int k = q.k + q.np;
          tri_decode(it - q.rows, (q.f - k + kTileU - 1) / kTileU, I, J);
          o = {q.F, q.W, q.X, q.f, k + I * kTileU, k + J * kTileU, k, q.np, q.k};
          return true;
        };
        Tile tile;
        TileRegs regs;
        bool have = false;
        const double* last = nullptr;  // whose D^-1 is in shared memory
        for (long long t = blockIdx.x; t < total; t += gridDim.x) {
          if (!have) {
            if (!tile_of(t, tile)) {
              const int fi = item_front(P, n, t);
              phase_a_item(s, s.big + list[c0 + fi], info[fi], (int)(t - P.ptr[fi]),
                           *reinterpret_cast<RowsSm*>(dsm));
              last = nullptr;
              continue;
            }
            load_tile(tile, true, regs);
          }
          stage_tile(tile, true, tile.X == last, regs, sm);
          last = tile.X;
          const Tile now = tile;
          double cur[4][2][2];
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 2; b++) {
              cur[a][b][0] = regs.cur[a][b][0];
              cur[a][b][1] = regs.cur[a][b][1];
            }
          have = t + gridDim.x < total && tile_of(t + gridDim.x, tile);
          if (have) load_tile(tile, true, regs);
          finish_tile(now, cur, sm);
        }
        __syncthreads();
      }
      grid.sync();
      continue;
    }
    // ---- A: the same items; the first one of a front commits the panel
    for (int c0 = 0; c0 < nl; c0 += kChunkFronts) {
      const int n = min(kChunkFronts, nl - c0);
      const long long total = front_prefix(P, n, [&](int i) {
        Info& o = info[i];
        if (nl > kChunkFronts) {
          front_place(s, s.big[list[c0 + i]], o);
          front_step(step, o);
        }
        if (o.rows > 0) o.np = xint(o.X)[kINp];
        return (long long)o.rows;
      });
      RowsSm& sm = *reinterpret_cast<RowsSm*>(dsm);
      for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        const int fi = item_front(P, n, t);
        phase_a_item(s, s.big + list[c0 + fi], info[fi], (int)(t - P.ptr[fi]), sm);
      }
      __syncthreads();
    }
    grid.sync();
    // ---- U (mixed precision): trailing-update tiles of the fronts that
    // accepted pivots, after the commit
    for (int c0 = 0; c0 < nl; c0 += kChunkFronts) {
      const int n = min(kChunkFronts, nl - c0);
      const long long total = front_prefix(P, n, [&](int i) {
        const BigFront& B = s.big[list[c0 + i]];
        return (active(s, B, step) && B.kw > 0) ? tri_tiles(B, umma::kTileM) : 0ll;
      });
      UpdSm& sm = *reinterpret_cast<UpdSm*>(dsm);
      for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        const int fi = item_front(P, n, t);
        const BigFront& B = s.big[list[c0 + fi]];
        int I, J;
        tri_decode(t - P.ptr[fi], (B.f - B.k + umma::kTileM - 1) / umma::kTileM, I, J);
        if (!tc_fail) {
          // the tensor-core operands share the dynamic shared memory with
          // the FP64 tiles' panels (a tile uses one or the other)
          float* ops = reinterpret_cast<float*>(dsm + kOpsOffset);
          tc_fail = phase_u_tile_mixed(s, B, I, J, sm, ops, &mbar, &phase, tmem);
        }
      }
      __syncthreads();
    }
    grid.sync();
  }
  // the step cap (never reached when every step makes progress)
  if (step > max_steps && blockIdx.x == 0 && tid == 0) counters[2] = 1;
  // every CTA has left the loop: the roots set aside take part in the
  // chained panels that follow
  if (blockIdx.x == 0) {
    const int nd = *((volatile int*)(meta + 19));
    for (int i = tid; i < nd; i += kThreads) s.big[done[i]].state = 0;
  }
  if (prm.mixed) {
    if (tc_fail) {
      // a tensor-core operation did not complete in time: the factorization
      // is reported failed; wait once more (bounded) before freeing TMEM
      if (tid == 0) counters[2] = 2;
      umma::mbar_wait(&mbar, phase ^ 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::);
    __syncthreads();
    if (warp == 0) umma::tmem_free_128(tmem);
  }
}

}  // namespace

cudaError_t launch_app_level(const DevState& s, const FactorParams& prm, int count, int max_fs,
                             const int* list, int* done, int* meta, cudaStream_t stream) {
  static_assert(kBlk == kBigPanelMax, "panel width");
  if (count <= 0) return cudaSuccess;
  int dev = 0, nsm = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, app_level_kernel, kThreads, kDynSmem);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorLaunchOutOfResources;
  const int grid = nsm * per;
  // every step of an active front accepts a pivot or delays a candidate
  int max_steps = max_fs + 8;
  DevState sa = s;
  FactorParams pa = prm;
  const int* la = list;
  int na = count;
  int* da = done;
  int* ma = meta;
  void* args[] = {(void*)&sa, (void*)&pa,        (void*)&la, (void*)&na,
                  (void*)&max_steps, (void*)&da, (void*)&ma};
  return cudaLaunchCooperativeKernel((const void*)app_level_kernel, dim3(grid), dim3(kThreads),
                                     args, kDynSmem, stream);
}

cudaError_t configure_app_kernels() {
  return cudaFuncSetAttribute(app_level_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kDynSmem);
}

}  // namespace b200ldl
