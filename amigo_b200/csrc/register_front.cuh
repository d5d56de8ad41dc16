// The fronts of one CTA, factored in registers.
#pragma once

#include <climits>

#include "ldl_internal.h"

namespace b200ldl {

namespace {

constexpr int kWarps = kFactorThreads / 32;

enum : int { kDelay = 0, kOne = 1, kTwo = 2, kNeedRow = 3, kZero = 4 };

constexpr double kAlphaBK = (1.0 + 4.1231056256176605) / 8.0;  // (1 + sqrt(17)) / 8

// largest non-NaN value of the lanes' non-negative v with the lowest index
// holding it, over the lanes that have one (i < INT_MAX); -1 and INT_MAX if
// none has. Non-negative doubles order as their bits, so the reductions are
// exact integer ones; +1 keeps a held 0.0 above the lanes without a value.
__device__ __forceinline__ void warp_argmax(double& v, int& i) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = i != INT_MAX ? (unsigned)(u >> 32) + 1u : 0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)u : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  i = __reduce_min_sync(0xffffffffu, (hi == mh && (unsigned)u == ml) ? i : INT_MAX);
  v = mh ? __longlong_as_double((long long)(((unsigned long long)(mh - 1u) << 32) | ml)) : -1.0;
}

// largest of the lanes' non-negative, non-NaN values
__device__ __forceinline__ double warp_max(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)u : 0u);
  return __longlong_as_double((long long)(((unsigned long long)mh << 32) | ml));
}

// The CTA's two column barriers (used in turn), split into halves: the warp
// that has published a column arrives and goes on, the others wait for it. A
// warp executes either as one, so its lanes come together first. (Compiled for
// the host, to run the CTA's threads under chosen schedules, the includer
// brings its own.)
#ifdef __CUDACC__
__device__ __forceinline__ void bar_arrive(int odd) {
  __syncwarp();
  if (odd)
    asm volatile("bar.arrive 2, %0;" ::"n"(kFactorThreads) : "memory");
  else
    asm volatile("bar.arrive 1, %0;" ::"n"(kFactorThreads) : "memory");
}
__device__ __forceinline__ void bar_wait(int odd) {
  __syncwarp();
  if (odd)
    asm volatile("bar.sync 2, %0;" ::"n"(kFactorThreads) : "memory");
  else
    asm volatile("bar.sync 1, %0;" ::"n"(kFactorThreads) : "memory");
}
#endif

// a b + c d with its roundings fixed. The products of the 2x2 pivots are formed
// in several places and by two algorithms, which have to give the same bits.
__device__ __forceinline__ double two_products(double a, double b, double c, double d) {
  return fma(a, b, __dmul_rn(c, d));
}

// The front of one CTA: assembled in shared memory, factored in registers.
struct Front {
  double* F;     // [f][ld], column-major lower triangle, then the factor columns
  double* vec;   // [kVecs][vec_len(f)] columns that travel between the warps
  int* fv;       // [f] front variables in the current order
  int* orig;     // [f] their positions at assembly
  int f, fs, ld;
};

struct Result {
  int npiv, npos, nneg;
  long long flops;
};

// row chunks of 32 that a front of f rows is factored with
__host__ __device__ __forceinline__ int row_chunks(int f) {
  return f <= 32 ? 1 : f <= 64 ? 2 : f <= 96 ? 3 : 5;
}

// A travelling column: entry i at [i] for the rows below its diagonal, zeros
// for the others from its chunk on (so that no reader has to compare rows),
// and the diagonal entry after the last chunk.
__host__ __device__ __forceinline__ int vec_len(int f) { return 32 * row_chunks(f) + 2; }

constexpr int kVecs = 6;  // of them

// Where the pivot chain stands, the same in every warp.
struct Chain {
  int k, ncand;
  double *cur, *nx1, *nx2;  // the column at k, the next, the one after
  bool forced;  // the candidate at k is accepted as it stands
  bool moved;   // the column at k stands in cur alone (after a delay)
  int phase;    // which column barrier is next
  double thr, tol;  // a 1x1 passes with |d| >= tol and |d| >= thr max|column|
  bool any;         // every 1x1 passes (Cholesky mode)
  bool root;
  Result out;
};

// Column j, whose rows this warp holds in col (chunks from c0 = j / 32 on),
// as a travelling column.
template <int kR>
__device__ __forceinline__ void put_column(const double (&col)[kR], int c0, int j, double* dst) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < kR; c++) {
    if (c < c0) continue;
    const int i = lane + 32 * c;
    dst[i] = (c > c0 || i > j) ? col[c] : 0.0;
    if (c == c0 && i == j) dst[32 * kR] = col[c];
  }
}

// 1x1 pivots of the positions [8 g, 8 g + 8) from k on, up to the first that
// does not pass as it stands; the slots before g are finished. Columns before
// k and beyond the front take part in the updates with whatever they hold:
// nothing reads them again, and the code stays free of branches.
template <int kR, int kS, int g>
__device__ __forceinline__ void stage(double (&v)[kS][kR], Chain& h, const Front& a) {
  constexpr int c0 = g / 4;
  constexpr int kD = 32 * kR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ld = a.ld;
  double* L = a.F;
  while (true) {
    const int k = h.k;
    const double* cur = h.cur;
    double w[kR];
    int m = 0;
#pragma unroll
    for (int c = c0; c < kR; c++) {
      w[c] = cur[lane + 32 * c];
      m = max(m, __double2hiint(w[c]) & 0x7fffffff);
    }
    const double d = cur[kD];
    const double absd = fabs(d);
    const double r = (h.root && d == 0.0) ? 0.0 : 1.0 / d;
    if (!h.forced && !h.any) {
      // a bound of the lane's largest entry from its high word: a pivot that
      // passes against it passes (the rounded product is monotone), the full
      // tests decide the others (and whatever is not finite)
      const bool ok = absd >= h.tol && absd > 0.0 && absd >= h.thr * __hiloint2double(m + 1, 0);
      if (!__all_sync(0xffffffffu, ok)) return;
    }
    h.forced = false;
    h.moved = false;
    const int nxt = k + 1;
    const bool more = nxt < h.ncand;
    const bool own = more && warp == nxt % kWarps;
    const bool late = nxt % kWarps == 0;  // the next column is the stage after's
    // the next column first, by its warp; then this warp's other columns
    double l[kS];
#pragma unroll
    for (int s = g; s < kS; s++) l[s] = cur[warp + kWarps * s] * r;
    if (own) {
      if (!late) {
#pragma unroll
        for (int c = c0; c < kR; c++) v[g][c] = fma(-w[c], l[g], v[g][c]);
        put_column<kR>(v[g], c0, nxt, h.nx1);
      } else if constexpr (g + 1 < kS) {
        constexpr int c1 = (g + 1) / 4;
#pragma unroll
        for (int c = c1; c < kR; c++) v[g + 1][c] = fma(-w[c], l[g + 1], v[g + 1][c]);
        put_column<kR>(v[g + 1], c1, nxt, h.nx1);
      }
      bar_arrive(h.phase);
    }
    if (!(own && !late)) {
#pragma unroll
      for (int c = c0; c < kR; c++) v[g][c] = fma(-w[c], l[g], v[g][c]);
    }
    if constexpr (g + 1 < kS) {
      if (!(own && late)) {
#pragma unroll
        for (int c = (g + 1) / 4; c < kR; c++) v[g + 1][c] = fma(-w[c], l[g + 1], v[g + 1][c]);
      }
    }
#pragma unroll
    for (int s = g + 2; s < kS; s++)
#pragma unroll
      for (int c = s / 4; c < kR; c++) v[s][c] = fma(-w[c], l[s], v[s][c]);
    if (warp == k % kWarps) {
      double* Lk = L + ld * k;
#pragma unroll
      for (int c = c0; c < kR; c++) {
        const int i = lane + 32 * c;
        if (i > k && i < a.f) Lk[i] = w[c] * r;
      }
      if (lane == 0) Lk[k] = d;
    }
    h.k = nxt;
    if (!more) return;
    if (own)
      __syncwarp();
    else
      bar_wait(h.phase);
    h.phase ^= 1;
    double* t = h.cur;
    h.cur = h.nx1;
    h.nx1 = h.nx2;
    h.nx2 = t;
    if (late) return;
  }
}

// the stage that position k is in
template <int kR, int kS, int g>
__device__ __forceinline__ void run_stage(double (&v)[kS][kR], Chain& h, const Front& a) {
  if constexpr (g + 1 < kS) {
    if (h.k >= kWarps * (g + 1)) {
      run_stage<kR, kS, g + 1>(v, h, a);
      return;
    }
  }
  stage<kR, kS, g>(v, h, a);
}

// Partial factorization of the candidates [0, fs), the front in registers:
// column j belongs to warp j % 8, slot j / 8; lane l holds rows l, l + 32, ..
// (kR chunks of 32, f <= 32 kR). It is the reference's algorithm one
// candidate at a time and right-looking, and each entry receives one fused
// multiply-add per 1x1 pivot (a two-term product per 2x2), in pivot order.
//
// What bounds it is the chain from one pivot column to the next, so the
// chain is kept short: the current column stands in shared memory; every
// warp reads it, votes on the common case (a 1x1 that passes where it
// stands: no reduction, the rounded product thr * max is monotone) and forms
// the reciprocal itself, so that no decision has to travel; the warp that
// owns the next column updates that column first and publishes it, and
// arrives at the barrier before it goes on to its other columns. One barrier
// and one shared-memory round trip per pivot: 0.4 us a pivot for a 68-row
// front (740 cycles with the code in the instruction cache), against about
// 2,800 cycles for the same algorithm in shared memory with a reduction and a
// barrier per pivot. Optimal control N = 1000, 167 such fronts one after
// another: 17.0 ms with that one and a launch per level, 6.9 ms now (41 us a
// front, of which the pivots are 26: the rest is the way from one front to
// the next). 512 systems of 50..400 nodes with 6 states: 13.3 and 7.3 ms. The
// other cases (statistics, imax column, delays, interchanges, 2x2) are also
// decided by every warp from the same values; an interchange moves two rows
// and columns between the registers through the published columns.
//
// `write` is called with the number of pivots and then the trailing columns
// (every lane's rows of its warp's columns) are handed to `store`.
template <int kR, typename Write, typename Store>
__device__ __forceinline__ Result factor_front(const Front& a, bool root, const FactorParams& prm,
                                               Write write, Store store) {
  constexpr int kD = 32 * kR;  // where a travelling column has its diagonal entry
  constexpr int kLen = kD + 2;
  constexpr int kS = 32 * kR < kSmemFrontMax ? 4 * kR : (kSmemFrontMax + kWarps - 1) / kWarps;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = a.f, ld = a.ld;
  double* L = a.F;  // once the front is in registers
  double v[kS][kR];  // chunks above the diagonal (c < s / 4) are never touched
#pragma unroll
  for (int s = 0; s < kS; s++) {
    const int j = warp + kWarps * s;
#pragma unroll
    for (int c = s / 4; c < kR; c++) {
      const int i = lane + 32 * c;
      v[s][c] = (j < f && i >= j && i < f) ? a.F[i + ld * j] : 0.0;
    }
  }
  // the current column, the next one, the one after (a warp may still read
  // the current one when the next but one is published), two for the imax
  // column and the interchanges, and the next candidate's imax column
  Chain h;
  h.cur = a.vec;
  h.nx1 = h.cur + kLen;
  h.nx2 = h.nx1 + kLen;
  double* V = h.nx2 + kLen;
  double* U = V + kLen;
  double* spare = U + kLen;
  h.k = 0;
  h.ncand = a.fs;
  h.forced = h.moved = false;
  h.phase = 0;
  h.thr = root ? kAlphaBK : prm.ustab;
  h.tol = root ? 0.0 : prm.pivot_tol;
  h.any = prm.cholesky != 0;
  h.root = root;
  h.out = {0, 0, 0, 0};
  double*& cur = h.cur;
  int& k = h.k;
  int& ncand = h.ncand;
  Result& out = h.out;

  // this warp's column j
  auto publish = [&](int j, double* dst) {
#pragma unroll
    for (int s = 0; s < kS; s++)
      if (warp + kWarps * s == j) put_column<kR>(v[s], s / 4, j, dst);
  };
  // Row and column b of the trailing matrix (positions from k on, k < b) as
  // column k would hold them after k and b change places: dst[b] the entry
  // (b, k), dst[r] the entry {b, r}. All warps; the caller synchronizes.
  auto form = [&](int k, int b, double* dst) {
#pragma unroll
    for (int c = 0; c < kR; c++) {
      const int bl = b - 32 * c;  // the lane of row b, if it is in this chunk
      if (bl < 0 || bl >= 32) continue;
#pragma unroll
      for (int s = 0; s < kS && s / 4 <= c; s++) {
        const int j = warp + kWarps * s;
        if (j > k && j < b && lane == bl) dst[j] = v[s][c];
      }
    }
    if (warp == b % kWarps) {
#pragma unroll
      for (int s = 0; s < kS; s++) {
        if (warp + kWarps * s != b) continue;
#pragma unroll
        for (int c = s / 4; c < kR; c++) {
          const int i = lane + 32 * c;
          if (i > b) dst[i] = v[s][c];
          if (i == b) dst[kD] = v[s][c];
        }
      }
      if (lane == 0) dst[b] = cur[b];
      if (lane <= k % 32) dst[k - k % 32 + lane] = 0.0;
    }
  };
  // Row and column b take the entries of the column src that stood at k
  auto replace = [&](int k, int b, const double* src) {
#pragma unroll
    for (int c = 0; c < kR; c++) {
      const int bl = b - 32 * c;
      if (bl < 0 || bl >= 32) continue;
#pragma unroll
      for (int s = 0; s < kS && s / 4 <= c; s++) {
        const int j = warp + kWarps * s;
        if (j > k && j < b && lane == bl) v[s][c] = src[j];
      }
    }
    if (warp == b % kWarps) {
#pragma unroll
      for (int s = 0; s < kS; s++) {
        if (warp + kWarps * s != b) continue;
#pragma unroll
        for (int c = s / 4; c < kR; c++) {
          const int i = lane + 32 * c;
          if (i >= b) v[s][c] = src[i == b ? kD : i];
        }
      }
    }
  };
  // rows x < y of the factor columns [0, k) and the variables change places
  auto swap_rows = [&](int k, int x, int y) {
    for (int t = tid; t < k; t += kFactorThreads) {
      const double p = L[x + ld * t], q = L[y + ld * t];
      L[x + ld * t] = q;
      L[y + ld * t] = p;
    }
    if (tid == 0) {
      int t = a.fv[x];
      a.fv[x] = a.fv[y];
      a.fv[y] = t;
      t = a.orig[x];
      a.orig[x] = a.orig[y];
      a.orig[y] = t;
    }
  };

  // the column at k is published and becomes the current one
  auto next_column = [&]() {
    if (k < ncand && warp == k % kWarps) publish(k, h.nx1);
    double* t = h.cur;
    h.cur = h.nx1;
    h.nx1 = h.nx2;
    h.nx2 = t;
    __syncthreads();
  };

  if (k < ncand && warp == 0) publish(0, cur);
  __syncthreads();
  while (k < ncand) {
    const int k0 = k;
    run_stage<kR, kS, 0>(v, h, a);
    if (k >= ncand || (k > k0 && k % kWarps == 0)) continue;
    // the candidate at k did not pass: the reference's tests in full
    const double d = cur[kD];
    const double absd = fabs(d);
    double bv = 0.0, cm = 0.0;
    int bi = INT_MAX;
#pragma unroll
    for (int c = 0; c < kR; c++) {
      const int i = lane + 32 * c;
      const double x = (i > k && i < f) ? fabs(cur[i]) : 0.0;
      if (i > k && i < f && x == x) {
        if (i >= ncand) {
          cm = fmax(cm, x);
        } else if (bi == INT_MAX || x > bv) {
          bv = x;
          bi = i;
        }
      }
    }
    __syncwarp();
    warp_argmax(bv, bi);
    cm = warp_max(cm);
    const bool has_cand = k + 1 < ncand;
    const double abswik = has_cand ? bv : 0.0;
    // bi stays INT_MAX only if every candidate entry is NaN; keep imax a
    // valid candidate index so the rest of the step stays in bounds
    const int imax = has_cand ? (bi < ncand ? bi : k + 1) : k;
    const double colmax = fmax(abswik, cm);
    int step, kpiv = k;
    if (root) {
      if (fmax(absd, colmax) == 0.0)
        step = kZero;
      else if (absd >= kAlphaBK * colmax)
        step = kOne;
      else
        step = kNeedRow;
    } else if (absd >= prm.pivot_tol && absd >= prm.ustab * colmax) {
      step = kOne;
    } else {
      step = has_cand ? kNeedRow : kDelay;
    }
    const bool formed = step == kNeedRow && has_cand;
    if (formed) {
      form(k, imax, V);
      __syncthreads();
      double rmax = 0.0;
#pragma unroll
      for (int c = 0; c < kR; c++) {
        const int i = lane + 32 * c;
        const double x = (i > k && i < f) ? fabs(V[i]) : 0.0;
        if (x == x) rmax = fmax(rmax, x);
      }
      __syncwarp();
      rmax = warp_max(rmax);
      const double wii = V[kD];
      const double abswii = fabs(wii);
      const double wik = cur[imax];
      if (root) {
        // Bunch-Kaufman partial pivoting (dsytf2, lower)
        if (absd >= kAlphaBK * colmax * (colmax / rmax)) {
          step = kOne;
        } else if (abswii >= kAlphaBK * rmax) {
          step = kOne;
          kpiv = imax;
        } else {
          step = kTwo;
          kpiv = imax;
        }
      } else if (abswii >= prm.pivot_tol && abswii >= prm.ustab * rmax) {
        step = kOne;
        kpiv = imax;
      } else {
        const double det = fabs(two_products(d, wii, -wik, wik));
        step = kDelay;
        if (det >= prm.pivot_tol) {
          const double delta = det / fmax(abswii + abswik, absd + abswik);
          if (delta >= prm.ustab * colmax && delta >= prm.ustab * rmax) {
            step = kTwo;
            kpiv = imax;
          }
        }
      }
    }
    if (step == kDelay) {
      ncand--;
      if (k < ncand) {
        if (imax == ncand) {  // its column is in V already
          double* t = U;
          U = V;
          V = t;
        } else {
          form(k, ncand, U);
          __syncthreads();
        }
        replace(k, ncand, cur);
        swap_rows(k, k, ncand);
        double* t = cur;
        cur = U;
        U = t;
        h.moved = true;
        __syncthreads();  // both may be formed again at once
      }
      continue;
    }
    if (step == kZero && d != 0.0) {
      // a zero pivot of a root whose diagonal is not a number, so that the
      // reciprocal of stage() would not be zero: its column is zero, or not a
      // number, which the products with zero keep
      h.moved = false;
      double w0[kR];
#pragma unroll
      for (int c = 0; c < kR; c++) {
        const int i = lane + 32 * c;
        w0[c] = (i > k && i < f) ? cur[i] : 0.0;
        if (warp == k % kWarps && i > k && i < f) L[i + ld * k] = w0[c] * 0.0;
      }
      if (warp == k % kWarps && lane == 0) L[k + ld * k] = d;
#pragma unroll
      for (int s = 0; s < kS; s++) {
        const int j = warp + kWarps * s;
        const double x = (j > k && j < f) ? cur[j] * 0.0 : 0.0;
#pragma unroll
        for (int c = s / 4; c < kR; c++) v[s][c] = fma(-w0[c], x, v[s][c]);
      }
      k++;
      next_column();
      continue;
    }
    if (step != kTwo) {
      if (kpiv != k) {
        replace(k, kpiv, cur);
        swap_rows(k, k, kpiv);
        double* t = cur;
        cur = V;
        V = t;
      }
      // In the stage the next column's warp only arrives at the barrier. If
      // its column does not pass either it goes on to form another row while
      // other warps may still read V (the old current column, after an
      // interchange): that row goes into the spare, and the barrier after it
      // is what lets V be formed in again.
      if (formed) {
        double* t = V;
        V = spare;
        spare = t;
      }
      h.forced = true;
      continue;
    }
    // a 2x2 pivot: columns k and k + 1, with imax at k + 1
    h.moved = false;
    const int q = kpiv;
    if (q != k + 1) {
      if (warp == (k + 1) % kWarps) publish(k + 1, U);
      __syncthreads();
      replace(k + 1, q, U);
      swap_rows(k, k + 1, q);
    }
    const double d11 = d;
    const double d21 = cur[q];
    const double d22 = V[kD];
    const double det = two_products(d11, d22, -d21, d21);
    const double detinv = 1.0 / det;
    const double i00 = d22 * detinv, i01 = -d21 * detinv, i11 = d11 * detinv;
    // the two columns' entries in row i (row q holds what stood at k + 1) and
    // their L entries, with the products' order fixed: L is formed in several
    // places and has to come out the same
    auto at0 = [&](int i) { return cur[i == q ? k + 1 : i]; };
    auto at1 = [&](int i) { return V[i == q ? k + 1 : i]; };
    auto l0 = [&](double x, double y) { return two_products(x, i00, y, i01); };
    auto l1 = [&](double x, double y) { return two_products(x, i01, y, i11); };
    double w0[kR], w1[kR];
#pragma unroll
    for (int c = 0; c < kR; c++) {
      const int i = lane + 32 * c;
      const bool on = i > k + 1 && i < f;
      w0[c] = on ? at0(i) : 0.0;
      w1[c] = on ? at1(i) : 0.0;
    }
    if (warp == k % kWarps) {
#pragma unroll
      for (int c = 0; c < kR; c++) {
        const int i = lane + 32 * c;
        if (i > k + 1 && i < f) {
          L[i + ld * k] = l0(w0[c], w1[c]);
          L[i + ld * (k + 1)] = l1(w0[c], w1[c]);
        }
      }
      if (lane == 0) {
        L[k + ld * k] = d11;
        L[k + 1 + ld * k] = d21;
        L[k + 1 + ld * (k + 1)] = d22;
      }
    }
#pragma unroll
    for (int s = 0; s < kS; s++) {
      const int j = warp + kWarps * s;
      const bool on = j > k + 1 && j < f;
      const double x = on ? at0(j) : 0.0, y = on ? at1(j) : 0.0;
      const double a0 = l0(x, y), a1 = l1(x, y);
#pragma unroll
      for (int c = s / 4; c < kR; c++) v[s][c] -= two_products(w0[c], a0, w1[c], a1);
    }
    if (tid == 0) {
      a.fv[k] = -(a.fv[k] + 1);
      a.fv[k + 1] = -(a.fv[k + 1] + 1);
    }
    if (det >= 0.0) {
      if (d11 >= 0.0)
        out.npos += 2;
      else
        out.nneg += 2;
    } else {
      out.npos++;
      out.nneg++;
    }
    const int r = f - k - 2;
    out.flops += 2 * r * (r + 1) + 6 * r;
    k += 2;
    next_column();
  }
  // a delayed candidate that was moved to k and stayed there
  if (h.moved && warp == k % kWarps) {
#pragma unroll
    for (int s = 0; s < kS; s++) {
      if (warp + kWarps * s != k) continue;
#pragma unroll
      for (int c = s / 4; c < kR; c++) {
        const int i = lane + 32 * c;
        if (i >= k) v[s][c] = cur[i == k ? kD : i];
      }
    }
  }
  out.npiv = k;
  write(out);
  if (warp == 0) {
    // the 1x1 pivots' signs and work (the 2x2 ones are counted above)
    int pos = 0, neg = 0, fl = 0;
    for (int t = lane; t < k; t += 32) {
      if (a.fv[t] < 0) continue;
      if (L[t + ld * t] >= 0.0)
        pos++;
      else
        neg++;
      fl += (f - t - 1) * (f - t + 1);
    }
    out.npos += __reduce_add_sync(0xffffffffu, pos);
    out.nneg += __reduce_add_sync(0xffffffffu, neg);
    out.flops += __reduce_add_sync(0xffffffffu, fl);
  }
#pragma unroll
  for (int s = 0; s < kS; s++) {
    const int j = warp + kWarps * s;
    if (j < k || j >= f) continue;
#pragma unroll
    for (int c = s / 4; c < kR; c++) {
      const int i = lane + 32 * c;
      if (i >= j && i < f) store(i, j, v[s][c]);
    }
  }
  return out;
}

}  // namespace

}  // namespace b200ldl
