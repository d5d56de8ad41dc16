// Numeric multifrontal LDL^T on sm_100a: one CTA per supernode of an
// elimination-tree level. The CTA assembles its front (CSR entries of its
// pivot columns, the diagonal vector, the children's contribution blocks),
// factors the fully summed part with threshold 1x1/2x2 pivoting (delaying
// candidates that fail, as the reference does in
// SparseLDL::factor_front_matrix_block, include/sparse_ldl.h:1316-1553) or
// with Bunch-Kaufman when the front has no contribution rows (the reference
// calls LAPACK dsytrf there, include/sparse_ldl.h:1226-1248), and writes the
// factor columns, its final front-variable order and its contribution block.
//
// Fronts up to kSmemFrontMax are assembled in shared memory and factored in
// registers (factor_front); larger ones are registered for the big-front
// kernels.
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
// warp executes either as one, so its lanes come together first.
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

// The front of one CTA: assembled in shared memory, factored in registers.
struct Front {
  double* F;     // [f][ld], column-major lower triangle, then the factor columns
  double* vec;   // [5][vec_len(f)] columns that travel between the warps
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
// and one shared-memory round trip per pivot: about 740 cycles a pivot for a
// 68-row front with the code in the instruction cache, against about 2,800
// for the same algorithm in shared memory with a reduction and a barrier per
// pivot (optimal control N = 1000, 167 such fronts one after another: 17.0 ms
// before, 7.2 ms now, launches included; 512 systems of 50..400 nodes: 13.3
// and 7.5 ms). The other cases (statistics,
// imax column, delays, interchanges, 2x2) are also decided by every warp from
// the same values; an interchange moves two rows and columns between the
// registers through the published columns.
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
  // the current one when the next but one is published), and two for the
  // imax column and the interchanges
  Chain h;
  h.cur = a.vec;
  h.nx1 = h.cur + kLen;
  h.nx2 = h.nx1 + kLen;
  double* V = h.nx2 + kLen;
  double* U = V + kLen;
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
    if (step == kNeedRow && has_cand) {
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
        const double det = fabs(fma(d, wii, -__dmul_rn(wik, wik)));
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
    if (step != kTwo) {
      if (kpiv != k) {
        replace(k, kpiv, cur);
        swap_rows(k, k, kpiv);
        double* t = cur;
        cur = V;
        V = t;
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
    const double det = fma(d11, d22, -__dmul_rn(d21, d21));
    const double detinv = 1.0 / det;
    const double i00 = d22 * detinv, i01 = -d21 * detinv, i11 = d11 * detinv;
    // the two columns' entries in row i (row q holds what stood at k + 1) and
    // their L entries, with the products' order fixed: L is formed in several
    // places and has to come out the same
    auto at0 = [&](int i) { return cur[i == q ? k + 1 : i]; };
    auto at1 = [&](int i) { return V[i == q ? k + 1 : i]; };
    auto l0 = [&](double x, double y) { return fma(x, i00, __dmul_rn(y, i01)); };
    auto l1 = [&](double x, double y) { return fma(x, i01, __dmul_rn(y, i11)); };
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
      for (int c = s / 4; c < kR; c++) v[s][c] -= fma(w0[c], a0, __dmul_rn(w1[c], a1));
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
    if (k < ncand && warp == k % kWarps) publish(k, h.nx1);
    double* t = h.cur;
    h.cur = h.nx1;
    h.nx1 = h.nx2;
    h.nx2 = t;
    __syncthreads();
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

__device__ __forceinline__ void keep_larger(double& bv, int& bi, double v, int i) {
  // larger magnitude wins; ties go to the lower index (idamax semantics)
  if (v > bv || (v == bv && i < bi)) {
    bv = v;
    bi = i;
  }
}

// Warp-wide (argmax, max) with the result in every lane.
__device__ __forceinline__ void warp_argmax_max(double& bv, int& bi, double& cm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    const double om = __shfl_xor_sync(0xffffffffu, cm, o);
    keep_larger(bv, bi, ov, oi);
    cm = fmax(cm, om);
  }
}

struct Reduce {
  double v[kWarps];
  int i[kWarps];
  double m[kWarps];
};

// Block-wide (argmax, max) reduction. Result valid for all threads after the
// trailing barrier.
__device__ __forceinline__ void block_argmax(Reduce& r, double& bv, int& bi, double& cm) {
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_down_sync(0xffffffffu, bv, o);
    const int oi = __shfl_down_sync(0xffffffffu, bi, o);
    const double om = __shfl_down_sync(0xffffffffu, cm, o);
    keep_larger(bv, bi, ov, oi);
    cm = fmax(cm, om);
  }
  if (lane == 0) {
    r.v[w] = bv;
    r.i[w] = bi;
    r.m[w] = cm;
  }
  __syncthreads();
  bv = r.v[0];
  bi = r.i[0];
  cm = r.m[0];
#pragma unroll
  for (int q = 1; q < kWarps; q++) {
    keep_larger(bv, bi, r.v[q], r.i[q]);
    cm = fmax(cm, r.m[q]);
  }
  __syncthreads();
}

// Symmetric interchange of rows/columns a < b of the lower-stored front,
// including the already factored columns left of a (sparse_ldl.h:1270-1292).
__device__ void symm_swap(double* F, int ld, int f, int a, int b, int* fv, int* orig) {
  const int n1 = a;              // F(a, 0:a) <-> F(b, 0:a)
  const int n2 = b - a - 1;      // F(j, a) <-> F(b, j), a < j < b
  const int n3 = f - b - 1;      // F(j, a) <-> F(j, b), j > b
  const int total = n1 + 1 + n2 + n3;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    double *p, *q;
    if (t < n1) {
      p = &F[a + (size_t)ld * t];
      q = &F[b + (size_t)ld * t];
    } else if (t == n1) {
      p = &F[a + (size_t)ld * a];
      q = &F[b + (size_t)ld * b];
    } else if (t < n1 + 1 + n2) {
      const int j = a + 1 + (t - n1 - 1);
      p = &F[j + (size_t)ld * a];
      q = &F[b + (size_t)ld * j];
    } else {
      const int j = b + 1 + (t - n1 - 1 - n2);
      p = &F[j + (size_t)ld * a];
      q = &F[j + (size_t)ld * b];
    }
    const double tmp = *p;
    *p = *q;
    *q = tmp;
  }
  if (threadIdx.x == 0) {
    int t = fv[a];
    fv[a] = fv[b];
    fv[b] = t;
    t = orig[a];
    orig[a] = orig[b];
    orig[b] = t;
  }
}

// The same factorization in shared memory, for the fronts of more than 96
// rows of a structure that still delays candidates through its fronts (dozens
// per front): a delay moves its two rows and columns in shared memory in one
// pass of the CTA, while the register front above forms and replaces them
// slot by slot, several thousand cycles a delay at 18 slots of 5 chunks
// (64 x 64 plane stress, first factorization: 95.6 ms with this one, 97.2
// with registers throughout).
template <typename Write, typename Store>
__device__ __forceinline__ Result general_front(const Front& a, bool root, const FactorParams& prm,
                                               Write write, Store store) {
  __shared__ Reduce red;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = a.f, ld = a.ld, fs = a.fs;
  double* F = a.F;
  int* fv = a.fv;
  int* orig = a.orig;
  // partial factorization of the fully summed candidates [0, ncand).
  // Right-looking, one barrier per accepted 1x1 pivot: the warp that updates
  // the next column also produces its pivot statistics, and the scaling of
  // a pivot column into L is deferred to the next update pass (it is a
  // per-row operation, so it commutes with the row interchanges in between).
  __shared__ double st_v, st_m;
  __shared__ int st_i;
  int k = 0;
  int ncand = fs;
  int npos = 0, nneg = 0;
  double flops = 0.0;
  int pend = 0, pc = 0;
  double pd0 = 0.0, pd1 = 0.0, pd2 = 0.0;
  bool need_stats = true;

  while (k < ncand) {
    if (!prm.cholesky && need_stats) {
      if (warp == 0) {
        double bv = -1.0, cm = 0.0;
        int bi = INT_MAX;
        const double* colk = F + (size_t)ld * k;
        for (int i = k + 1 + lane; i < f; i += 32) {
          const double a = fabs(colk[i]);
          if (i < ncand)
            keep_larger(bv, bi, a, i);
          else
            cm = fmax(cm, a);
        }
        warp_argmax_max(bv, bi, cm);
        if (lane == 0) {
          st_v = bv;
          st_i = bi;
          st_m = cm;
        }
      }
      __syncthreads();
    }
    int step;
    int kpiv = k;
    if (prm.cholesky) {
      step = kOne;
    } else {
      const double wkk = F[k + (size_t)ld * k];
      const double abswkk = fabs(wkk);
      const bool has_cand = (k + 1 < ncand);
      const double abswik = has_cand ? st_v : 0.0;
      // st_i stays INT_MAX only if every candidate entry is NaN; keep imax a
      // valid candidate index so the rest of the step stays in bounds
      const int imax = has_cand ? (st_i < ncand ? st_i : k + 1) : k;
      const double colmax = fmax(abswik, st_m);
      if (root) {
        if (fmax(abswkk, colmax) == 0.0)
          step = kZero;
        else if (abswkk >= kAlphaBK * colmax)
          step = kOne;
        else
          step = kNeedRow;
      } else if (abswkk >= prm.pivot_tol && abswkk >= prm.ustab * colmax) {
        step = kOne;
      } else {
        step = has_cand ? kNeedRow : kDelay;
      }
      if (step == kNeedRow) {
        // row/column imax off the diagonal: F(imax, k:imax), F(imax+1:, imax)
        double rv = -1.0, rmax = 0.0;
        int ri = INT_MAX;
        const int n1 = imax - k;
        const int n2 = f - imax - 1;
        for (int t = tid; t < n1 + n2; t += blockDim.x) {
          const double a = (t < n1) ? fabs(F[imax + (size_t)ld * (k + t)])
                                    : fabs(F[(imax + 1 + (t - n1)) + (size_t)ld * imax]);
          rmax = fmax(rmax, a);
        }
        block_argmax(red, rv, ri, rmax);
        const double wii = F[imax + (size_t)ld * imax];
        const double abswii = fabs(wii);
        const double wik = F[imax + (size_t)ld * k];
        if (root) {
          // Bunch-Kaufman partial pivoting (dsytf2, lower)
          if (abswkk >= kAlphaBK * colmax * (colmax / rmax)) {
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
          const double det = fabs(wkk * wii - wik * wik);
          step = kDelay;
          if (det >= prm.pivot_tol) {
            const double delta = det / fmax(abswii + abswik, abswkk + abswik);
            if (delta >= prm.ustab * colmax && delta >= prm.ustab * rmax) {
              step = kTwo;
              kpiv = imax;
            }
          }
        }
      }
    }

    if (step == kDelay) {
      if (k < ncand - 1) symm_swap(F, ld, f, k, ncand - 1, fv, orig);
      __syncthreads();
      ncand -= 1;
      need_stats = true;
      continue;
    }
    const int nstep = (step == kTwo) ? 2 : 1;
    const int ksrc = k + nstep - 1;
    if (kpiv != ksrc) {
      symm_swap(F, ld, f, ksrc, kpiv, fv, orig);
      __syncthreads();
    }

    // deferred scaling of the previous pivot column(s)
    if (pend == 1) {
      double* c0 = F + (size_t)ld * pc;
      for (int i = pc + 1 + tid; i < f; i += blockDim.x) c0[i] *= pd0;
    } else if (pend == 2) {
      double* c0 = F + (size_t)ld * pc;
      double* c1 = c0 + ld;
      for (int i = pc + 2 + tid; i < f; i += blockDim.x) {
        const double a = c0[i];
        const double b = c1[i];
        c0[i] = a * pd0 + b * pd1;
        c1[i] = a * pd1 + b * pd2;
      }
    }

    const double* colk = F + (size_t)ld * k;
    const int nxt = k + nstep;  // the next candidate column
    const bool want_stats = !prm.cholesky && nxt < ncand;
    if (nstep == 1) {
      const double d = colk[k];
      const double dinv = (step == kZero || (root && d == 0.0)) ? 0.0 : 1.0 / d;
      for (int j = k + 1 + warp; j < f; j += kWarps) {
        const double lj = colk[j] * dinv;
        double* colj = F + (size_t)ld * j;
        if (j == nxt && want_stats) {
          double bv = -1.0, cm = 0.0;
          int bi = INT_MAX;
          for (int i = j + lane; i < f; i += 32) {
            const double v = colj[i] - colk[i] * lj;
            colj[i] = v;
            if (i > j) {
              const double a = fabs(v);
              if (i < ncand)
                keep_larger(bv, bi, a, i);
              else
                cm = fmax(cm, a);
            }
          }
          warp_argmax_max(bv, bi, cm);
          if (lane == 0) {
            st_v = bv;
            st_i = bi;
            st_m = cm;
          }
        } else {
          for (int i = j + lane; i < f; i += 32) colj[i] -= colk[i] * lj;
        }
      }
      if (tid == 0) {
        if (d >= 0.0)
          npos++;
        else
          nneg++;
        const double r = (double)(f - k - 1);
        flops += r * (r + 1.0) + r;
      }
      pend = 1;
      pc = k;
      pd0 = dinv;
    } else {
      const double* colk1 = colk + ld;
      const double d11 = colk[k];
      const double d21 = colk[k + 1];
      const double d22 = colk1[k + 1];
      const double det = d11 * d22 - d21 * d21;
      const double detinv = 1.0 / det;
      const double i00 = d22 * detinv, i01 = -d21 * detinv, i11 = d11 * detinv;
      for (int j = k + 2 + warp; j < f; j += kWarps) {
        const double a = colk[j];
        const double b = colk1[j];
        const double l0 = a * i00 + b * i01;
        const double l1 = a * i01 + b * i11;
        double* colj = F + (size_t)ld * j;
        if (j == nxt && want_stats) {
          double bv = -1.0, cm = 0.0;
          int bi = INT_MAX;
          for (int i = j + lane; i < f; i += 32) {
            const double v = colj[i] - (colk[i] * l0 + colk1[i] * l1);
            colj[i] = v;
            if (i > j) {
              const double aa = fabs(v);
              if (i < ncand)
                keep_larger(bv, bi, aa, i);
              else
                cm = fmax(cm, aa);
            }
          }
          warp_argmax_max(bv, bi, cm);
          if (lane == 0) {
            st_v = bv;
            st_i = bi;
            st_m = cm;
          }
        } else {
          for (int i = j + lane; i < f; i += 32) colj[i] -= colk[i] * l0 + colk1[i] * l1;
        }
      }
      if (tid == 0) {
        fv[k] = -(fv[k] + 1);
        fv[k + 1] = -(fv[k + 1] + 1);
        if (det >= 0.0) {
          if (d11 >= 0.0)
            npos += 2;
          else
            nneg += 2;
        } else {
          npos++;
          nneg++;
        }
        const double r = (double)(f - k - 2);
        flops += 2.0 * r * (r + 1.0) + 6.0 * r;
      }
      pend = 2;
      pc = k;
      pd0 = i00;
      pd1 = i01;
      pd2 = i11;
    }
    __syncthreads();
    // the warp owning column nxt covered every row below it only if nxt < f
    need_stats = !(want_stats);
    k += nstep;
  }
  // last deferred scaling
  if (pend == 1) {
    double* c0 = F + (size_t)ld * pc;
    for (int i = pc + 1 + tid; i < f; i += blockDim.x) c0[i] *= pd0;
  } else if (pend == 2) {
    double* c0 = F + (size_t)ld * pc;
    double* c1 = c0 + ld;
    for (int i = pc + 2 + tid; i < f; i += blockDim.x) {
      const double a = c0[i];
      const double b = c1[i];
      c0[i] = a * pd0 + b * pd1;
      c1[i] = a * pd1 + b * pd2;
    }
  }
  __syncthreads();

  Result out = {k, npos, nneg, (long long)flops};
  write(out);
  for (int j = k + warp; j < f; j += kWarps)
    for (int i = j + lane; i < f; i += 32) store(i, j, F[i + (size_t)ld * j]);
  return out;
}

// A front of more than kSmemFrontMax rows: its place in the pools, its
// variables, and its entry in the level's lists, by the CTA; assembly and
// factorization are the big-front kernels'.
__device__ void register_big(const DevPlan& p, const DevState& s, const FactorParams& prm,
                             int node, int ns, int nc, int nd_in, long long& sh_ioff,
                             long long& sh_doff, int& sh_nopool) {
  const int tid = threadIdx.x;
  const int fs = ns + nd_in;
  const int f = fs + nc;
  const int kb = p.kid_ptr[node];
  const int ke = p.kid_ptr[node + 1];
  if (tid == 0) {
    int fail = 0;
    const unsigned long long io = atomicAdd(s.used, 2ull * (unsigned long long)f);
    if (io + 2ull * f > s.icap) fail = 1;
    sh_ioff = (long long)io;
    // the front itself plus the panel's W columns; fronts above the
    // on-chip limit also get the chained panel's W by physical row and its
    // permutation scratch
    unsigned long long need = (unsigned long long)f * f + (unsigned long long)kBigPanelMax * f;
    const unsigned long long chain =
        (unsigned long long)kBigPanelMax * f + (unsigned long long)(fs + 1) * f;
    if (prm.app && f >= prm.app_min_f) {
      // a root may finish with the chained panels: their scratch too
      need += (unsigned long long)kAppScratch + (nc == 0 ? chain : 0ull);
    } else if (f > s.cf_limit[4]) {
      need += chain;
    }
    const unsigned long long dofs = atomicAdd(s.used + 1, need);
    if (dofs + need > s.dcap) fail = 1;
    sh_doff = (long long)dofs;
    if (fail) {
      atomicOr(s.err, 1);  // a pool ran out
      atomicCAS(s.err + 1, -1, node);
    }
    sh_nopool = fail;
  }
  __syncthreads();
  if (sh_nopool) return;
  int* fv = s.ivars + sh_ioff;
  int* orig = fv + f;
  // front variables now; assembly and factorization by the big-front kernels
  const int v0b = p.var_ptr[node];
  for (int t = tid; t < ns; t += blockDim.x) fv[t] = p.node_to_var[v0b + t];
  int offb = ns;
  for (int c = kb; c < ke; c++) {
    const int ch = p.kids[c];
    const int nd = s.ndel[ch];
    const int* cfv = s.ivars + s.fv_off[ch] + s.npiv[ch];
    for (int t = tid; t < nd; t += blockDim.x) fv[offb + t] = cfv[t];
    offb += nd;
  }
  const int cb0 = p.cptr[node];
  for (int t = tid; t < nc; t += blockDim.x) fv[fs + t] = p.contrib_rows[cb0 + t];
  for (int t = tid; t < f; t += blockDim.x) orig[t] = t;
  if (tid == 0) {
    const int slot = atomicAdd(s.big_meta, 1);
    atomicMax(s.big_meta + 1, f);
    atomicMax(s.big_meta + 2, fs);
    const bool app = prm.app && f >= prm.app_min_f;
    int cls = 5;
    if (app) {
      cls = 6;
    } else {
      for (int c = 4; c >= 0; c--)
        if (f <= s.cf_limit[c]) cls = c;
    }
    if (cls == 6) {
      const int q = atomicAdd(s.big_meta + 16, 1);
      atomicMax(s.big_meta + 17, f);
      atomicMax(s.big_meta + 18, fs);
      s.class_list[(size_t)6 * p.num_nodes + q] = slot;
    } else if (cls == 5) {
      const int q = atomicAdd(s.big_meta + 3, 1);
      atomicMax(s.big_meta + 4, fs);
      atomicMax(s.big_meta + 15, f);
      s.class_list[(size_t)5 * p.num_nodes + q] = slot;
    } else {
      const int q = atomicAdd(s.big_meta + 5 + cls, 1);
      atomicMax(s.big_meta + 10 + cls, f);
      s.class_list[(size_t)cls * p.num_nodes + q] = slot;
    }
    BigFront b;
    b.node = node;
    b.f = f;
    b.fs = fs;
    b.ns = ns;
    b.nd_in = nd_in;
    b.nc = nc;
    b.k = 0;
    b.ncand = fs;
    b.kstart = 0;
    b.kw = 0;
    b.state = 0;
    b.npos = 0;
    b.nneg = 0;
    b.pad = 0;
    b.app = app ? 1 : 0;
    b.pending = -1;
    b.ioff = sh_ioff;
    b.doff = sh_doff;
    b.woff = sh_doff + (long long)f * f;
    // a-posteriori scratch after the panel's W (and, for a root, after the
    // chained panels' scratch)
    b.xoff = b.woff + (long long)kBigPanelMax * f +
             ((app && nc == 0) ? (long long)kBigPanelMax * f + (long long)(fs + 1) * f : 0ll);
    b.flops = 0.0;
    s.big[slot] = b;
  }
}

// kMax: row chunks of the largest front the launch may meet on chip, or
// kGeneral. CTAs per SM: what the registers of the largest front allow.
//
// A launch covers `count` fronts in level order. With `ticket`, they are
// those of several levels: the CTAs take them in order, and a front waits for
// its children's completion flags (s.done). A CTA holds one front at a time
// and a front's children come before it in the order, so the front that is
// first among the unfinished ones never waits and every wait ends; after a
// failure in any CTA (s.err) or kWaitPolls polls the wait is given up.
// Without `ticket` the launch is one level, a front per CTA, and the
// children are those of earlier launches.
//
// One launch for several levels saves what a level costs beside its
// arithmetic: the launch, the cold instruction cache (a level's front takes
// the code through once), and, while a CTA waits for the children, the
// loads of the front's own values.
constexpr int kGeneral = 4;  // fronts of more than 96 rows by general_front
template <int kMax>
__global__ void __launch_bounds__(kFactorThreads, kMax == 1 ? 4 : kMax == 2 ? 3 : kMax < 5 ? 2 : 1)
    factor_level_kernel(DevPlan p, DevState s, const int* __restrict__ nodes, int count,
                        int* ticket, const double* __restrict__ vals,
                        const double* __restrict__ diag, FactorParams prm, int fcap,
                        int allow_big) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int sh_item, sh_fail, sh_nopool, sh_nd;
  __shared__ long long sh_ioff, sh_doff;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;

  for (;;) {
    if (tid == 0) sh_item = ticket ? atomicAdd(ticket, 1) : (int)blockIdx.x;
    __syncthreads();
    const int item = sh_item;
    if (item >= count) return;
    const int node = nodes[item];
    const int ns = p.ns[node];
    const int nc = p.nc[node];
    const int kb = p.kid_ptr[node];
    const int ke = p.kid_ptr[node + 1];
    const int v0 = p.var_ptr[node];
    const int c0 = p.cptr[node];

    // the children are done, and the sum of their delayed candidates
    auto children = [&]() {
      if (warp == 0) {
        int nd = 0, fail = 0;
        for (int c = kb + lane; c < ke; c += 32) {
          const int ch = p.kids[c];
          if (ticket && !wait_flag(s.done + ch, 1, s.err, 8)) fail = 1;
          nd += __ldcg(s.ndel + ch);
        }
        nd = __reduce_add_sync(0xffffffffu, nd);
        fail = __any_sync(0xffffffffu, fail);
        if (lane == 0) {
          sh_nd = nd;
          sh_fail = fail || *((volatile int*)s.err) != 0;
        }
      }
      __syncthreads();
    };

    // the front with its own entries: zero, Sigma on the own variables'
    // diagonal (d + v and v + d of the values added to it are the same
    // number), the front variables (own, delayed, contribution), the CSR
    // entries of the pivot columns (distinct positions)
    Front fr;
    fr.F = smem;
    int* pos = nullptr;  // [m]: a child's rows in this front
    int nd_in = 0;
    auto own_entries = [&]() {
      const int fs = ns + nd_in;
      const int f = fs + nc;
      fr.f = f;
      fr.fs = fs;
      fr.ld = f | 1;
      fr.vec = fr.F + (size_t)fr.ld * f;
      fr.fv = reinterpret_cast<int*>(fr.vec + 5 * vec_len(f));
      fr.orig = fr.fv + f;
      pos = reinterpret_cast<int*>(fr.vec);
      for (int j = warp; j < f; j += kWarps) {
        double* col = fr.F + fr.ld * j;
        const double dj = (diag && j < ns) ? diag[p.node_to_var[v0 + j]] : 0.0;
        for (int i = j + lane; i < f; i += 32) col[i] = (i == j) ? 0.0 + dj : 0.0;
      }
      for (int t = tid; t < ns; t += kFactorThreads) fr.fv[t] = p.node_to_var[v0 + t];
      for (int t = tid; t < nc; t += kFactorThreads) fr.fv[fs + t] = p.contrib_rows[c0 + t];
      for (int t = tid; t < f; t += kFactorThreads) fr.orig[t] = t;
      __syncthreads();
      const int64_t b0 = p.scat_ptr[node];
      const int64_t b1 = p.scat_ptr[node + 1];
      for (int64_t e = b0 + tid; e < b1; e += kFactorThreads) {
        int r = p.scat_row[e];
        if (r >= ns) r += nd_in;
        fr.F[r + fr.ld * p.scat_col[e]] += csr_value(s, vals, p.scat_csr[e]);
      }
      __syncthreads();
    };
    // while the children may still run, with no delays from them (the usual
    // case); otherwise again once their number is known
    const bool early = ticket && ns + nc <= fcap;
    if (early) own_entries();
    children();
    if (sh_fail) return;
    nd_in = sh_nd;
    const int f = ns + nd_in + nc;
    const bool big = f > kSmemFrontMax;
    // the launch's shared memory holds fronts up to fcap: a larger one stops
    // the factorization, which the host repeats with room for every front; a
    // big front in a level the host does not prepare big fronts for stops it
    // too, and the host repeats it with every level prepared
    if ((!big && f > fcap) || (big && !allow_big)) {
      if (tid == 0) {
        atomicOr(s.err, big ? 4 : 2);
        atomicCAS(s.err + 1, -1, node);
      }
      return;
    }
    if (big) {
      register_big(p, s, prm, node, ns, nc, nd_in, sh_ioff, sh_doff, sh_nopool);
      return;
    }
    if (tid == 0) {
      const unsigned long long io = atomicAdd(s.used, 2ull * (unsigned long long)f);
      sh_ioff = (long long)io;
      sh_nopool = io + 2ull * f > s.icap;
    }
    if (!early || nd_in > 0) own_entries();

    // extend-add the children's contribution blocks, one child at a time: the
    // rows' positions first, then whole columns, whose entries (at most
    // kSmemFrontMax / 32 + 1 per lane) are loaded together. What other CTAs of
    // this launch wrote is read from L2.
    {
      double* F = fr.F;
      const int ld = fr.ld;
      int off = ns;
      for (int c = kb; c < ke; c++) {
        const int ch = p.kids[c];
        const int nd = __ldcg(s.ndel + ch);
        const int np = __ldcg(s.npiv + ch);
        const int m = __ldcg(s.f + ch) - np;
        const double* cb = s.dpool + __ldcg(s.cb_off + ch);
        const int cld = __ldcg(s.cb_ld + ch);
        const int* cm = p.cmap + p.cptr[ch];
        const int* cfv = s.ivars + __ldcg(s.fv_off + ch) + np;
        for (int t = tid; t < m; t += kFactorThreads) {
          int q;
          if (t < nd) {
            q = off + t;
            fr.fv[q] = __ldcg(cfv + t);
          } else {
            q = cm[t - nd];
            if (q >= ns) q += nd_in;
          }
          pos[t] = q;
        }
        __syncthreads();
        constexpr int kC = kSmemFrontMax / 32 + 1;
        for (int r2 = warp; r2 < m; r2 += kWarps) {
          const int p2 = pos[r2];
          const double* col = cb + (size_t)cld * r2;
          double v[kC];
#pragma unroll
          for (int u = 0; u < kC; u++) {
            const int r1 = r2 + lane + 32 * u;
            v[u] = r1 < m ? __ldcg(col + r1) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < kC; u++) {
            const int r1 = r2 + lane + 32 * u;
            if (r1 < m) {
              const int p1 = pos[r1];
              if (p1 >= p2)
                F[p1 + ld * p2] += v[u];
              else
                F[p2 + ld * p1] += v[u];
            }
          }
        }
        __syncthreads();
        off += nd;
      }
      if (kb == ke) __syncthreads();
    }

    // partial factorization, then the factor columns and the contribution
    // block
    const bool root = (nc == 0);
    const bool no_ints = sh_nopool != 0;
    double* C = nullptr;
    int m = 0;
    auto write = [&](const Result& o) {
      const int npiv = o.npiv;
      m = f - npiv;
      if (tid == 0) {
        const unsigned long long need = (unsigned long long)f * npiv + (unsigned long long)m * m;
        const unsigned long long dofs = atomicAdd(s.used + 1, need);
        sh_doff = (long long)dofs;
        const int fail = no_ints || dofs + need > s.dcap;
        if (fail) {
          atomicOr(s.err, 1);  // a pool ran out
          atomicCAS(s.err + 1, -1, node);
        }
        sh_nopool = fail;
      }
      __syncthreads();
      if (sh_nopool) return;
      int* gfv = s.ivars + sh_ioff;
      for (int t = tid; t < f; t += kFactorThreads) {
        gfv[t] = fr.fv[t];
        gfv[f + t] = fr.orig[t];
      }
      double* L = s.dpool + sh_doff;
      C = L + (size_t)f * npiv;
      for (int j = warp; j < npiv; j += kWarps)
        for (int i = lane; i < f; i += 32) L[i + (size_t)f * j] = fr.F[i + fr.ld * j];
    };
    auto store = [&](int i, int j, double x) {
      if (C) C[(i + m - f) + (size_t)m * (j + m - f)] = x;
    };
    Result o;
    const int chunks = row_chunks(f);
    if (chunks == 1)
      o = factor_front<1>(fr, root, prm, write, store);
    else if (kMax >= 2 && chunks == 2)
      o = factor_front<(kMax < 2 ? kMax : 2)>(fr, root, prm, write, store);
    else if (kMax >= 3 && chunks == 3)
      o = factor_front<(kMax < 3 ? kMax : 3)>(fr, root, prm, write, store);
    else if constexpr (kMax == kGeneral)
      o = general_front(fr, root, prm, write, store);
    else
      o = factor_front<kMax>(fr, root, prm, write, store);
    if (sh_nopool) return;
    if (tid == 0) {
      s.f[node] = f;
      s.fs[node] = fr.fs;
      s.npiv[node] = o.npiv;
      s.ndel[node] = fr.fs - o.npiv;
      s.fv_off[node] = sh_ioff;
      s.L_off[node] = sh_doff;
      s.L_ld[node] = f;
      s.cb_off[node] = sh_doff + (long long)f * o.npiv;
      s.cb_ld[node] = m > 0 ? m : 1;
    }
    __syncthreads();
    if (tid == 0) {
      flag_set(s.done + node, 1);
      s.u_off[node] = (long long)atomicAdd(s.used + 2, (unsigned long long)m);
      if (!prm.cholesky) {
        atomicAdd(s.inertia, o.npos);
        atomicAdd(s.inertia + 1, o.nneg);
      }
      atomicAdd(s.flops, (double)o.flops);
    }
    if (!ticket) return;
  }
}

}  // namespace

int factor_variant(int fmax) { return row_chunks(fmax); }

size_t factor_smem_bytes(int f) {
  // the front (ld = f | 1), the travelling columns, the variables and their
  // positions at assembly
  const size_t ld = (size_t)(f | 1);
  return (ld * f + 5 * (size_t)vec_len(f)) * sizeof(double) + 2 * (size_t)f * sizeof(int);
}

namespace {

template <int kMax>
cudaError_t configure_chunks() {
  const int fmax = kMax < kGeneral ? 32 * kMax : kSmemFrontMax;
  return cudaFuncSetAttribute(factor_level_kernel<kMax>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)factor_smem_bytes(fmax));
}

}  // namespace

void launch_factor_level(const DevPlan& p, const DevState& s, const int* nodes, int count,
                         int* ticket, int grid, int fmax, int allow_big,
                         const FactorParams& prm, cudaStream_t stream, const double* vals,
                         const double* diag) {
  if (count <= 0) return;
  auto* kernel = fmax <= 32   ? factor_level_kernel<1>
                 : fmax <= 64 ? factor_level_kernel<2>
                 : fmax <= 96 ? factor_level_kernel<3>
                 : prm.app || ticket ? factor_level_kernel<5>
                                     : factor_level_kernel<kGeneral>;
  kernel<<<grid, kFactorThreads, factor_smem_bytes(fmax), stream>>>(
      p, s, nodes, count, ticket, vals, diag, prm, fmax, allow_big);
}

cudaError_t configure_factor_kernels() {
  cudaError_t e = configure_chunks<1>();
  if (e == cudaSuccess) e = configure_chunks<2>();
  if (e == cudaSuccess) e = configure_chunks<3>();
  if (e == cudaSuccess) e = configure_chunks<kGeneral>();
  if (e == cudaSuccess) e = configure_chunks<5>();
  return e;
}

}  // namespace b200ldl
