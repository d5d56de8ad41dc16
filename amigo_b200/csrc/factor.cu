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
// registers (factor_front) or where they stand (general_front); larger ones
// are registered for the big-front kernels.
#include <climits>

#include "ldl_internal.h"
#include "register_front.cuh"

namespace b200ldl {

namespace {

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

// The same factorization in shared memory, with the same bits: the one for
// fronts of more than 96 rows on a level with a launch of its own, unless the
// structure was re-planned from a pivot record. Those are the levels beside
// big fronts (and all levels of a first factorization, whose sizes are not
// known yet). Where a tree has such levels without a record, its fronts delay
// candidates by the dozen, and a delay moves two rows and columns in one pass
// of the CTA here, while the register fronts form and replace them slot by
// slot, several thousand cycles a delay at 18 slots of 5 chunks: plane stress
// 64 x 64 in the first order, small fronts 7.1 ms of the factorization's 83.8
// with this one, 8.7 of 85.5 with registers throughout (24 x 24: 14.3 and
// 14.9 ms). Levels that share a launch have registers: optimal control with
// 48 states, N = 40, 8.7 ms against 13.4 with this one, 64 systems of N = 20
// of them, 530 delays each, 4.5 against 6.8.
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
          const double det = fabs(two_products(wkk, wii, -wik, wik));
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
        c0[i] = two_products(a, pd0, b, pd1);
        c1[i] = two_products(a, pd1, b, pd2);
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
            const double v = fma(-colk[i], lj, colj[i]);
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
          for (int i = j + lane; i < f; i += 32) colj[i] = fma(-colk[i], lj, colj[i]);
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
      const double det = two_products(d11, d22, -d21, d21);
      const double detinv = 1.0 / det;
      const double i00 = d22 * detinv, i01 = -d21 * detinv, i11 = d11 * detinv;
      for (int j = k + 2 + warp; j < f; j += kWarps) {
        const double a = colk[j];
        const double b = colk1[j];
        const double l0 = two_products(a, i00, b, i01);
        const double l1 = two_products(a, i01, b, i11);
        double* colj = F + (size_t)ld * j;
        if (j == nxt && want_stats) {
          double bv = -1.0, cm = 0.0;
          int bi = INT_MAX;
          for (int i = j + lane; i < f; i += 32) {
            const double v = colj[i] - two_products(colk[i], l0, colk1[i], l1);
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
          for (int i = j + lane; i < f; i += 32)
            colj[i] -= two_products(colk[i], l0, colk1[i], l1);
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
      c0[i] = two_products(a, pd0, b, pd1);
      c1[i] = two_products(a, pd1, b, pd2);
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
          if (ticket && !wait_flag(s.done + ch, 1, s.err, 8, prm.wait_polls)) fail = 1;
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
      fr.fv = reinterpret_cast<int*>(fr.vec + kVecs * vec_len(f));
      fr.orig = fr.fv + f;
      pos = reinterpret_cast<int*>(fr.vec);
      // a thread per own variable for the diagonal: two dependent loads each
      for (int t = tid; t < ns; t += kFactorThreads) {
        const int v = p.node_to_var[v0 + t];
        fr.fv[t] = v;
        fr.F[t + fr.ld * t] = 0.0 + (diag ? diag[v] : 0.0);
      }
      for (int j = warp; j < f; j += kWarps) {
        double* col = fr.F + fr.ld * j;
        for (int i = j + lane + (j < ns && lane == 0 ? 32 : 0); i < f; i += 32) col[i] = 0.0;
      }
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
      if (ticket)
        flag_set(s.done + node, 1);
      else
        s.done[node] = 1;  // for the launches that follow
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
  return (ld * f + kVecs * (size_t)vec_len(f)) * sizeof(double) + 2 * (size_t)f * sizeof(int);
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
  // above 96 rows: see general_front
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
