// Supernodal solves with the stored multifrontal factor.
//
// Forward (leaves to roots): each supernode assembles a front vector from the
// right-hand side at its own variables and the update vectors of its
// children, applies its unit-lower pivot block (1x1 and 2x2 pivots) down the
// whole front, writes D^{-1} t to the solution at its pivot variables and
// leaves the rest of the front as its own update vector for the parent. No
// two supernodes of a level write the same location, so the sweep is
// deterministic and needs no atomics.
//
// Backward (roots to leaves): gather the final solution at the delayed and
// contribution rows, subtract L21^T x2, back-substitute L11^T and scatter to
// the pivot variables.
//
// Same arithmetic as the reference's solve_ldl (include/sparse_ldl.h:
// 1825-1926: solve_pivot_lower, L21 product, scatter_subtract,
// solve_pivot_diagonal, and the transposed sweep), reorganised so that the
// descendants' contributions travel as update vectors instead of
// scatter-subtracts into the shared solution vector, and blocked: one warp
// per right-hand side solves each diagonal block of up to 32 pivots while the
// other warps load the rows below, and the whole CTA applies the block to
// them.
//
// A launch covers the supernodes of one or more consecutive levels, a CTA
// each. What bounds a narrow tree is the path from one supernode to the next
// (two 32-step substitutions of about 35 cycles a step, and the global
// round trips of the update vector and its flag), so the levels are not
// separated by launches: the CTAs take the supernodes in level order, load
// what does not depend on the neighbours (variables, maps, the first block of
// the factor), and wait for the children's flags (forward) or the parent's
// (backward). Both sweeps share a launch when no supernode needs a cluster.
// Optimal control N = 1000 (167 supernodes of 64..68 rows one after another),
// eight right-hand sides: 11.9 ms with a launch per level and sweep, 3.2 ms
// now; one right-hand side of 512 such systems: 9.8 and 2.8 ms.
#include <algorithm>

#include "ldl_internal.h"
#include "solve_common.cuh"

namespace b200ldl {

namespace {

constexpr int kSWarps = kSolveThreads / 32;
constexpr int kBlk = 32;
constexpr int kTileLd = kBlk + 1;
constexpr int kMaxRhs = kSWarps;  // right-hand sides per launch: a warp each

// Progress of a supernode in the solve numbered `epoch`: its flags hold
// 2 epoch once the update vector is written, 2 epoch + 1 once the forward
// solution is, and, in the backward sweep's array, 2 epoch + 1 once the final
// solution is. They grow from solve to solve, so that a solve needs no
// clearing (the host clears them and starts over after some thousand solves).

// end of the pivot block starting at jb: at most 32 pivots, and 2x2 pairs
// never straddle two blocks
__device__ __forceinline__ int block_end(const int* fv, int jb, int npiv) {
  // pairs are consecutive 2x2-marked entries; blocks start on a pair boundary
  const int lane = threadIdx.x & 31;
  const int last = min(jb + kBlk, npiv);
  if (last == npiv) return npiv;
  // the run of marked entries that ends at the block's last position: odd
  // length means that its last entry opens a pair
  const unsigned neg = __ballot_sync(0xffffffffu, fv[jb + lane] < 0);
  const int run = __clz(~neg);
  return (run & 1) ? last - 1 : last;
}

// Bit t set if position jb + t is the second row of a 2x2 pivot. Blocks
// start on a pair boundary, so inside a run of negative (2x2-marked) entries
// the odd offsets are the second rows.
__device__ __forceinline__ unsigned second_rows(const int* fv, int jb, int je, int lane) {
  const bool neg = (jb + lane < je) && fv[jb + lane] < 0;
  const unsigned negm = __ballot_sync(0xffffffffu, neg);
  const unsigned below = lane == 0 ? 0u : (~negm) & ((1u << lane) - 1u);
  const int start = below ? (32 - __clz(below)) : 0;
  return __ballot_sync(0xffffffffu, neg && ((lane - start) & 1));
}

// Front vectors in shared memory, the right-hand sides of a row together
// (padded so that 16-byte accesses of consecutive rows meet different banks).
template <int kNr>
constexpr int kVld = kNr <= 2 ? kNr : kNr + 2;

// The diagonal block [jb, je) of L, column-major in a tile: four columns a
// warp, loaded together and stored by put_tile.
struct TilePart {
  double v[kBlk / kSWarps];
};
__device__ __forceinline__ TilePart get_tile(const double* L, int ldl, int jb, int je, int warp,
                                             int lane) {
  TilePart t;
#pragma unroll
  for (int u = 0; u < kBlk / kSWarps; u++) {
    const int j = jb + warp + kSWarps * u;
    t.v[u] = (j < je && jb + lane < je) ? L[(jb + lane) + (size_t)ldl * j] : 0.0;
  }
  return t;
}
__device__ __forceinline__ void put_tile(double* tile, const TilePart& t, int warp, int lane) {
#pragma unroll
  for (int u = 0; u < kBlk / kSWarps; u++) tile[(warp + kSWarps * u) * kTileLd + lane] = t.v[u];
}

// One warp: forward substitution of the rows [jb, je) of one right-hand side
// (row stride ldv) with the unit-lower block (column stride ldt). Returns the
// second rows of the block's 2x2 pivots.
__device__ __forceinline__ unsigned fwd_block(const double* tile, int ldt, const int* fv, int jb,
                                              int je, double* v, int ldv, int lane) {
  const int nb = je - jb;
  const unsigned sec = second_rows(fv, jb, je, lane);
  double Lrow[kBlk];
#pragma unroll
  for (int j = 0; j < kBlk; j++) Lrow[j] = (j < nb && lane < nb) ? tile[j * ldt + lane] : 0.0;
  double vr = lane < nb ? v[(jb + lane) * ldv] : 0.0;
#pragma unroll
  for (int j = 0; j < kBlk; j++) {
    if (j < nb) {
      const bool first = j + 1 < nb && ((sec >> (j + 1)) & 1u);
      const bool upd = lane > j && !(first && lane == j + 1);
      const double vj = __shfl_sync(0xffffffffu, vr, j);
      if (upd) vr = fma(-Lrow[j], vj, vr);
    }
  }
  if (lane < nb) v[(jb + lane) * ldv] = vr;
  return sec;
}

// One warp: back substitution with the transposed block.
__device__ __forceinline__ void bwd_block(const double* tile, int ldt, const int* fv, int jb,
                                          int je, double* v, int ldv, int lane) {
  const int nb = je - jb;
  const unsigned sec = second_rows(fv, jb, je, lane);
  double Lcol[kBlk];
#pragma unroll
  for (int q = 0; q < kBlk; q++) Lcol[q] = (q < nb && lane < nb) ? tile[lane * ldt + q] : 0.0;
  double vr = lane < nb ? v[(jb + lane) * ldv] : 0.0;
#pragma unroll
  for (int jj = kBlk - 1; jj >= 0; jj--) {
    if (jj < nb) {
      const bool upd = lane < jj && !(((sec >> jj) & 1u) && lane == jj - 1);
      const double vj = __shfl_sync(0xffffffffu, vr, jj);
      if (upd) vr = fma(-Lcol[jj], vj, vr);
    }
  }
  if (lane < nb) v[(jb + lane) * ldv] = vr;
}

// Sums over the warp of kN values per lane (kN a power of two up to 32), the
// sum of value i in the lanes whose top bits are i's: with every halving of
// the lanes a lane keeps half of its values. Each value's partial sums meet
// in the pairs (l, l + 16), (l, l + 8), ..., as in a shuffle-down tree, so
// the sum has the bits of that tree.
template <int kN>
__device__ __forceinline__ double warp_sums(double (&a)[kN], int lane) {
  int o = 16;
#pragma unroll
  for (int n = kN / 2; n >= 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const double keep = up ? a[i + n] : a[i];
      const double send = up ? a[i] : a[i + n];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = a[0];
#pragma unroll
  for (; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// v[j][r] -= sum_{i in [i0, i1)} L(i, j) v[i][r] for the columns j0, j0 + 8,
// .. of one warp pass (at most kColsPer, below j1), four rows per lane at a
// time: their loads are in flight together. A lane's rows are i0 + lane + 32 t
// in order, whatever the number of columns.
template <int kNr>
constexpr int kColsPer = kNr >= 8 ? 2 : 4;

template <int kNr>
__device__ __forceinline__ void gemv_t(const double* L, int ldl, int j0, int j1, int i0, int i1,
                                       double* v, int nr, int lane) {
  constexpr int kC = kColsPer<kNr>;
  constexpr int kLd = kVld<kNr>;
  double acc[kC * kNr];
#pragma unroll
  for (int q = 0; q < kC * kNr; q++) acc[q] = 0.0;
  for (int ib = i0 + lane; ib < i1; ib += 128) {
    double l4[kC][4];
#pragma unroll
    for (int c = 0; c < kC; c++) {
      const double* lj = L + (size_t)ldl * (j0 + kSWarps * c);
#pragma unroll
      for (int u = 0; u < 4; u++)
        l4[c][u] = (j0 + kSWarps * c < j1 && ib + 32 * u < i1) ? lj[ib + 32 * u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = ib + 32 * u;
      if (i < i1) {
#pragma unroll
        for (int r = 0; r < kNr; r++) {
          const double vi = v[i * kLd + r];
#pragma unroll
          for (int c = 0; c < kC; c++) acc[c * kNr + r] = fma(l4[c][u], vi, acc[c * kNr + r]);
        }
      }
    }
  }
  __syncwarp();
  const double s = warp_sums<kC * kNr>(acc, lane);
  constexpr int kLanes = 32 / (kC * kNr);  // lanes that hold the same sum
  const int q = lane / kLanes;
  const int c = q / kNr, r = q % kNr;
  const int j = j0 + kSWarps * c;
  if (lane % kLanes == 0 && r < nr && j < j1) v[j * kLd + r] -= s;
}

struct SolveArgs {
  const int* nodes;   // the launch's supernodes in level order
  int count;
  int* ticket;        // nullptr: a CTA per supernode, neighbours done before
  const int* parent;  // [num_nodes] -1 for roots
  int* fdone;         // [num_nodes] flags of the forward sweep
  int* bdone;         // [num_nodes] and of the backward sweep
  int epoch;
  int* fail;          // set when a wait was given up
  int* host_fail;     // the same for the host to read
  int wait_polls;     // limit of a wait
  int sweeps;         // 1: forward, 2: backward, 3: forward, then backward
  double* x;
  int ldx, nrhs, r0, nr;
  double* upool;
  int stage_cap;      // doubles of shared memory for a supernode's factor
};

// A supernode whose factor columns fit `stage_cap` doubles keeps them in
// shared memory: they are loaded before the wait for the neighbours, and the
// substitutions then never leave the SM.
__device__ __forceinline__ void stage_factor(double* Ls, int ld, const double* L, int ldl, int f,
                                             int npiv, int warp, int lane) {
  for (int j0 = warp; j0 < npiv; j0 += 4 * kSWarps) {
    double t[4][3];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = j0 + kSWarps * u;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = j + lane + 32 * c;
        t[u][c] = (j < npiv && i < f) ? L[i + (size_t)ldl * j] : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = j0 + kSWarps * u;
      if (j >= npiv) break;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = j + lane + 32 * c;
        if (i < f) Ls[i + ld * j] = t[u][c];
      }
      for (int i = j + lane + 96; i < f; i += 32) Ls[i + ld * j] = L[i + (size_t)ldl * j];
    }
  }
}

template <int kNr>
__device__ __forceinline__ bool forward_node(const DevPlan& p, const DevState& s,
                                             const SolveArgs& a, int node, double* sm,
                                             int* sh_fail, ChildBatch* kids) {
  constexpr int kLd = kVld<kNr>;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nr = a.nr;
  const int f = s.f[node];
  const int fs = s.fs[node];
  const int npiv = s.npiv[node];
  const int ns = p.ns[node];
  const int m = f - npiv;
  const int nd_in = fs - ns;
  const int* fv = s.ivars + s.fv_off[node];
  const int* orig = fv + f;
  const double* L = s.dpool + s.L_off[node];
  const int ldl = s.L_ld[node];
  const int kb = p.kid_ptr[node];
  const int ke = p.kid_ptr[node + 1];
  const long long uoff = s.u_off[node];
  // an only child's place in the update vectors, before the wait
  int nd = 0, mc = 0, cptr = 0;
  long long cu = 0;
  if (ke - kb == 1) {
    const int ch = p.kids[kb];
    nd = s.ndel[ch];
    mc = s.f[ch] - s.npiv[ch];
    cu = s.u_off[ch];
    cptr = p.cptr[ch];
  }
  double* tile = sm;                                    // [2][kBlk][kTileLd], or the factor
  double* v = tile + a.stage_cap;                       // [f][kLd], post-pivot order
  int* post_of = reinterpret_cast<int*>(v + (size_t)kLd * f);  // [f]
  int* sfv = post_of + f;                               // [f]
  const int lds = f | 1;
  const bool staged = lds * npiv <= a.stage_cap;

  // the factor (or its first block) does not depend on the children, nor
  // does the right-hand side at the own variables (zero elsewhere)
  for (int q = tid; q < f; q += kSolveThreads) {
    const int o = q < fs ? orig[q] : q;
    const int e = fv[q];
    const int var = e >= 0 ? e : -e - 1;
    post_of[o] = q;
    sfv[q] = e;
    double t[kNr];
#pragma unroll
    for (int r = 0; r < kNr; r++)
      t[r] = (o < ns && r < nr) ? a.x[(size_t)a.ldx * (a.r0 + r) + var] : 0.0;
#pragma unroll
    for (int r = 0; r < kNr; r++) v[q * kLd + r] = t[r];
  }
  if (staged) {
    stage_factor(tile, lds, L, ldl, f, npiv, warp, lane);
  } else {
    const TilePart t = get_tile(L, ldl, 0, min(npiv, kBlk), warp, lane);
    put_tile(tile, t, warp, lane);
  }
  // the children's update vectors, one child at a time (fixed summation
  // order)
  if (a.ticket && warp == 0) {
    bool ok = true;
    for (int c = kb + lane; c < ke; c += 32)
      ok = wait_flag(a.fdone + p.kids[c], 2 * a.epoch, a.fail, 1, a.wait_polls) && ok;
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0 && !ok) *sh_fail = 1;
  }
  __syncthreads();
  if (*sh_fail) return false;
  if (ke - kb > 1)
    add_children<kNr>(p, s, *kids, kb, ke, ns, nd_in, a.upool, a.nrhs, a.r0, nr, post_of,
                      [&](int q, int r, double u) { v[q * kLd + r] += u; });
  int off = ns;
  for (int c = kb; c < ke && ke - kb == 1; c++) {
    const double* uc = a.upool + cu * a.nrhs + (size_t)a.r0 * mc;
    const int* cm = p.cmap + cptr;
    for (int t = tid; t < mc; t += kSolveThreads) {
      double u[kNr];
#pragma unroll
      for (int r = 0; r < kNr; r++) u[r] = r < nr ? __ldcg(uc + (size_t)r * mc + t) : 0.0;
      int q;
      if (t < nd) {
        q = off + t;
      } else {
        q = cm[t - nd];
        if (q >= ns) q += nd_in;
      }
      q = post_of[q];
#pragma unroll
      for (int r = 0; r < kNr; r++)
        if (r < nr) v[q * kLd + r] += u[r];
    }
    __syncthreads();
    off += nd;
  }

  // blocked unit-lower solve
  int* second = post_of;  // [npiv] 1 at the second rows of 2x2 pivots
  int buf = 0;
  for (int jb = 0; jb < npiv;) {
    const int je = block_end(sfv, jb, npiv);
    const int nb = je - jb;
    const double* tl = staged ? tile + jb + lds * jb : tile + buf * kBlk * kTileLd;
    const int ldt = staged ? lds : kTileLd;
    if (warp < nr) {
      const unsigned sec = fwd_block(tl, ldt, sfv, jb, je, v + warp, kLd, lane);
      if (warp == 0 && lane < nb) second[jb + lane] = (sec >> lane) & 1u;
    }
    if (staged) {
      // a warp takes 32 rows and two right-hand sides (the last block has few
      // rows below it)
      constexpr int kRp = kNr < 2 ? 1 : 2;
      constexpr int kG = kNr / kRp;
      __syncthreads();
      const int r0 = (warp % kG) * kRp;
      for (int i = je + 32 * (warp / kG) + lane; i < f; i += 32 * (kSWarps / kG)) {
        double acc[kRp];
#pragma unroll
        for (int r = 0; r < kRp; r++) acc[r] = 0.0;
        const double* li = tile + i + lds * jb;
        const double* vj = v + jb * kLd + r0;
        if (nb == kBlk) {
#pragma unroll
          for (int j = 0; j < kBlk; j++) {
            const double l = li[lds * j];
#pragma unroll
            for (int r = 0; r < kRp; r++) acc[r] = fma(l, vj[j * kLd + r], acc[r]);
          }
        } else {
#pragma unroll 4
          for (int j = 0; j < nb; j++) {
            const double l = li[lds * j];
#pragma unroll
            for (int r = 0; r < kRp; r++) acc[r] = fma(l, vj[j * kLd + r], acc[r]);
          }
        }
#pragma unroll
        for (int r = 0; r < kRp; r++) v[i * kLd + r0 + r] -= acc[r];
      }
    } else {
      // a thread takes a row and every right-hand side; the warps without a
      // right-hand side come first, and the first row's entries are loaded
      // while the blocks are solved
      const int i0 = je + ((tid + kSolveThreads - 32 * min(nr, kSWarps - 1)) % kSolveThreads);
      double lv[kBlk];
      const double* li = L + i0 + (size_t)ldl * jb;
#pragma unroll
      for (int j = 0; j < kBlk; j++) lv[j] = (i0 < f && j < nb) ? li[(size_t)ldl * j] : 0.0;
      TilePart nt;
      const bool next = je < npiv;
      if (next) nt = get_tile(L, ldl, je, min(npiv, je + kBlk), warp, lane);
      __syncthreads();
      for (int i = i0; i < f; i += kSolveThreads) {
        double acc[kNr];
#pragma unroll
        for (int r = 0; r < kNr; r++) acc[r] = 0.0;
        if (i != i0) {
          const double* lr = L + i + (size_t)ldl * jb;
#pragma unroll
          for (int j = 0; j < kBlk; j++) lv[j] = j < nb ? lr[(size_t)ldl * j] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kBlk; j++) {
          // beyond the block both factors are zero: the sum stays as it is
#pragma unroll
          for (int r = 0; r < kNr; r++)
            acc[r] = fma(lv[j], j < nb ? v[(jb + j) * kLd + r] : 0.0, acc[r]);
        }
#pragma unroll
        for (int r = 0; r < kNr; r++) v[i * kLd + r] -= acc[r];
      }
      buf ^= 1;
      if (next) put_tile(tile + buf * kBlk * kTileLd, nt, warp, lane);
    }
    __syncthreads();
    jb = je;
  }
  double* uo = a.upool + uoff * a.nrhs + (size_t)a.r0 * m;
  for (int t = tid; t < m; t += kSolveThreads) {
#pragma unroll
    for (int r = 0; r < kNr; r++)
      if (r < nr) uo[(size_t)r * m + t] = v[(npiv + t) * kLd + r];
  }
  __syncthreads();
  if (tid == 0) flag_set(a.fdone + node, 2 * a.epoch);
  // D^{-1}: 1x1 pivots divide; 2x2 pairs use their partner's value
  const double* Ld = staged ? tile : L;
  const int ldd = staged ? lds : ldl;
  for (int q = tid; q < npiv; q += kSolveThreads) {
    const int e = sfv[q];
    const int vi = e >= 0 ? e : -e - 1;
    const bool is_sec = second[q] != 0;
    const bool is_first = e < 0 && !is_sec;
    const double dd = Ld[q + (size_t)ldd * q];
    double d11 = dd, d21 = 0.0, d22 = dd;
    if (is_first) {
      d21 = Ld[(q + 1) + (size_t)ldd * q];
      d22 = Ld[(q + 1) + (size_t)ldd * (q + 1)];
    } else if (is_sec) {
      d21 = Ld[q + (size_t)ldd * (q - 1)];
      d11 = Ld[(q - 1) + (size_t)ldd * (q - 1)];
    }
    for (int r = 0; r < nr; r++) {
      const double* vr = v + r;
      double y;
      if (is_first)
        y = (d22 * vr[q * kLd] - d21 * vr[(q + 1) * kLd]) / (d11 * d22 - d21 * d21);
      else if (is_sec)
        y = (d11 * vr[q * kLd] - d21 * vr[(q - 1) * kLd]) / (d11 * d22 - d21 * d21);
      else
        y = vr[q * kLd] / dd;
      a.x[(size_t)a.ldx * (a.r0 + r) + vi] = y;
    }
  }
  __syncthreads();
  if (tid == 0) flag_set(a.fdone + node, 2 * a.epoch + 1);
  return true;
}

template <int kNr>
__device__ __forceinline__ bool backward_node(const DevPlan& p, const DevState& s,
                                              const SolveArgs& a, int node, double* sm,
                                              int* sh_fail) {
  constexpr int kLd = kVld<kNr>;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nr = a.nr;
  const int f = s.f[node];
  const int npiv = s.npiv[node];
  const int* fv = s.ivars + s.fv_off[node];
  const double* L = s.dpool + s.L_off[node];
  const int ldl = s.L_ld[node];
  double* tile = sm;                                     // [2][kBlk][kTileLd], or the factor
  double* v = tile + a.stage_cap;                        // [f][kLd]
  int* sfv = reinterpret_cast<int*>(v + (size_t)kLd * f);  // [f]
  int* bst = sfv + f;                                    // block starts
  const int lds = f | 1;
  const bool staged = lds * npiv <= a.stage_cap;

  for (int q = tid; q < f; q += kSolveThreads) sfv[q] = fv[q];
  if (staged) stage_factor(tile, lds, L, ldl, f, npiv, warp, lane);
  __syncthreads();
  if (warp == 0) {
    int nb = 0;
    for (int jb = 0; jb < npiv;) {
      if (lane == 0) bst[nb] = jb;
      nb++;
      jb = block_end(sfv, jb, npiv);
    }
    if (lane == 0) bst[nb] = npiv;
  }
  if (a.sweeps == 3 && tid == 32 &&
      !wait_flag(a.fdone + node, 2 * a.epoch + 1, a.fail, 1, a.wait_polls))
    *sh_fail = 1;  // the own forward solution
  __syncthreads();
  if (*sh_fail) return false;
  // blocks: all but the last hold 31 or 32 pivots
  int b = npiv > 0 ? (npiv - 1) / kBlk : -1;
  while (b >= 0 && bst[b + 1] != npiv) b++;
  // the last diagonal block and the own rows do not depend on the parent
  if (b >= 0 && !staged) {
    const TilePart t = get_tile(L, ldl, bst[b], npiv, warp, lane);
    put_tile(tile, t, warp, lane);
  }
  auto gather = [&](int q0, int q1) {
    for (int q = q0 + tid; q < q1; q += kSolveThreads) {
      const int e = sfv[q];
      const int var = e >= 0 ? e : -e - 1;
      double t[kNr];
#pragma unroll
      for (int r = 0; r < kNr; r++)
        t[r] = r < nr ? __ldcg(a.x + (size_t)a.ldx * (a.r0 + r) + var) : 0.0;
#pragma unroll
      for (int r = 0; r < kNr; r++) v[q * kLd + r] = t[r];
    }
  };
  gather(0, npiv);
  if (a.ticket && tid == 0) {
    const int par = a.parent[node];
    if (par >= 0 && !wait_flag(a.bdone + par, 2 * a.epoch + 1, a.fail, 1, a.wait_polls))
      *sh_fail = 1;
  }
  __syncthreads();
  if (*sh_fail) return false;
  gather(npiv, f);
  __syncthreads();
  // t1 -= L21^T x2
  constexpr int kStep = kSWarps * kColsPer<kNr>;
  const double* Lg = staged ? tile : L;
  const int ldg = staged ? lds : ldl;
  if (npiv < f) {
    for (int j = warp; j < npiv; j += kStep)
      gemv_t<kNr>(Lg, ldg, j, npiv, npiv, f, v, nr, lane);
    __syncthreads();
  }
  // L11^T back substitution, block by block from the last
  int buf = 0;
  for (; b >= 0; b--) {
    const int jb = bst[b];
    const int je = bst[b + 1];
    if (je < npiv) {
      for (int j = jb + warp; j < je; j += kStep)
        gemv_t<kNr>(Lg, ldg, j, je, je, npiv, v, nr, lane);
      __syncthreads();
    }
    TilePart nt;
    const bool next = b > 0 && !staged;
    if (next) nt = get_tile(L, ldl, bst[b - 1], jb, warp, lane);
    if (warp < nr)
      bwd_block(staged ? tile + jb + lds * jb : tile + buf * kBlk * kTileLd,
                staged ? lds : kTileLd, sfv, jb, je, v + warp, kLd, lane);
    buf ^= 1;
    if (next) put_tile(tile + buf * kBlk * kTileLd, nt, warp, lane);
    __syncthreads();
  }
  for (int q = tid; q < npiv; q += kSolveThreads) {
    const int e = sfv[q];
    const int var = e >= 0 ? e : -e - 1;
#pragma unroll
    for (int r = 0; r < kNr; r++)
      if (r < nr) a.x[(size_t)a.ldx * (a.r0 + r) + var] = v[q * kLd + r];
  }
  __syncthreads();
  if (tid == 0) flag_set(a.bdone + node, 2 * a.epoch + 1);
  return true;
}

// The supernodes of a launch in level order, forward, and in the opposite
// order, backward. The CTAs take them in turn (ticket); a supernode's
// neighbours that it waits for come before it in that order, so the first
// unfinished one never waits and every wait ends; after kWaitPolls polls it is
// given up, and the others with it.
template <int kNr>
__global__ void __launch_bounds__(kSolveThreads, 2)
    solve_kernel(DevPlan p, DevState s, SolveArgs a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int sh_item, sh_fail;
  __shared__ ChildBatch kids;
  const int items = a.sweeps == 3 ? 2 * a.count : a.count;
  if (threadIdx.x == 0) sh_fail = 0;
  for (;;) {
    if (threadIdx.x == 0) sh_item = a.ticket ? atomicAdd(a.ticket, 1) : (int)blockIdx.x;
    __syncthreads();
    const int item = sh_item;
    if (item >= items) return;
    bool ok;
    if ((a.sweeps & 1) && item < a.count)
      ok = forward_node<kNr>(p, s, a, a.nodes[item], sm, &sh_fail, &kids);
    else
      ok = backward_node<kNr>(p, s, a, a.nodes[items - 1 - item], sm, &sh_fail);
    if (!ok) {
      if (threadIdx.x == 0) *((volatile int*)a.host_fail) = 1;
      return;
    }
    if (!a.ticket) return;
    __syncthreads();
  }
}

constexpr size_t kSolveSmemMax = 224 * 1024;

// doubles for the factor columns of a supernode: two diagonal blocks at
// least (stage_doubles)
constexpr int kStageMin = 2 * kBlk * kTileLd;

size_t solve_smem(int fmax, int nr, int stage_cap) {
  const int ld = nr == 1 ? 1 : nr == 2 ? 2 : nr <= 4 ? kVld<4> : kVld<8>;
  return (stage_cap + (size_t)ld * fmax) * sizeof(double) +
         (2 * (size_t)fmax + fmax / 31 + 4) * sizeof(int);
}

// Room for the factor columns in a launch of fronts up to fmax rows: all of
// the largest front's, but at most 40 KB, so that two CTAs per SM (as many as
// the registers allow) leave more than half of the SM's memory to L1, where
// the fronts that do not fit are read; where two CTAs would not fit with that,
// the two diagonal blocks.
int stage_doubles(int fmax, int nr) {
  const size_t most = 40 * 1024 / sizeof(double);
  const int all = (int)std::min((size_t)(fmax | 1) * fmax, most);
  return solve_smem(fmax, nr, all) <= 112 * 1024 ? std::max(kStageMin, all) : kStageMin;
}

}  // namespace

cudaError_t configure_solve_kernels() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* k) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kSolveSmemMax);
  };
  set(solve_kernel<1>);
  set(solve_kernel<2>);
  set(solve_kernel<4>);
  set(solve_kernel<8>);
  return e;
}

// right-hand sides per launch so that the front vectors fit
int solve_rhs_chunk(int fmax, int nrhs) {
  int c = nrhs < kMaxRhs ? nrhs : kMaxRhs;
  while (c > 0 && solve_smem(fmax, c, kStageMin) > kSolveSmemMax) c--;
  return c;
}

void launch_solve(const DevPlan& p, const DevState& s, const SolveSpan& sp, int sweeps, double* x,
                  int ldx, int nrhs, int r0, int nr, double* upool, cudaStream_t stream) {
  if (sp.count <= 0) return;
  SolveArgs a;
  a.nodes = sp.nodes;
  a.count = sp.count;
  a.ticket = sp.ticket;
  a.parent = sp.parent;
  a.fdone = sp.fdone;
  a.bdone = sp.bdone;
  a.epoch = sp.epoch;
  a.fail = sp.fail;
  a.host_fail = sp.host_fail;
  a.wait_polls = sp.wait_polls;
  a.sweeps = sweeps;
  a.x = x;
  a.ldx = ldx;
  a.nrhs = nrhs;
  a.r0 = r0;
  a.nr = nr;
  a.upool = upool;
  auto* k = nr == 1 ? solve_kernel<1> : nr == 2 ? solve_kernel<2> : nr <= 4 ? solve_kernel<4>
                                                                             : solve_kernel<8>;
  a.stage_cap = stage_doubles(sp.fmax, nr);
  k<<<sp.grid, kSolveThreads, solve_smem(sp.fmax, nr, a.stage_cap), stream>>>(p, s, a);
}

}  // namespace b200ldl
