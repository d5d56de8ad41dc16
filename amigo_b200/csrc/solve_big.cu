// Solves with the supernodes of large fronts, one thread-block cluster of
// 16 CTAs per supernode.
//
// A single CTA streams the whole factor block of a large supernode from HBM
// at the bandwidth of one SM; the cluster splits the front's rows (multiples
// of 32 rows per CTA) so that the factor is read by 16 SMs, and moves the
// solved values between CTAs through distributed shared memory. The
// arithmetic is the reference's solve_ldl (include/sparse_ldl.h:1825-1926):
// forward unit-lower solve with the pivot block, D^{-1}, backward solve with
// the transposed block, with the 2x2 pivots' off-diagonal D entry (stored in
// the L slot below the first row of the pair) excluded from the triangular
// sweeps.
//
// Forward, per 32-row pivot tile, one cluster barrier: the tile's owner has
// pushed the solved values to every CTA; the owner of the next tile brings
// that tile's rows up to date, solves it (a warp per right-hand side, the
// factor blocks already in shared memory) and pushes it, while every warp
// updates its other rows. Backward, per tile from the last: every CTA forms
// L(rows below, tile)^T x on its own rows and pushes the partial sums to the
// tile's owner, one cluster barrier, then the owner subtracts them and
// back-substitutes the tile. Both are bound by this chain, not by the bytes
// (plane stress 128 x 128, one right-hand side, 23 such supernodes of up to
// 3,326 rows among 39,679: 6.8 -> 4.7 ms forward, 4.3 -> 2.8 ms backward).
#include <cooperative_groups.h>

#include "ldl_internal.h"
#include "solve_common.cuh"

namespace cg = cooperative_groups;

namespace b200ldl {

namespace {

constexpr int kSbCL = 16;
constexpr int kSbThreads = 256;
constexpr int kSbWarps = kSbThreads / 32;
constexpr int kTileR = 32;
constexpr int kSbRhs = 8;  // right-hand sides per launch
static_assert(4 * kSbWarps == kTileR, "backward: four tile columns per warp");
static_assert(kSbRhs <= kSbWarps, "a warp per right-hand side");

template <typename T>
__device__ __forceinline__ T* at_rank(cg::cluster_group& cl, T* ptr, int r, int rank) {
  return (r == rank) ? ptr : cl.map_shared_rank(ptr, (unsigned)r);
}

// rows per CTA: a multiple of the tile height so that no tile is split
__host__ __device__ __forceinline__ int sb_rows(int f) {
  const int per = (f + kSbCL - 1) / kSbCL;
  return ((per + kTileR - 1) / kTileR) * kTileR;
}

// Bit t of secw[w]: position 32 w + t < npiv is the second row of a 2x2
// pivot. Inside a run of 2x2-marked positions the pairs start at the run's
// first position, so the second rows are the odd offsets into the run.
__device__ void second_row_bits(const int* fv, int npiv, unsigned* secw, int lane) {
  int carry = 0;  // parity of the run length entering the chunk
  for (int w = 0; w * 32 < npiv; w++) {
    const int p = 32 * w + lane;
    const bool neg = p < npiv && fv[p] < 0;
    const unsigned negm = __ballot_sync(0xffffffffu, neg);
    const unsigned nonneg_below = (~negm) & ((1u << lane) - 1u);
    const int ridx = nonneg_below ? lane - 32 + __clz(nonneg_below) : lane + carry;
    const unsigned secm = __ballot_sync(0xffffffffu, neg && (ridx & 1));
    if (lane == 0) secw[w] = secm;
    const int r31 = __shfl_sync(0xffffffffu, ridx, 31);
    carry = ((negm >> 31) & 1u) ? ((r31 + 1) & 1) : 0;
  }
}

__device__ __forceinline__ bool is_second(const unsigned* secw, int p) {
  return (secw[p >> 5] >> (p & 31)) & 1u;
}

// A 32 x 32 block of L, rows [i0, i1), columns [j0, j1): four columns a warp.
constexpr int kTld = kTileR + 1;
struct Part32 {
  double v[kTileR / kSbWarps];
};
__device__ __forceinline__ Part32 get32(const double* L, int ldl, int i0, int i1, int j0, int j1,
                                        int warp, int lane) {
  Part32 t;
#pragma unroll
  for (int u = 0; u < kTileR / kSbWarps; u++) {
    const int j = j0 + warp + kSbWarps * u;
    t.v[u] = (i0 + lane < i1 && j < j1) ? L[(i0 + lane) + (size_t)ldl * j] : 0.0;
  }
  return t;
}
__device__ __forceinline__ void put32(double* tile, const Part32& t, int warp, int lane) {
#pragma unroll
  for (int u = 0; u < kTileR / kSbWarps; u++) tile[(warp + kSbWarps * u) * kTld + lane] = t.v[u];
}

// Doubles of shared memory beside the vectors: the pulled tiles, the factor
// blocks of the forward sweep
template <int kNr>
constexpr int kFwdTiles = 2 * kTileR * kNr + 4 * kTileR * kTld;

template <int kNr>
__global__ void __launch_bounds__(kSbThreads, 1)
    forward_big_kernel(DevPlan p, DevState s, const int* __restrict__ nodes,
                       double* __restrict__ x, int ldx, int nrhs, int r0rhs, int nr,
                       double* __restrict__ upool, int* done, int done_value) {
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int node = nodes[blockIdx.x / kSbCL];
  extern __shared__ __align__(16) double sm[];
  __shared__ ChildBatch kids;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int gt = rank * kSbThreads + tid;
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
  const int R = sb_rows(f);
  const int rb = rank * R;        // first own row
  const int re = min(f, rb + R);  // end of own rows
  double* tb = sm;                                // [2][kTileR][kNr] solved tiles
  double* blk = tb + 2 * kTileR * kNr;            // [2][2][kTileR][kTld] factor blocks
  double* v = blk + 4 * kTileR * kTld;            // [nr][R] own rows, post-pivot order
  int* post_of = reinterpret_cast<int*>(v + (size_t)nr * R);  // [f]
  unsigned* secw = reinterpret_cast<unsigned*>(post_of + f);  // [npiv / 32 + 1]

  for (int q = tid; q < f; q += kSbThreads) post_of[q < fs ? orig[q] : q] = q;
  for (int q = tid; q < nr * R; q += kSbThreads) v[q] = 0.0;
  if (warp == 0) second_row_bits(fv, npiv, secw, lane);
  cl.sync();
  // right-hand side at the supernode's own variables, into the owners' rows
  const int v0 = p.var_ptr[node];
  for (int t = gt; t < ns; t += kSbCL * kSbThreads) {
    const int q = post_of[t];
    const int o = q / R;
    double* dst = at_rank(cl, v, o, rank) + (q - o * R);
    const int var = p.node_to_var[v0 + t];
    for (int r = 0; r < nr; r++) dst[(size_t)r * R] = x[(size_t)ldx * (r0rhs + r) + var];
  }
  cl.sync();
  // children's update vectors, one child at a time (fixed summation order).
  // Every CTA reads each child's entries and adds the ones that land in its
  // own rows, so no two CTAs write a row and a CTA barrier separates the
  // children
  add_children<kNr>(p, s, kids, p.kid_ptr[node], p.kid_ptr[node + 1], ns, nd_in, upool, nrhs,
                    r0rhs, nr, post_of, [&](int q, int r, double u) {
                      if (q >= rb && q < re) v[(size_t)r * R + (q - rb)] += u;
                    });

  // unit-lower solve, tile by tile
  const int ntile = (npiv + kTileR - 1) / kTileR;
  auto owner = [&](int b) { return b * kTileR / R; };
  auto end_of = [&](int b) { return min((b + 1) * kTileR, npiv); };
  // the block of L beside tile b and above it (rows of tile b, columns of the
  // tile before) and its diagonal block, into buffer b & 1
  auto fetch = [&](int b, Part32& side, Part32& diag) {
    const int jb = b * kTileR, je = end_of(b);
    if (b > 0) side = get32(L, ldl, jb, je, jb - kTileR, jb, warp, lane);
    diag = get32(L, ldl, jb, je, jb, je, warp, lane);
  };
  auto store = [&](int b, const Part32& side, const Part32& diag) {
    double* t = blk + (b & 1) * 2 * kTileR * kTld;
    if (b > 0) put32(t, side, warp, lane);
    put32(t + kTileR * kTld, diag, warp, lane);
  };
  // warp r < nr of the owner: right-hand side r of tile b minus the tile
  // before, solved, and pushed to every CTA
  auto solve_tile = [&](int b) {
    const int jb = b * kTileR, nb = end_of(b) - jb;
    const double* side = blk + (b & 1) * 2 * kTileR * kTld;
    const double* diag = side + kTileR * kTld;
    const bool mine = lane < nb;
    double* vrow = v + (size_t)warp * R + (jb - rb) + lane;
    double vr = mine ? *vrow : 0.0;
    if (b > 0) {
      const double* t = tb + ((b - 1) & 1) * kTileR * kNr + warp;
      // a 2x2 pair across the boundary: its D slot is not an entry of L
      const bool cut = is_second(secw, jb) && lane == 0;
      double acc = 0.0;
#pragma unroll
      for (int j = 0; j < kTileR; j++) {
        const double l = (cut && j == kTileR - 1) ? 0.0 : side[j * kTld + lane];
        acc = fma(l, t[j * kNr], acc);
      }
      vr -= acc;
    }
    const unsigned sec = secw[jb >> 5];  // tiles are 32-aligned
    double Lrow[kTileR];
#pragma unroll
    for (int j = 0; j < kTileR; j++) Lrow[j] = diag[j * kTld + lane];
#pragma unroll
    for (int j = 0; j < kTileR; j++) {
      if (j < nb) {
        // the L slot below the first row of a 2x2 pair holds D, not L
        const bool skip = (j + 1 < kTileR) && ((sec >> (j + 1)) & 1u) && lane == j + 1;
        const bool upd = lane > j && !skip;
        const double vj = __shfl_sync(0xffffffffu, vr, j);
        if (upd) vr = fma(-Lrow[j], vj, vr);
      }
    }
    if (mine) *vrow = vr;
    double* t = tb + (b & 1) * kTileR * kNr + lane * kNr + warp;
    for (int d = 0; d < kSbCL; d++) *at_rank(cl, t, d, rank) = mine ? vr : 0.0;
  };
  // first of a CTA's rows below tile b that it updates in the common pass
  // (the next tile's owner has dealt with that tile's rows)
  auto first_row = [&](int b) {
    const int je = end_of(b);
    if (b + 1 < ntile && rank == owner(b + 1)) return end_of(b + 1);
    return max(je, rb);
  };
  // a tile's entries of this thread's first row: loaded a tile ahead (they do
  // not depend on the solved values)
  double lvn[kTileR];
  auto prefetch = [&](int b) {
    const int jb = b * kTileR, je = end_of(b);
    const int i = first_row(b) + tid;
    const double* li = L + i + (size_t)ldl * jb;
#pragma unroll
    for (int j = 0; j < kTileR; j++) lvn[j] = (i < re && jb + j < je) ? li[(size_t)ldl * j] : 0.0;
  };
  if (ntile > 0) {
    Part32 side, diag;
    if (rank == owner(0)) {
      fetch(0, side, diag);
      store(0, side, diag);
    }
    if (ntile > 1 && rank == owner(1)) {
      fetch(1, side, diag);
      store(1, side, diag);
    }
    prefetch(0);
    __syncthreads();
    if (rank == owner(0) && warp < nr) solve_tile(0);
  }
  for (int b = 0; b < ntile; b++) {
    const int jb = b * kTileR;
    const int je = end_of(b);
    const int nb = je - jb;
    cl.sync();  // the tile's solved values are in every CTA
    if (b + 1 < ntile && rank == owner(b + 1) && warp < nr) solve_tile(b + 1);
    // the blocks of the tile after, while the rows are updated
    Part32 side, diag;
    const bool ahead = b + 2 < ntile && rank == owner(b + 2);
    if (ahead) fetch(b + 2, side, diag);
    const double* t = tb + (b & 1) * kTileR * kNr;
    // a 2x2 pair across the tile boundary: its D slot (je, je - 1) is skipped
    const int skip_i = (je < npiv && is_second(secw, je)) ? je : -1;
    const int i0 = first_row(b) + tid;
    double lv[kTileR];
#pragma unroll
    for (int j = 0; j < kTileR; j++) lv[j] = lvn[j];
    if (b + 1 < ntile) prefetch(b + 1);
    for (int i = i0; i < re; i += kSbThreads) {
      if (i != i0) {
        const double* li = L + i + (size_t)ldl * jb;
#pragma unroll
        for (int j = 0; j < kTileR; j++) lv[j] = (j < nb) ? li[(size_t)ldl * j] : 0.0;
      }
      double acc[kNr];
#pragma unroll
      for (int r = 0; r < kNr; r++) acc[r] = 0.0;
#pragma unroll
      for (int j = 0; j < kTileR; j++) {
        const double l = (i == skip_i && j == nb - 1) ? 0.0 : lv[j];
#pragma unroll
        for (int r = 0; r < kNr; r++) acc[r] = fma(l, t[j * kNr + r], acc[r]);
      }
#pragma unroll
      for (int r = 0; r < kNr; r++)
        if (r < nr) v[(size_t)r * R + (i - rb)] -= acc[r];
    }
    // buffer b & 1 was last read for tile b, before this step's barrier
    if (ahead) store(b + 2, side, diag);
  }
  cl.sync();

  // D^{-1} at the pivots (a 2x2 pair reads its partner, possibly in another
  // CTA), the solution at the pivot variables; the rest is the update vector
  for (int i = rb + tid; i < min(re, npiv); i += kSbThreads) {
    const bool sec = is_second(secw, i);
    const bool first = (i + 1 < npiv) && is_second(secw, i + 1);
    const int var = fv[i];
    const int vi = var >= 0 ? var : -var - 1;
    const double dd = L[i + (size_t)ldl * i];
    int pp = -1;
    double d11 = 0.0, d21 = 0.0, d22 = 0.0;
    if (first) {
      pp = i + 1;
      d11 = dd;
      d21 = L[(i + 1) + (size_t)ldl * i];
      d22 = L[(i + 1) + (size_t)ldl * (i + 1)];
    } else if (sec) {
      pp = i - 1;
      d11 = L[(i - 1) + (size_t)ldl * (i - 1)];
      d21 = L[i + (size_t)ldl * (i - 1)];
      d22 = dd;
    }
    const double* vp = nullptr;
    if (pp >= 0) {
      const int op = pp / R;
      vp = at_rank(cl, v, op, rank) + (pp - op * R);
    }
    for (int r = 0; r < nr; r++) {
      const double t = v[(size_t)r * R + (i - rb)];
      double y;
      if (first) {
        const double u = vp[(size_t)r * R];
        y = (d22 * t - d21 * u) / (d11 * d22 - d21 * d21);
      } else if (sec) {
        const double u = vp[(size_t)r * R];
        y = (d11 * t - d21 * u) / (d11 * d22 - d21 * d21);
      } else {
        y = t / dd;
      }
      x[(size_t)ldx * (r0rhs + r) + vi] = y;
    }
  }
  double* uo = upool + s.u_off[node] * nrhs + (size_t)r0rhs * m;
  for (int i = max(rb, npiv) + tid; i < re; i += kSbThreads)
    for (int r = 0; r < nr; r++) uo[(size_t)r * m + (i - npiv)] = v[(size_t)r * R + (i - rb)];
  cl.sync();  // partners read through DSMEM are done
  if (rank == 0 && tid == 0) done[node] = done_value;  // for the launches that follow
}

template <int kNr>
__global__ void __launch_bounds__(kSbThreads)
    backward_big_kernel(DevPlan p, DevState s, const int* __restrict__ nodes,
                        double* __restrict__ x, int ldx, int r0rhs, int nr, int* done,
                        int done_value) {
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int node = nodes[blockIdx.x / kSbCL];
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int f = s.f[node];
  const int npiv = s.npiv[node];
  const int* fv = s.ivars + s.fv_off[node];
  const double* L = s.dpool + s.L_off[node];
  const int ldl = s.L_ld[node];
  const int R = sb_rows(f);
  const int rb = rank * R;
  const int re = min(f, rb + R);
  double* diag = sm;                                 // [2][kTileR][kTld] diagonal blocks
  double* part = diag + 2 * kTileR * kTld;           // [2][kSbCL][kTileR][kNr]
  double* v = part + 2 * kSbCL * kTileR * kNr;       // [nr][R]
  unsigned* secw = reinterpret_cast<unsigned*>(v + (size_t)nr * R);

  for (int q = tid; q < nr * R; q += kSbThreads) {
    const int r = q / R;
    const int i = rb + (q - r * R);
    double val = 0.0;
    if (i < re) {
      const int var = fv[i];
      val = x[(size_t)ldx * (r0rhs + r) + (var >= 0 ? var : -var - 1)];
    }
    v[q] = val;
  }
  if (warp == 0) second_row_bits(fv, npiv, secw, lane);

  const int ntile = (npiv + kTileR - 1) / kTileR;
  auto owner = [&](int b) { return b * kTileR / R; };
  auto end_of = [&](int b) { return min((b + 1) * kTileR, npiv); };
  // the first 128 of this CTA's rows below tile b, warp w's columns
  // 4 w .. 4 w + 3: loaded a tile ahead
  const int j0 = 4 * warp;
  double nx[4][4];
  auto load_rows = [&](int b, int ib, double (&lv)[4][4]) {
    const int jb = b * kTileR, je = end_of(b), nb = je - jb;
    const int skip_i = (je < npiv && is_second(secw, je)) ? je : -1;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = ib + 32 * u;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int j = j0 + c;
        lv[u][c] = (i < re && j < nb && !(i == skip_i && j == nb - 1))
                       ? L[i + (size_t)ldl * (jb + j)]
                       : 0.0;
      }
    }
  };
  __syncthreads();
  if (ntile > 0) {
    const int b = ntile - 1;
    if (rank == owner(b))
      put32(diag + (b & 1) * kTileR * kTld,
            get32(L, ldl, b * kTileR, end_of(b), b * kTileR, end_of(b), warp, lane), warp, lane);
    load_rows(b, max(end_of(b), rb) + lane, nx);
  }
  cl.sync();  // every CTA has started: the partial sums go to another's memory
  for (int b = ntile - 1; b >= 0; b--) {
    const int jb = b * kTileR;
    const int je = end_of(b);
    const int nb = je - jb;
    const int ob = owner(b);
    const int par = b & 1;
    // partial sums of L(i, j) x(i) over own rows i >= je
    {
      double acc[4 * kNr];
#pragma unroll
      for (int q = 0; q < 4 * kNr; q++) acc[q] = 0.0;
      const int ib0 = max(je, rb) + lane;
      for (int ib = ib0; ib < re; ib += 128) {
        double lv[4][4];
        if (ib == ib0) {
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int c = 0; c < 4; c++) lv[u][c] = nx[u][c];
        } else {
          load_rows(b, ib, lv);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int i = ib + 32 * u;
          if (i < re) {
#pragma unroll
            for (int r = 0; r < kNr; r++) {
              const double xr = (r < nr) ? v[(size_t)r * R + (i - rb)] : 0.0;
#pragma unroll
              for (int c = 0; c < 4; c++) acc[c * kNr + r] = fma(lv[u][c], xr, acc[c * kNr + r]);
            }
          }
        }
      }
      __syncwarp();
      // the next tile's rows, while the sums are formed and sent
      Part32 dn;
      const bool ahead = b > 0 && rank == owner(b - 1);
      if (ahead) dn = get32(L, ldl, jb - kTileR, jb, jb - kTileR, jb, warp, lane);
      if (b > 0) load_rows(b - 1, max(jb, rb) + lane, nx);
      // with every halving of the warp a lane keeps half of the sums, whose
      // pairs of lanes are those of a butterfly
      int o = 16;
#pragma unroll
      for (int n = 2 * kNr; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; i++) {
          const double keep = up ? acc[i + n] : acc[i];
          const double send = up ? acc[i] : acc[i + n];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      double sum = acc[0];
#pragma unroll
      for (; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      constexpr int kLanes = 32 / (4 * kNr);
      if (lane % kLanes == 0) {
        const int q = lane / kLanes, c = q / kNr, r = q % kNr;
        double* dst = at_rank(cl, part, ob, rank);
        dst[((size_t)(par * kSbCL + rank) * kTileR + (j0 + c)) * kNr + r] = sum;
      }
      if (ahead) put32(diag + ((b - 1) & 1) * kTileR * kTld, dn, warp, lane);
    }
    cl.sync();  // partials at the owner
    if (rank == ob && warp < nr) {
      // right-hand side `warp` of the tile
      const bool mine = lane < nb;
      const unsigned sec = secw[jb >> 5];
      const double* tile = diag + par * kTileR * kTld;
      double Lcol[kTileR];
#pragma unroll
      for (int q = 0; q < kTileR; q++) Lcol[q] = tile[lane * kTld + q];
      double* vrow = v + (size_t)warp * R + (jb - rb) + lane;
      double vr = 0.0;
      if (mine) {
        vr = *vrow;
        const double* pp = part + ((size_t)par * kSbCL * kTileR + lane) * kNr + warp;
        double t[kSbCL];
#pragma unroll
        for (int c = 0; c < kSbCL; c++) t[c] = pp[(size_t)c * kTileR * kNr];
#pragma unroll
        for (int c = 0; c < kSbCL; c++) vr -= t[c];
      }
      __syncwarp();
#pragma unroll
      for (int jj = kTileR - 1; jj >= 0; jj--) {
        if (jj < nb) {
          const bool upd = lane < jj && !(((sec >> jj) & 1u) && lane == jj - 1);
          const double vj = __shfl_sync(0xffffffffu, vr, jj);
          if (upd) vr = fma(-Lcol[jj], vj, vr);
        }
      }
      if (mine) *vrow = vr;
    }
    __syncthreads();
  }
  for (int q = tid; q < nr * R; q += kSbThreads) {
    const int r = q / R;
    const int i = rb + (q - r * R);
    if (i < min(re, npiv)) {
      const int var = fv[i];
      x[(size_t)ldx * (r0rhs + r) + (var >= 0 ? var : -var - 1)] = v[q];
    }
  }
  cl.sync();
  if (rank == 0 && tid == 0) done[node] = done_value;
}

size_t fwd_big_smem(int fmax, int kn) {
  const size_t R = (size_t)sb_rows(fmax);
  const size_t tiles = kn == 1 ? kFwdTiles<1> : kn == 2 ? kFwdTiles<2> : kn == 4 ? kFwdTiles<4>
                                                                                  : kFwdTiles<8>;
  return (R * kn + tiles) * sizeof(double) + (size_t)fmax * sizeof(int) +
         ((size_t)fmax / 32 + 2) * sizeof(unsigned) + 16;
}

size_t bwd_big_smem(int fmax, int kn) {
  const size_t R = (size_t)sb_rows(fmax);
  return (R * kn + 2 * kTileR * kTld + (size_t)2 * kSbCL * kTileR * kn) * sizeof(double) +
         ((size_t)fmax / 32 + 2) * sizeof(unsigned) + 16;
}

// the kernels' number of right-hand sides for nr of them
int big_rhs(int nr) { return nr <= 2 ? nr : nr <= 4 ? 4 : 8; }

cudaLaunchConfig_t cluster_cfg(int count, size_t smem, cudaStream_t st, cudaLaunchAttribute* a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(count * kSbCL, 1, 1);
  cfg.blockDim = dim3(kSbThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  a[0].id = cudaLaunchAttributeClusterDimension;
  a[0].val.clusterDim.x = kSbCL;
  a[0].val.clusterDim.y = 1;
  a[0].val.clusterDim.z = 1;
  cfg.attrs = a;
  cfg.numAttrs = 1;
  return cfg;
}

constexpr size_t kSbSmemMax = 200 * 1024;

}  // namespace

int solve_big_rhs(int f) {
  int kn = kSbRhs;
  while (kn > 0 && (fwd_big_smem(f, kn) > kSbSmemMax || bwd_big_smem(f, kn) > kSbSmemMax)) kn /= 2;
  return kn;
}

cudaError_t configure_solve_big_kernels() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* k) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSbSmemMax);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  };
  set(forward_big_kernel<1>);
  set(forward_big_kernel<2>);
  set(forward_big_kernel<4>);
  set(forward_big_kernel<8>);
  set(backward_big_kernel<1>);
  set(backward_big_kernel<2>);
  set(backward_big_kernel<4>);
  set(backward_big_kernel<8>);
  return e;
}

cudaError_t launch_forward_big(const DevPlan& p, const DevState& s, const SolveSpan& sp, double* x,
                               int ldx, int nrhs, int r0, int nr, double* upool,
                               cudaStream_t stream) {
  if (sp.count <= 0) return cudaSuccess;
  const int kn = big_rhs(nr);
  cudaLaunchAttribute a[1];
  cudaLaunchConfig_t cfg = cluster_cfg(sp.count, fwd_big_smem(sp.fmax, kn), stream, a);
  auto* k = kn == 1 ? forward_big_kernel<1> : kn == 2 ? forward_big_kernel<2>
          : kn == 4 ? forward_big_kernel<4> : forward_big_kernel<8>;
  return cudaLaunchKernelEx(&cfg, k, p, s, sp.nodes, x, ldx, nrhs, r0, nr, upool, sp.fdone,
                            2 * sp.epoch + 1);
}

cudaError_t launch_backward_big(const DevPlan& p, const DevState& s, const SolveSpan& sp,
                                double* x, int ldx, int r0, int nr, cudaStream_t stream) {
  if (sp.count <= 0) return cudaSuccess;
  const int kn = big_rhs(nr);
  cudaLaunchAttribute a[1];
  cudaLaunchConfig_t cfg = cluster_cfg(sp.count, bwd_big_smem(sp.fmax, kn), stream, a);
  auto* k = kn == 1 ? backward_big_kernel<1> : kn == 2 ? backward_big_kernel<2>
          : kn == 4 ? backward_big_kernel<4> : backward_big_kernel<8>;
  return cudaLaunchKernelEx(&cfg, k, p, s, sp.nodes, x, ldx, r0, nr, sp.bdone, 2 * sp.epoch + 1);
}

}  // namespace b200ldl
