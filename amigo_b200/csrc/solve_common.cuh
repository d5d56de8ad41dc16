// Pieces shared by the one-CTA and the cluster solves.
#pragma once

#include "ldl_internal.h"

namespace b200ldl {

// A batch of children of one supernode, in shared memory.
constexpr int kChildBatch = 32;
struct ChildBatch {
  int mc[kChildBatch];   // rows of the update vector
  int nd[kChildBatch];   // of which delayed candidates
  int off[kChildBatch];  // first position of those in the parent
  int cptr[kChildBatch];
  long long u[kChildBatch];
  int next_off;
};

// Adds the update vectors of the children kids[kb, ke) to the front's rows,
// one child after another (fixed summation order), by the whole CTA:
// add(row in post-pivot order, right-hand side, value). A child costs a
// barrier and an addition; what it takes to find and read its vector is done
// for kAhead children at once (one after another the chain of global loads
// took 1,500 cycles a child, and the large fronts have up to 256).
template <int kNr, typename Add>
__device__ __forceinline__ void add_children(const DevPlan& p, const DevState& s, ChildBatch& kids,
                                             int kb, int ke, int ns, int nd_in,
                                             const double* upool, int nrhs, int r0, int nr,
                                             const int* post_of, Add add) {
  constexpr int kAhead = kNr >= 8 ? 2 : 4;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int nt = blockDim.x;
  if (tid == 0) kids.next_off = ns;
  for (int c0 = kb; c0 < ke; c0 += kChildBatch) {
    const int n = min(kChildBatch, ke - c0);
    __syncthreads();
    if (tid < 32) {
      int nd = 0;
      if (lane < n) {
        const int ch = p.kids[c0 + lane];
        nd = s.ndel[ch];
        kids.nd[lane] = nd;
        kids.mc[lane] = s.f[ch] - s.npiv[ch];
        kids.u[lane] = s.u_off[ch];
        kids.cptr[lane] = p.cptr[ch];
      }
      int incl = nd;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const int base = kids.next_off;
      if (lane < n) kids.off[lane] = base + incl - nd;
      __syncwarp();
      if (lane == 31) kids.next_off = base + incl;
    }
    __syncthreads();
    auto row = [&](int c, int t) {
      const int nd = kids.nd[c];
      int q;
      if (t < nd) {
        q = kids.off[c] + t;
      } else {
        q = p.cmap[kids.cptr[c] + t - nd];
        if (q >= ns) q += nd_in;
      }
      return q;
    };
    for (int g = 0; g < n; g += kAhead) {
      int q[kAhead];
      double u[kAhead][kNr];
#pragma unroll
      for (int a = 0; a < kAhead; a++) {
        const int c = g + a;
        const bool on = c < n && tid < kids.mc[c];
        q[a] = on ? row(c, tid) : -1;
        const double* uc = on ? upool + kids.u[c] * nrhs + (size_t)r0 * kids.mc[c] + tid : nullptr;
#pragma unroll
        for (int r = 0; r < kNr; r++)
          u[a][r] = (on && r < nr) ? __ldcg(uc + (size_t)r * kids.mc[c]) : 0.0;
      }
#pragma unroll
      for (int a = 0; a < kAhead; a++) {
        const int c = g + a;
        if (c >= n) break;
        if (q[a] >= 0) {
          const int at = post_of[q[a]];
#pragma unroll
          for (int r = 0; r < kNr; r++)
            if (r < nr) add(at, r, u[a][r]);
        }
        // rows beyond one per thread
        const int mc = kids.mc[c];
        for (int t = tid + nt; t < mc; t += nt) {
          const double* uc = upool + kids.u[c] * nrhs + (size_t)r0 * mc + t;
          double w[kNr];
#pragma unroll
          for (int r = 0; r < kNr; r++) w[r] = r < nr ? __ldcg(uc + (size_t)r * mc) : 0.0;
          const int at = post_of[row(c, t)];
#pragma unroll
          for (int r = 0; r < kNr; r++)
            if (r < nr) add(at, r, w[r]);
        }
        __syncthreads();
      }
    }
  }
}

}  // namespace b200ldl
