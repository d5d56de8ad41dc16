// The register fronts (amigo_b200/csrc/register_front.cuh) compiled for the
// host: the 256 threads of the CTA as fibers that a scheduler runs warp by
// warp, in an order drawn from a seed in which some warps run as far ahead as
// the barriers let them. A result that depends on the order is a race. The
// same factorization, written as plain loops, says what the result is.
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <random>
#include <vector>

using std::max;
using std::min;

static struct {
  int x;
} threadIdx;

namespace sim {

constexpr int kThreads = 256, kLanes = 32, kWarps = kThreads / kLanes;
enum State { kRun, kWarp, kBar, kDone };

struct Fiber {
  ucontext_t ctx;
  std::vector<char> stack;
  State state = kRun;
  int bar = -1;
  unsigned parity = 0;
};

struct Sim {
  Fiber fib[kThreads];
  ucontext_t home;
  uint64_t slot[2][kThreads];
  int arrived[3];
  char seen[3][kThreads];
  const char* error = nullptr;
  std::function<void()> body;
};
static Sim* g = nullptr;

static void yield() { swapcontext(&g->fib[threadIdx.x].ctx, &g->home); }

static void arrive(int id) {
  if (g->seen[id][threadIdx.x]) g->error = "a thread arrived twice at one barrier";
  g->seen[id][threadIdx.x] = 1;
  if (++g->arrived[id] == kThreads) {
    g->arrived[id] = 0;
    std::memset(g->seen[id], 0, kThreads);
    for (auto& f : g->fib)
      if (f.state == kBar && f.bar == id) f.state = kRun;
  }
}

static void wait(int id) {
  const int before = g->arrived[id];
  Fiber& f = g->fib[threadIdx.x];
  f.state = kBar;
  f.bar = id;
  arrive(id);
  (void)before;
  if (f.state == kBar) yield();
}

// the warp's values of v, by lane
static const uint64_t* exchange(uint64_t v) {
  const int t = threadIdx.x;
  Fiber& f = g->fib[t];
  const unsigned q = f.parity++ & 1;
  g->slot[q][t] = v;
  f.state = kWarp;
  yield();
  return g->slot[q] + (t / kLanes) * kLanes;
}

static void entry(int t) {
  threadIdx.x = t;
  g->body();
  g->fib[t].state = kDone;
  yield();
}

// Runs body on every thread; how: 0 = the warps in turn, else a seed.
static const char* run(Sim& s, unsigned how) {
  g = &s;
  std::mt19937 rng(how);
  std::memset(s.arrived, 0, sizeof(s.arrived));
  std::memset(s.seen, 0, sizeof(s.seen));
  for (int t = 0; t < kThreads; t++) {
    Fiber& f = s.fib[t];
    f.stack.resize(96 * 1024);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.data();
    f.ctx.uc_stack.ss_size = f.stack.size();
    f.ctx.uc_link = &s.home;
    makecontext(&f.ctx, reinterpret_cast<void (*)()>(entry), 1, t);
  }
  std::vector<int> rank(kWarps);
  for (int w = 0; w < kWarps; w++) rank[w] = w;
  int left = 0, last = 0;
  while (!s.error) {
    if (how && left-- <= 0) {
      std::shuffle(rank.begin(), rank.end(), rng);
      left = 1 + (int)(rng() % 400);
    }
    int pick = -1;
    bool done = true;
    for (int q = 0; q < kWarps; q++) {
      const int w = how ? rank[q] : (last + 1 + q) % kWarps;
      bool runnable = false;
      for (int l = 0; l < kLanes; l++) {
        const State st = s.fib[w * kLanes + l].state;
        runnable = runnable || st == kRun;
        done = done && st == kDone;
      }
      if (runnable && pick < 0) pick = w;
    }
    if (done) break;
    if (pick < 0) return "every warp waits";
    last = pick;
    const bool back = how && (rng() & 1);
    for (int q = 0; q < kLanes; q++) {
      const int t = pick * kLanes + (back ? kLanes - 1 - q : q);
      if (s.fib[t].state != kRun) continue;
      threadIdx.x = t;
      swapcontext(&s.home, &s.fib[t].ctx);
    }
    int at = 0;
    for (int l = 0; l < kLanes; l++) at += s.fib[pick * kLanes + l].state == kWarp;
    if (at == kLanes)
      for (int l = 0; l < kLanes; l++) s.fib[pick * kLanes + l].state = kRun;
  }
  return s.error;
}

}  // namespace sim

// what the header uses of CUDA
static double bits(uint64_t u) {
  double d;
  std::memcpy(&d, &u, 8);
  return d;
}
static uint64_t bits(double d) {
  uint64_t u;
  std::memcpy(&u, &d, 8);
  return u;
}
static int __double2hiint(double d) { return (int)(bits(d) >> 32); }
static double __hiloint2double(int hi, int lo) {
  return bits((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo);
}
static long long __double_as_longlong(double d) { return (long long)bits(d); }
static double __longlong_as_double(long long u) { return bits((uint64_t)u); }
static double __dmul_rn(double a, double b) { return a * b; }
static int atomicOr(int* p, int v) {  // named by the header, not used here
  const int old = *p;
  *p |= v;
  return old;
}
static void __syncwarp() { sim::exchange(0); }
static void __syncthreads() { sim::wait(0); }
static int __all_sync(unsigned, int v) {
  const uint64_t* x = sim::exchange(v != 0);
  return (int)*std::min_element(x, x + 32);
}
static unsigned __reduce_max_sync(unsigned, unsigned v) {
  const uint64_t* x = sim::exchange(v);
  return (unsigned)*std::max_element(x, x + 32);
}
static int __reduce_min_sync(unsigned, int v) {
  const uint64_t* x = sim::exchange((uint64_t)(int64_t)v);
  int m = v;
  for (int l = 0; l < 32; l++) m = std::min(m, (int)(int64_t)x[l]);
  return m;
}
static int __reduce_add_sync(unsigned, int v) {
  const uint64_t* x = sim::exchange((uint64_t)(int64_t)v);
  int m = 0;
  for (int l = 0; l < 32; l++) m += (int)(int64_t)x[l];
  return m;
}
static void bar_arrive(int odd) {
  __syncwarp();
  sim::arrive(1 + odd);
}
static void bar_wait(int odd) {
  __syncwarp();
  sim::wait(1 + odd);
}

#include "register_front.cuh"

using namespace b200ldl;

// The factorization as plain loops: F is f x f, lower triangle; L and the
// trailing matrix are left in place.
static Result plain(double* F, int f, int fs, bool root, const FactorParams& prm, int* fv,
                    int* orig) {
  auto at = [&](int i, int j) -> double& { return i >= j ? F[i + f * j] : F[j + f * i]; };
  auto swap = [&](int a, int b) {
    if (a == b) return;
    std::swap(at(a, a), at(b, b));
    for (int j = 0; j < f; j++)
      if (j != a && j != b) std::swap(at(a, j), at(b, j));
    std::swap(fv[a], fv[b]);
    std::swap(orig[a], orig[b]);
  };
  Result o = {0, 0, 0, 0};
  int k = 0, ncand = fs;
  while (k < ncand) {
    int step = kOne, kpiv = k;
    const double d = at(k, k);
    if (!prm.cholesky) {
      const bool has = k + 1 < ncand;
      double bv = -1.0, cm = 0.0;
      int bi = INT_MAX;
      for (int i = k + 1; i < f; i++) {
        const double x = std::fabs(at(i, k));
        if (i < ncand) {
          if (x > bv) bv = x, bi = i;
        } else {
          cm = std::fmax(cm, x);
        }
      }
      const double abswik = has ? bv : 0.0;
      const int imax = has ? (bi < ncand ? bi : k + 1) : k;
      const double colmax = std::fmax(abswik, cm);
      const double absd = std::fabs(d);
      if (root)
        step = std::fmax(absd, colmax) == 0.0 ? kZero : absd >= kAlphaBK * colmax ? kOne : kNeedRow;
      else if (absd >= prm.pivot_tol && absd >= prm.ustab * colmax)
        step = kOne;
      else
        step = has ? kNeedRow : kDelay;
      if (step == kNeedRow) {
        double rmax = 0.0;
        for (int i = k; i < f; i++)
          if (i != imax) rmax = std::fmax(rmax, std::fabs(at(imax, i)));
        const double wii = at(imax, imax), abswii = std::fabs(wii), wik = at(imax, k);
        if (root) {
          if (absd >= kAlphaBK * colmax * (colmax / rmax))
            step = kOne;
          else
            step = abswii >= kAlphaBK * rmax ? kOne : kTwo, kpiv = imax;
        } else if (abswii >= prm.pivot_tol && abswii >= prm.ustab * rmax) {
          step = kOne;
          kpiv = imax;
        } else {
          const double det = std::fabs(std::fma(d, wii, -(wik * wik)));
          const double delta = det / std::fmax(abswii + abswik, absd + abswik);
          if (det >= prm.pivot_tol && delta >= prm.ustab * colmax && delta >= prm.ustab * rmax)
            step = kTwo, kpiv = imax;
          else
            step = kDelay;
        }
      }
    }
    if (step == kDelay) {
      swap(k, --ncand);
      continue;
    }
    if (step != kTwo) {
      swap(k, kpiv);
      const double p = at(k, k);
      const double r = step == kZero || (root && p == 0.0) ? 0.0 : 1.0 / p;
      for (int j = k + 1; j < f; j++) {
        const double l = at(j, k) * r;
        for (int i = j; i < f; i++) at(i, j) = std::fma(-at(i, k), l, at(i, j));
      }
      for (int i = k + 1; i < f; i++) at(i, k) *= r;
      p >= 0.0 ? o.npos++ : o.nneg++;
      const long long m = f - k - 1;
      o.flops += m * (m + 1) + m;
      k++;
      continue;
    }
    swap(k + 1, kpiv);
    const double d11 = at(k, k), d21 = at(k + 1, k), d22 = at(k + 1, k + 1);
    const double det = std::fma(d11, d22, -(d21 * d21)), di = 1.0 / det;
    const double i00 = d22 * di, i01 = -d21 * di, i11 = d11 * di;
    auto l0 = [&](int i) { return std::fma(at(i, k), i00, at(i, k + 1) * i01); };
    auto l1 = [&](int i) { return std::fma(at(i, k), i01, at(i, k + 1) * i11); };
    for (int j = k + 2; j < f; j++)
      for (int i = j; i < f; i++)
        at(i, j) -= std::fma(at(i, k), l0(j), at(i, k + 1) * l1(j));
    for (int i = k + 2; i < f; i++) {
      const double x = l0(i), y = l1(i);
      at(i, k) = x;
      at(i, k + 1) = y;
    }
    fv[k] = -(fv[k] + 1);
    fv[k + 1] = -(fv[k + 1] + 1);
    if (det >= 0.0)
      (d11 >= 0.0 ? o.npos : o.nneg) += 2;
    else
      o.npos++, o.nneg++;
    const long long m = f - k - 2;
    o.flops += 2 * m * (m + 1) + 6 * m;
    k += 2;
  }
  o.npiv = k;
  return o;
}

template <int kR>
static Result registers(const Front& a, bool root, const FactorParams& prm, double* out, int f) {
  int npiv = 0;
  auto write = [&](const Result& o) {
    // the CTA's barrier before the factor columns are read
    __syncthreads();
    if (threadIdx.x == 0) {
      npiv = o.npiv;
      for (int j = 0; j < npiv; j++)
        for (int i = j; i < f; i++) out[i + f * j] = a.F[i + a.ld * j];
    }
  };
  auto store = [&](int i, int j, double x) { out[i + f * j] = x; };
  return factor_front<kR>(a, root, prm, write, store);
}

// a: f x f, lower triangle. 0 if the schedules `first` .. `first + count - 1`
// (0: warps in turn) all give the plain loops' result; else 1 + the schedule.
extern "C" int front_schedules(int chunks, int f, int fs, int root, int cholesky, double ustab,
                               double tol, const double* a, unsigned first, unsigned count,
                               int* result, char* why, int whylen) {
  FactorParams prm{};
  prm.ustab = ustab;
  prm.pivot_tol = tol;
  prm.cholesky = cholesky;
  const int ld = f | 1, len = 32 * chunks + 2, guard = 16;
  std::vector<double> want(a, a + (size_t)f * f);
  std::vector<int> wv(f), wo(f);
  for (int i = 0; i < f; i++) wv[i] = 7 * i, wo[i] = i;
  const Result w = plain(want.data(), f, fs, root, prm, wv.data(), wo.data());
  result[0] = w.npiv;
  result[1] = w.npos;
  result[2] = w.nneg;
  int two = 0;
  for (int i = 0; i < f; i++) two += wv[i] < 0;
  result[3] = two / 2;
  result[4] = 0;
  for (int i = 0; i < f; i++) result[4] += wo[i] != i;
  const double nan = std::nan("");
  for (unsigned how = first; how < first + count; how++) {
    std::vector<double> mem((size_t)ld * f + kVecs * len + 2 * guard, nan);
    std::vector<double> got((size_t)f * f, 0.0);
    std::vector<int> fv(f), orig(f);
    Front fr;
    fr.F = mem.data() + guard;
    fr.vec = fr.F + (size_t)ld * f;
    fr.fv = fv.data();
    fr.orig = orig.data();
    fr.f = f;
    fr.fs = fs;
    fr.ld = ld;
    for (int j = 0; j < f; j++)
      for (int i = j; i < f; i++) fr.F[i + ld * j] = a[i + (size_t)f * j];
    for (int i = 0; i < f; i++) fv[i] = 7 * i, orig[i] = i;
    Result r{};
    sim::Sim s;
    s.body = [&] {
      const Result q = chunks == 1   ? registers<1>(fr, root, prm, got.data(), f)
                       : chunks == 2 ? registers<2>(fr, root, prm, got.data(), f)
                       : chunks == 3 ? registers<3>(fr, root, prm, got.data(), f)
                                     : registers<5>(fr, root, prm, got.data(), f);
      if (threadIdx.x == 0) r = q;
    };
    const char* bad = sim::run(s, how);
    const double* end = fr.vec + kVecs * len;
    for (int i = 0; i < guard && !bad; i++)
      if (!std::isnan(mem[i]) || !std::isnan(end[i])) bad = "a write out of range";
    if (!bad && (r.npiv != w.npiv || r.npos != w.npos || r.nneg != w.nneg || r.flops != w.flops))
      bad = "counts differ";
    if (!bad && (fv != wv || orig != wo)) bad = "pivot order differs";
    for (int j = 0; j < f && !bad; j++)
      for (int i = j; i < f && !bad; i++) {
        const double x = got[i + f * j], y = want[i + f * j];
        if (!(x == y || (std::isnan(x) && std::isnan(y)))) bad = "entries differ";
      }
    if (bad) {
      std::snprintf(why, whylen, "%s", bad);
      return 1 + (int)how;
    }
  }
  return 0;
}
