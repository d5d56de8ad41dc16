// KKT assembly: element Hessian blocks into the values of the fixed CSR
// pattern, on the device, deterministically.
//
// The reference zeroes the matrix and, for each component group in turn,
// each element in turn and each column j of the element's Hessian, adds
// the column into CSR row conn[e][j] at the columns conn[e][i], dropping
// entries outside the pattern (OptimizationProblem::hessian,
// include/optimization_problem.h:1063-1088; ComponentGroup::
// add_hessian_kernel, include/component_group.h:144-162; CSRMat::add_row,
// include/csr_matrix.h:554-567). Its GPU backend scatters the same values
// with atomicAdd through a per-entry position table
// (include/cuda/component_group_backend.cuh:157-190), so its sums come in
// an order that changes from run to run.
//
// Here the scatter is inverted once per pattern on the host: for every CSR
// entry, the positions of its contributions in the concatenated element
// blocks, in the reference's sequential order (group, element, j, i). The
// kernel then gathers: one thread per CSR entry, summing from zero in that
// order, so the values are bit-identical to the reference's CPU assembly
// and need no atomics. Traffic: the block values and one 8-byte source
// index per contribution read once, the values written once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/b200ldl.h"
#include "ldl_internal.h"

namespace {

// Contributions per CSR entry are few (1 to 4 in the mesh workloads), so an
// entry is bound by the latency of ptr -> src -> block value and the kernel by
// the bytes of the plan: the indices are 32-bit where the plan allows (half
// the plan's bytes), and a thread takes kPer entries at a time, whose first
// two contributions are loaded before any is added. An entry's sum stays in
// order from zero. Plane-stress elements, 256 x 256 (151 MB of blocks, 6.09 M
// entries): 69.4 us with 64-bit indices and an entry at a time, 53.1 us now (one
// entry at a time 62, four 64).
constexpr int kPer = 2;

// 32-bit indices take a plan whose contributions b, b + 1 and b + 2 of an
// entry that begins at b can be named, also where it has none and begins at
// the end of the list
constexpr bool fits_32(long long values, long long contributions) {
  return values <= 2147483647LL && contributions <= 2147483647LL - 2;
}
static_assert(fits_32(2147483647LL, 2147483645LL) && !fits_32(1, 2147483646LL) &&
                  !fits_32(1, 2147483647LL) && !fits_32(2147483648LL, 1),
              "the last entry's b + 2 is an int");

template <typename Index>
__global__ void __launch_bounds__(256)
    csr_gather_kernel(int nnz, const Index* __restrict__ ptr, const Index* __restrict__ src,
                      const double* __restrict__ blocks, double* __restrict__ vals) {
  const int per_cta = blockDim.x * kPer;
  for (long long p0 = (long long)blockIdx.x * per_cta; p0 < nnz;
       p0 += (long long)gridDim.x * per_cta) {
    Index b[kPer], e[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const long long p = p0 + threadIdx.x + u * blockDim.x;
      b[u] = p < nnz ? __ldg(ptr + p) : 0;
      e[u] = p < nnz ? __ldg(ptr + p + 1) : 0;
    }
    Index s0[kPer], s1[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      s0[u] = b[u] < e[u] ? __ldg(src + b[u]) : 0;
      s1[u] = b[u] + 1 < e[u] ? __ldg(src + b[u] + 1) : 0;
    }
    double x0[kPer], x1[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      x0[u] = b[u] < e[u] ? blocks[s0[u]] : 0.0;
      x1[u] = b[u] + 1 < e[u] ? blocks[s1[u]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const long long p = p0 + threadIdx.x + u * blockDim.x;
      if (p >= nnz) continue;
      double v = 0.0;
      if (b[u] < e[u]) v += x0[u];
      if (b[u] + 1 < e[u]) v += x1[u];
      for (Index q = b[u] + 2; q < e[u]; q++) v += blocks[src[q]];
      __stcs(vals + p, v);
    }
  }
}

template <typename T>
struct DevArr {
  T* ptr = nullptr;
  ~DevArr() { release(); }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
  }
};

}  // namespace

struct b200ldl_assembly {
  int n = 0, nnz = 0;
  long long nvals = 0;    // block values expected (sum over groups of nelem * ncomp^2)
  long long dropped = 0;  // contributions outside the pattern
  // the plan, host copy: 32-bit where it fits
  std::vector<long long> ptr, src;
  std::vector<int> ptr32, src32;
  bool narrow = false;
  long long kept() const { return narrow ? (long long)src32.size() : (long long)src.size(); }
  // and the device copy, one of the pairs, complete once `uploaded` is set
  DevArr<long long> d_ptr, d_src;
  DevArr<int> d_ptr32, d_src32;
  mutable std::mutex mu;  // of the upload
  bool uploaded = false;
  std::string last_error;
};

namespace {

int afail(b200ldl_assembly* a, int code, const char* fmt, ...) {
  if (a) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    a->last_error = buf;
  }
  return code;
}

// CSR index of (row, col), or -1 when the pattern has no such entry
inline long long find_entry(const int* rowp, const int* cols, int row, int col) {
  const int* b = cols + rowp[row];
  const int* e = cols + rowp[row + 1];
  const int* it = std::lower_bound(b, e, col);
  return (it != e && *it == col) ? (long long)(it - cols) : -1;
}

template <typename T>
cudaError_t to_device(DevArr<T>& d, const std::vector<T>& h) {
  d.release();
  cudaError_t e = cudaMalloc(&d.ptr, std::max<size_t>(1, h.size()) * sizeof(T));
  if (e != cudaSuccess) d.ptr = nullptr;
  if (e == cudaSuccess && !h.empty())
    e = cudaMemcpy(d.ptr, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
  return e;
}

// Threads may share a plan: the first to come uploads it, and it counts as
// uploaded once both copies have arrived (the copies' stream does not order
// the streams that read them).
int upload(b200ldl_assembly* a) {
  std::lock_guard<std::mutex> lock(a->mu);
  if (a->uploaded) return 0;
  cudaError_t e = a->narrow ? to_device(a->d_ptr32, a->ptr32) : to_device(a->d_ptr, a->ptr);
  if (e == cudaSuccess) e = a->narrow ? to_device(a->d_src32, a->src32) : to_device(a->d_src, a->src);
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  if (e != cudaSuccess) {
    a->d_ptr32.release();
    a->d_src32.release();
    a->d_ptr.release();
    a->d_src.release();
    cudaGetLastError();  // reported here, not by the thread's next launch
    return afail(a, -3, "CUDA error: %s", cudaGetErrorString(e));
  }
  a->uploaded = true;
  return 0;
}

}  // namespace

extern "C" {

int b200ldl_assembly_create(b200ldl_assembly_t* out, int n, const int* rowp, const int* cols,
                            int ngroups, const int* nelems, const int* ncomp, const int* conn) {
  if (!out) return -1;
  *out = nullptr;
  auto* a = new b200ldl_assembly;
  *out = a;
  if (n < 0 || !rowp || (n > 0 && !cols) || ngroups < 0 || (ngroups > 0 && (!nelems || !ncomp)))
    return afail(a, -1, "bad arguments");
  if (rowp[0] != 0) return afail(a, -1, "rowp[0] must be 0");
  for (int r = 0; r < n; r++) {
    if (rowp[r + 1] < rowp[r]) return afail(a, -1, "rowp must be non-decreasing");
    for (int t = rowp[r] + 1; t < rowp[r + 1]; t++)
      if (cols[t] <= cols[t - 1]) return afail(a, -1, "columns of row %d not sorted", r);
  }
  a->n = n;
  a->nnz = rowp[n];
  long long nconn = 0;
  for (int g = 0; g < ngroups; g++) {
    if (nelems[g] < 0 || ncomp[g] < 0) return afail(a, -1, "group %d: negative size", g);
    nconn += (long long)nelems[g] * ncomp[g];
    a->nvals += (long long)nelems[g] * ncomp[g] * ncomp[g];
  }
  if (nconn > 0 && !conn) return afail(a, -1, "conn is null");
  for (long long t = 0; t < nconn; t++)
    if (conn[t] < 0 || conn[t] >= n)
      return afail(a, -1, "connectivity entry %lld = %d out of range", t, conn[t]);
  // pass 1: contributions per CSR entry; pass 2: their sources, in order
  std::vector<long long> cnt((size_t)a->nnz + 1, 0);
  for (int pass = 0; pass < 2; pass++) {
    const int* c = conn;
    long long off = 0;  // first block value of the group
    for (int g = 0; g < ngroups; g++) {
      const int m = ncomp[g];
      for (int e = 0; e < nelems[g]; e++, c += m) {
        for (int j = 0; j < m; j++) {
          for (int i = 0; i < m; i++) {
            const long long p = find_entry(rowp, cols, c[j], c[i]);
            if (p < 0) {
              if (pass == 0) a->dropped++;
              continue;
            }
            if (pass == 0)
              cnt[p + 1]++;
            else if (a->narrow)
              a->src32[cnt[p]++] = (int)(off + ((long long)e * m + j) * m + i);
            else
              a->src[cnt[p]++] = off + ((long long)e * m + j) * m + i;
          }
        }
      }
      off += (long long)nelems[g] * m * m;
    }
    if (pass == 0) {
      for (int p = 0; p < a->nnz; p++) cnt[p + 1] += cnt[p];
      a->ptr = cnt;
      a->narrow = fits_32(a->nvals, cnt[a->nnz]);
      if (a->narrow) {
        a->ptr32.assign(a->ptr.begin(), a->ptr.end());
        std::vector<long long>().swap(a->ptr);
        a->src32.assign((size_t)cnt[a->nnz], 0);
      } else {
        a->src.assign((size_t)cnt[a->nnz], 0);
      }
    }
  }
  return 0;
}

int b200ldl_assembly_values(b200ldl_assembly_t a, const double* blocks, double* vals,
                            void* stream) {
  if (!a) return -1;
  if (a->nnz > 0 && !vals) return afail(a, -1, "vals is null");
  if (a->kept() > 0 && !blocks) return afail(a, -1, "blocks is null");
  if (a->nnz == 0) return 0;
  const int st = upload(a);
  if (st != 0) return st;
  const int threads = 256;
  const int per_cta = threads * kPer;
  const int grid = std::max(1, std::min((a->nnz - 1) / per_cta + 1, b200ldl::kSMs * 64));
  const cudaStream_t st_ = static_cast<cudaStream_t>(stream);
  if (a->narrow)
    csr_gather_kernel<<<grid, threads, 0, st_>>>(a->nnz, a->d_ptr32.ptr, a->d_src32.ptr, blocks,
                                                 vals);
  else
    csr_gather_kernel<<<grid, threads, 0, st_>>>(a->nnz, a->d_ptr.ptr, a->d_src.ptr, blocks, vals);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return afail(a, -3, "CUDA error: %s", cudaGetErrorString(e));
  return 0;
}

int b200ldl_assembly_info(b200ldl_assembly_t a, long long* out, int nout) {
  if (!a || !out) return -1;
  const long long v[4] = {a->kept(), a->dropped, a->nvals, (long long)a->nnz};
  for (int t = 0; t < nout && t < 4; t++) out[t] = v[t];
  return 0;
}

int b200ldl_assembly_plan(b200ldl_assembly_t a, long long* ptr, long long* src) {
  if (!a) return -1;
  if (a->narrow) {
    if (ptr) std::copy(a->ptr32.begin(), a->ptr32.end(), ptr);
    if (src) std::copy(a->src32.begin(), a->src32.end(), src);
  } else {
    if (ptr) std::copy(a->ptr.begin(), a->ptr.end(), ptr);
    if (src) std::copy(a->src.begin(), a->src.end(), src);
  }
  return 0;
}

const char* b200ldl_assembly_last_error(b200ldl_assembly_t a) {
  return a ? a->last_error.c_str() : "null handle";
}

void b200ldl_assembly_destroy(b200ldl_assembly_t a) { delete a; }

}  // extern "C"

namespace b200ldl {

int assembly_device_plan(const ::b200ldl_assembly* a, int* n, int* nnz, AsmPlan* plan) {
  if (!a) return -1;
  std::lock_guard<std::mutex> lock(a->mu);
  if (!a->uploaded) return -1;
  *n = a->n;
  *nnz = a->nnz;
  *plan = AsmPlan{a->d_ptr32.ptr, a->d_src32.ptr, a->d_ptr.ptr, a->d_src.ptr};
  return 0;
}

}  // namespace b200ldl
