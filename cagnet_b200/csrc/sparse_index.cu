// Integer index work on the sparse operand: COO row indices -> CSR row offsets, and validation.
// Pure integer arithmetic, bit-exact by construction.
#include <limits.h>

#include "common.cuh"

namespace cagnet {

static thread_local char g_last_error[256] = "";
char* last_error_buf() { return g_last_error; }

// rowptr[i] = first e with rows[e] >= i  (= number of entries whose row index is < i).
// One thread per output; used when rows are few compared with nonzeros (log2(nnz) probes each,
// the top of the search tree stays in L1/L2).
__global__ void coo2csr_search_kernel(const int* __restrict__ rows, int nnz, int n, int* __restrict__ rowptr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  int lo = 0, hi = nnz;
  while (lo < hi) {
    const int mid = lo + ((hi - lo) >> 1);
    if (__ldg(rows + mid) < i) lo = mid + 1; else hi = mid;
  }
  rowptr[i] = lo;
}

// Same result by boundary detection: entry e closes every row in (rows[e-1], rows[e]].
// One coalesced pass over the row indices; used when n is comparable with nnz.
__global__ void coo2csr_boundary_kernel(const int* __restrict__ rows, int nnz, int n, int* __restrict__ rowptr) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e > nnz) return;
  const int prev = (e == 0) ? -1 : max(-1, __ldg(rows + e - 1));
  const int cur = (e == nnz) ? n : min(n, __ldg(rows + e));   // clamped: malformed input cannot write out of range
  for (int r = prev + 1; r <= cur; ++r) rowptr[r] = static_cast<int>(e);
}

__global__ void check_csr_kernel(const int* __restrict__ rowptr, const int* __restrict__ col,
                                 const int* __restrict__ rows, int n, int m, int nnz, int* status) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (rows && t < nnz) {
    const int r = rows[t];
    if (r < 0 || r >= n) atomicMax(status, 5);
    else if (t > 0 && rows[t - 1] > r) atomicMax(status, 3);
  }
  if (t == 0) {
    if (rowptr[0] != 0) atomicMax(status, 1);
    if (rowptr[n] != nnz) atomicMax(status, 2);
  }
  if (t < n && rowptr[t] > rowptr[t + 1]) atomicMax(status, 3);
  if (t < nnz) {
    const int c = col[t];
    if (c < 0 || c >= m) atomicMax(status, 4);
  }
}

// The indices of a row-sorted COO list: 16 bytes of each array per thread and step where they are aligned (8 M entries: 20 us
// for one entry per thread, 11 us so).
__global__ void __launch_bounds__(256) check_coo_kernel(const int* __restrict__ rows, const int* __restrict__ cols, int n, int m,
                                                        int64_t nnz, int vec4, int* status) {
  pdl_trigger();
  pdl_wait();
  int code = 0;
  const int64_t steps = (nnz + 3) / 4;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < steps;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t e = t * 4;
    const int live = static_cast<int>(nnz - e < 4 ? nnz - e : 4);
    int r[4], c[4];
    if (vec4 && live == 4) {
      const int4 a = __ldg(reinterpret_cast<const int4*>(rows + e)), b = __ldg(reinterpret_cast<const int4*>(cols + e));
      r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
      c[0] = b.x; c[1] = b.y; c[2] = b.z; c[3] = b.w;
    } else {
      for (int j = 0; j < live; ++j) {
        r[j] = __ldg(rows + e + j);
        c[j] = __ldg(cols + e + j);
      }
    }
    int before = e > 0 ? __ldg(rows + e - 1) : INT_MIN;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j >= live) break;
      if (c[j] < 0 || c[j] >= m) code = max(code, 4);
      if (r[j] < 0 || r[j] >= n) code = max(code, 5);
      else if (before > r[j]) code = max(code, 3);
      before = r[j];
    }
  }
  if (code) atomicMax(status, code);
}

}  // namespace cagnet

using namespace cagnet;

extern "C" int cagnet_version(void) { return 100; }

extern "C" const char* cagnet_last_error_string(void) { return last_error_buf(); }

extern "C" int cagnet_coo2csr_i32(const int32_t* rows, int64_t nnz, int32_t n, int32_t* rowptr, void* stream) {
  if (n < 0 || nnz < 0 || !rowptr || (nnz > 0 && !rows)) return fail(CAGNET_E_ARG, "cagnet_coo2csr_i32: bad argument");
  if (nnz > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_coo2csr_i32: nnz %s%lld exceeds int32", "", nnz);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int innz = static_cast<int>(nnz);
  if (nnz > 16 * static_cast<int64_t>(n)) {
    coo2csr_search_kernel<<<(n + 1 + 255) / 256, 256, 0, s>>>(rows, innz, n, rowptr);
  } else {
    coo2csr_boundary_kernel<<<static_cast<unsigned>((nnz + 1 + 255) / 256), 256, 0, s>>>(rows, innz, n, rowptr);
  }
  return check_launch("cagnet_coo2csr_i32");
}

extern "C" int cagnet_check_csr_i32(const int32_t* rowptr, const int32_t* col, const int32_t* rows, int32_t n, int32_t m,
                                    int64_t nnz, int32_t* status_dev, void* stream) {
  if (n < 0 || m < 0 || nnz < 0 || !rowptr || !status_dev || (nnz > 0 && !col))
    return fail(CAGNET_E_ARG, "cagnet_check_csr_i32: bad argument");
  if (nnz > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_check_csr_i32: nnz %s%lld exceeds int32", "", nnz);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(status_dev, 0, sizeof(int), s);
  const int64_t work = (nnz > n ? nnz : n) + 1;
  check_csr_kernel<<<static_cast<unsigned>((work + 255) / 256), 256, 0, s>>>(rowptr, col, rows, n, m,
                                                                            static_cast<int>(nnz), status_dev);
  return check_launch("cagnet_check_csr_i32");
}

extern "C" int cagnet_check_coo_i32(const int32_t* rows, const int32_t* cols, int32_t n, int32_t m, int64_t nnz,
                                    int32_t* status_dev, void* stream) {
  if (n < 0 || m < 0 || nnz < 0 || !status_dev || (nnz > 0 && (!rows || !cols)))
    return fail(CAGNET_E_ARG, "cagnet_check_coo_i32: bad argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(status_dev, 0, sizeof(int), s);
  if (nnz == 0) return check_launch("cagnet_check_coo_i32");
  const int64_t blocks = ((nnz + 3) / 4 + 255) / 256;
  const int vec4 = aligned(rows, 16) && aligned(cols, 16) ? 1 : 0;
  check_coo_kernel<<<static_cast<unsigned>(blocks < 16 * kNumSMs ? blocks : 16 * kNumSMs), 256, 0, s>>>(rows, cols, n, m, nnz, vec4,
                                                                                                       status_dev);
  return check_launch("cagnet_check_coo_i32");
}
