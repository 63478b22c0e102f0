// Shared host-side helpers of the cagnet_b200 C ABI (error reporting, launch checks).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/cagnet_b200.h"

namespace cagnet {

// Last error text of the calling thread (returned by cagnet_last_error_string).
char* last_error_buf();

inline int fail(int code, const char* fmt, const char* a = "", long long b = 0, long long c = 0) {
  snprintf(last_error_buf(), 256, fmt, a, b, c);
  return code;
}

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    snprintf(last_error_buf(), 256, "%s: CUDA launch failed: %s", what, cudaGetErrorString(e));
    return CAGNET_E_LAUNCH;
  }
  return CAGNET_OK;
}

__host__ __device__ inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

constexpr int kNumSMs = 148;  // B200

// k length of one tensor-core accumulation of the dense-core multiply (tuning knob "core_chunk")
int core_chunk();
int set_core_chunk(int value);
// the same for the integer-core multiply (tuning knob "core_chunk_int")
int core_chunk_int();
int set_core_chunk_int(int value);

__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// Programmatic dependent launch: a kernel launched through launch_pdl may be scheduled while the kernel in front of it
// in the stream is still running (its launch latency and prologue then cost nothing), and must call pdl_wait() before
// it touches memory: that returns when everything in front is complete and visible.  pdl_trigger() lets the kernel
// behind it be scheduled early in turn.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

template <typename... P, typename... A>
inline cudaError_t launch_pdl_if(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  return launch_pdl_if(true, kernel, grid, block, smem, stream, args...);
}

// The row kernels of spmm.cu with what the host knows about the block: hub_rows = rows listed in the plan, -1 = unknown.
int spmm_rows_f32(const int32_t* rowptr, const int32_t* col, const float* val, int32_t n, int32_t m, int64_t nnz,
                  const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f, float beta, const void* plan,
                  int32_t hub_rows, void* stream);
int spmm_forced_tile();      // "spmm_tile" when a sweep has set it: such multiplies run the row kernels

// X . W on the tensor cores (dense_tc.cu), where it applies
bool gemm_nn_tc_applies(const float* X, int64_t ldx, int64_t n, int K, int N, int epilogue);
int gemm_nn_tc(const float* X, int64_t ldx, const float* W, int64_t ldw, int transW, float* Z, int64_t ldz, int64_t n, int K, int N,
               int epilogue, const float* aux, int64_t ldaux, cudaStream_t s);
// The masked NLL of log-softmax rows and its gradient before the log-softmax, written with them by the product's epilogue.
struct TcLoss {
  const int64_t* y;
  const uint8_t* mask;
  float* dz;
  float* parts;              // partial sums of the labels' log-probabilities, kTcLossParts at most
  int64_t lddz;
  int cls_lo, cls_hi;
  float inv_count;
};
constexpr int kTcLossParts = kNumSMs * 16;
int gemm_nn_tc_nll(const float* X, int64_t ldx, const float* W, int64_t ldw, float* Z, int64_t ldz, int64_t n, int K, int N, const TcLoss& loss,
                   int32_t* parts, cudaStream_t s);
bool gemm_tn_tc_applies(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int K, int N);
int gemm_tn_tc_blocks(int64_t n, int K, int N);
int gemm_tn_tc(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int K, int N, float* part, cudaStream_t s);
int gemm_tc_error();      // 1 if one of its kernels gave up on a wait

}  // namespace cagnet
