// Dense side of the GCN layer for sm_100a: tall-skinny fp32 products with fused activations,
// the split-row weight-gradient product, row-wise log-softmax and the masked NLL loss.
//
// All of these are HBM-bound at GCN shapes (a 233K x 602 operand against a 602 x 16 weight has
// ~7 flop/byte), so they run on the fp32 FMA pipes from shared-memory tiles: the tall operand is
// read exactly once, coalesced; the small operand lives in shared memory.
#include <limits.h>
#include <math.h>

#include "common.cuh"

namespace cagnet {

// ------------------------------------------------------------------------------------------------
// Z[n x N] = epilogue(X[n x K] * W) for tall X and small W, fp32 FMAs.
//
// A thread owns TM rows and NP groups of 4 columns; LC lanes side by side cover one row of the tile (LC * 4 * NP columns), the
// 32 / LC row groups of a warp share their W values through broadcasts.  Per k that is TM / 4 + NP 128-bit shared-memory reads
// for 4 TM NP FMAs (8 x 4: three reads for 32), so the FMA pipe and HBM are what bounds it: 233K x 602 x 16 is 62 us of FMAs
// at the peak rate over 86 us of X at the copy rate.  X tiles are fetched row by row (whole 64- or 128-byte pieces), held in
// registers while the previous tile is multiplied, and stored k-major with rows permuted by k / 4 (xor of row bits 2-4),
// which makes both the transposing stores and the row-vector reads conflict-free.
template <int BK>
__device__ __forceinline__ int x_swizzle(int k) { return (32 / (BK / 4)) * ((k >> 2) & (BK / 4 - 1)); }

struct GemmArgs {
  const float *X, *W, *aux;
  float* Z;
  int64_t ldx, ldw, ldz, ldaux, n;
  int transW, K, N, epilogue, x_vec4, z_vec4;
  TcLoss loss;
};

// 4 consecutive k of row gr (zeros outside the matrix)
__device__ __forceinline__ float4 load_x4(const GemmArgs& a, int64_t gr, int k) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (gr < a.n && k < a.K) {
    const float* p = a.X + gr * a.ldx + k;
    if (a.x_vec4 && k + 3 < a.K) {
      v = __ldg(reinterpret_cast<const float4*>(p));
    } else {
      v.x = __ldg(p);
      if (k + 1 < a.K) v.y = __ldg(p + 1);
      if (k + 2 < a.K) v.z = __ldg(p + 2);
      if (k + 3 < a.K) v.w = __ldg(p + 3);
    }
  }
  return v;
}
__device__ __forceinline__ float load_w(const GemmArgs& a, int k, int j) {
  if (k >= a.K || j >= a.N) return 0.f;
  return __ldg(a.W + (a.transW ? static_cast<int64_t>(j) * a.ldw + k : static_cast<int64_t>(k) * a.ldw + j));
}

template <int BK, int LC, int NP, int TM>
__device__ __forceinline__ void tile_product(const float* __restrict__ Xs, int ldxs, const float* __restrict__ Ws, int r0, int lc,
                                             float (&acc)[TM][NP][4]) {
  constexpr int BN = LC * 4 * NP;
#pragma unroll
  for (int k = 0; k < BK; ++k) {
    float x[TM];
    const float* xp = Xs + k * ldxs;
    const int sw = x_swizzle<BK>(k);
    if constexpr (TM >= 4) {
#pragma unroll
      for (int q = 0; q < TM / 4; ++q) {
        const float4 t = *reinterpret_cast<const float4*>(xp + ((r0 + 4 * q) ^ sw));
        x[4 * q] = t.x; x[4 * q + 1] = t.y; x[4 * q + 2] = t.z; x[4 * q + 3] = t.w;
      }
    } else {
      const float2 t = *reinterpret_cast<const float2*>(xp + (r0 ^ sw));
      x[0] = t.x; x[1] = t.y;
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float4 w = *reinterpret_cast<const float4*>(Ws + k * BN + p * (LC * 4) + lc * 4);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        acc[i][p][0] = fmaf(x[i], w.x, acc[i][p][0]);
        acc[i][p][1] = fmaf(x[i], w.y, acc[i][p][1]);
        acc[i][p][2] = fmaf(x[i], w.z, acc[i][p][2]);
        acc[i][p][3] = fmaf(x[i], w.w, acc[i][p][3]);
      }
    }
  }
}

// Four columns of a row through the elementwise epilogues and out.
__device__ __forceinline__ void store_z4(const GemmArgs& a, int64_t gr, int c, float4 v) {
  const int live = a.N - c;
  if (live <= 0) return;
  float* z = a.Z + gr * a.ldz + c;
  float r[4] = {v.x, v.y, v.z, v.w};
  if (a.epilogue == CAGNET_EPI_RELU) {
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = fmaxf(r[j], 0.f);
  } else if (a.epilogue == CAGNET_EPI_RELU_MASK) {
    const float* p = a.aux + gr * a.ldaux + c;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < live) r[j] = __ldg(p + j) > 0.f ? r[j] : 0.f;
  } else if (a.epilogue == CAGNET_EPI_ACCUMULATE) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < live) r[j] += z[j];
  }
  if (live >= 4 && a.z_vec4) {
    *reinterpret_cast<float4*>(z) = make_float4(r[0], r[1], r[2], r[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < live) z[j] = r[j];
  }
}

// log(sum(exp)) of a row spread over LANES neighbouring lanes, COLS values each; columns from `live` on do not count.
template <int LANES, int COLS>
__device__ __forceinline__ float row_lse(const float (&v)[COLS], const bool (&live)[COLS]) {
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < COLS; ++j)
    if (live[j]) mx = fmaxf(mx, v[j]);
#pragma unroll
  for (int off = 1; off < LANES; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < COLS; ++j) sum += live[j] ? expf(v[j] - mx) : 0.f;
#pragma unroll
  for (int off = 1; off < LANES; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  return mx + logf(sum);
}

// NLL: log-softmax with its masked NLL and the gradient before the log-softmax, as the tensor-core kernel writes them (a kernel of
// 2.4 us and its launch less per epoch of 16 K vertices).
template <int LC, int NP, int TM, int WARPS, int BK, bool NLL>
__global__ void __launch_bounds__(WARPS * 32) gemm_nn_kernel(GemmArgs a) {
  constexpr int BN = LC * 4 * NP, WR = 32 / LC * TM, BM = WARPS * WR, T = WARPS * 32;
  constexpr int XV = BM * BK / 4 / T;            // float4 of X per thread and tile
  constexpr int WV = (BK * BN + T - 1) / T;
  static_assert(BM % 32 == 0 && BM * BK / 4 % T == 0, "tile shape");
  __shared__ __align__(16) float Xs[BK * BM];
  __shared__ __align__(16) float Ws[BK * BN];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lc = lane % LC, r0 = warp * WR + lane / LC * TM;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * BM;
  const int n0 = blockIdx.y * BN;

  float acc[TM][NP][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][p][j] = 0.f;

  float4 xv[XV];
  float wv[WV];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const int idx = tid + T * u;
      xv[u] = load_x4(a, row0 + idx / (BK / 4), k0 + idx % (BK / 4) * 4);
    }
#pragma unroll
    for (int u = 0; u < WV; ++u) {
      const int idx = tid + T * u;
      wv[u] = idx < BK * BN ? load_w(a, k0 + idx / BN, n0 + idx % BN) : 0.f;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < a.K; k0 += BK) {
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const int idx = tid + T * u;
      const int r = idx / (BK / 4), k = idx % (BK / 4) * 4;
      const int at = r ^ x_swizzle<BK>(k);
      Xs[(k + 0) * BM + at] = xv[u].x;
      Xs[(k + 1) * BM + at] = xv[u].y;
      Xs[(k + 2) * BM + at] = xv[u].z;
      Xs[(k + 3) * BM + at] = xv[u].w;
    }
#pragma unroll
    for (int u = 0; u < WV; ++u) {
      const int idx = tid + T * u;
      if (idx < BK * BN) Ws[idx] = wv[u];
    }
    __syncthreads();
    if (k0 + BK < a.K) fetch(k0 + BK);
    tile_product<BK, LC, NP, TM>(Xs, BM, Ws, r0, lc, acc);
    __syncthreads();
  }

  [[maybe_unused]] float picked = 0.f;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t gr = row0 + r0 + i;            // no early exit: the shuffles need all lanes
    if (NLL || a.epilogue == CAGNET_EPI_LOG_SOFTMAX || a.epilogue == CAGNET_EPI_LOG_SOFTMAX_256) {
      float v[NP * 4];
      bool live[NP * 4];
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[p * 4 + j] = acc[i][p][j];
          live[p * 4 + j] = p * (LC * 4) + lc * 4 + j < a.N;
        }
      const float lse = row_lse<LC, NP * 4>(v, live);
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][p][j] -= lse;
    }
    if (gr < a.n) {
#pragma unroll
      for (int p = 0; p < NP; ++p)
        store_z4(a, gr, n0 + p * (LC * 4) + lc * 4, make_float4(acc[i][p][0], acc[i][p][1], acc[i][p][2], acc[i][p][3]));
      if constexpr (NLL) {
        int at = -1;
        if (a.loss.mask[gr]) {
          const int64_t label = a.loss.y[gr];
          if (label >= a.loss.cls_lo && label < a.loss.cls_hi) at = static_cast<int>(label - a.loss.cls_lo);
        }
        const float w = a.loss.inv_count;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const int c = p * (LC * 4) + lc * 4;
          float g[4] = {0.f, 0.f, 0.f, 0.f};
          if (at >= 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              g[j] = (c + j == at ? -w : 0.f) + expf(acc[i][p][j]) * w;
              if (c + j == at) picked += acc[i][p][j];
            }
          }
          float* d = a.loss.dz + gr * a.loss.lddz + c;
          if (c + 4 <= a.N && a.z_vec4) {
            *reinterpret_cast<float4*>(d) = make_float4(g[0], g[1], g[2], g[3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (c + j < a.N) d[j] = g[j];
          }
        }
      }
    }
  }
  if constexpr (NLL) {
    __shared__ float red[WARPS];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) picked += __shfl_xor_sync(0xffffffffu, picked, off);
    if (lane == 0) red[warp] = picked;
    __syncthreads();
    if (tid == 0) {
      float t = red[0];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) t += red[w];
      a.loss.parts[blockIdx.x] = t;
    }
  }
}

// The same product for few rows and a long K: 16 rows per block, its 8 warps take K tiles in turn (own tiles, no block
// barrier), their sums are added in warp order.  2,708 x 1,433 x 16 is 11 blocks of the kernel above, each a chain of 90
// tiles (35 us); here 170 blocks of 6 tiles per warp (N <= 64).
template <int LC, int TM>
__global__ void __launch_bounds__(256) gemm_nn_splitk_kernel(GemmArgs a) {
  constexpr int BK = LC == 4 ? 32 : 16, BN = LC * 4, ROWS = 32 / LC * TM, WARPS = 8, CPT = BN / 16;      // 48 KB of tiles
  static_assert(ROWS == 16, "16 rows per warp");
  __shared__ __align__(16) float Xs[WARPS][BK * 32];        // 16 rows used: the permutation moves rows inside 32
  __shared__ __align__(16) float Ws[WARPS][BK * BN];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lc = lane % LC, r0 = lane / LC * TM;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * ROWS;
  float acc[TM][1][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][0][j] = 0.f;
  constexpr int XV = ROWS * BK / 4 / 32, WV = BK * BN / 4 / 32;
  const bool w_vec4 = !a.transW && a.N == BN && a.ldw % 4 == 0 && aligned(a.W, 16);
  float4 xv[XV], wv[WV];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const int idx = lane + 32 * u;
      xv[u] = load_x4(a, row0 + idx / (BK / 4), k0 + idx % (BK / 4) * 4);
    }
#pragma unroll
    for (int u = 0; u < WV; ++u) {
      const int idx = (lane + 32 * u) * 4, k = k0 + idx / BN, j = idx % BN;
      if (w_vec4 && k < a.K) wv[u] = __ldg(reinterpret_cast<const float4*>(a.W + static_cast<int64_t>(k) * a.ldw + j));
      else wv[u] = make_float4(load_w(a, k, j), load_w(a, k, j + 1), load_w(a, k, j + 2), load_w(a, k, j + 3));
    }
  };
  int k0 = warp * BK;
  fetch(k0);
  for (; k0 < a.K; k0 += WARPS * BK) {
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const int idx = lane + 32 * u;
      const int r = idx / (BK / 4), k = idx % (BK / 4) * 4;
      const int at = r ^ x_swizzle<BK>(k);
      Xs[warp][(k + 0) * 32 + at] = xv[u].x;
      Xs[warp][(k + 1) * 32 + at] = xv[u].y;
      Xs[warp][(k + 2) * 32 + at] = xv[u].z;
      Xs[warp][(k + 3) * 32 + at] = xv[u].w;
    }
#pragma unroll
    for (int u = 0; u < WV; ++u) *reinterpret_cast<float4*>(&Ws[warp][(lane + 32 * u) * 4]) = wv[u];
    __syncwarp();
    if (k0 + WARPS * BK < a.K) fetch(k0 + WARPS * BK);
    tile_product<BK, LC, 1, TM>(Xs[warp], 32, Ws[warp], r0, lc, acc);
    __syncwarp();
  }
  // sums of the 8 warps, each in its own W tile
#pragma unroll
  for (int i = 0; i < TM; ++i)
    *reinterpret_cast<float4*>(&Ws[warp][(r0 + i) * BN + lc * 4]) = make_float4(acc[i][0][0], acc[i][0][1], acc[i][0][2], acc[i][0][3]);
  __syncthreads();
  // 16 lanes per row, CPT columns each
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * CPT;
  float v[CPT];
  bool live[CPT];
#pragma unroll
  for (int j = 0; j < CPT; ++j) {
    v[j] = 0.f;
    live[j] = c + j < a.N;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) v[j] += Ws[w][r * BN + c + j];
  }
  if (a.epilogue == CAGNET_EPI_LOG_SOFTMAX) {
    const float lse = row_lse<16, CPT>(v, live);
#pragma unroll
    for (int j = 0; j < CPT; ++j) v[j] -= lse;
  }
  const int64_t gr = row0 + r;
  if (gr >= a.n) return;
#pragma unroll
  for (int j = 0; j < CPT; ++j) {
    if (!live[j]) continue;
    float* z = a.Z + gr * a.ldz + c + j;
    float t = v[j];
    if (a.epilogue == CAGNET_EPI_RELU) t = fmaxf(t, 0.f);
    else if (a.epilogue == CAGNET_EPI_RELU_MASK) t = __ldg(a.aux + gr * a.ldaux + c + j) > 0.f ? t : 0.f;
    else if (a.epilogue == CAGNET_EPI_ACCUMULATE) t += *z;
    *z = t;
  }
}

// ------------------------------------------------------------------------------------------------
// out[K x N] = H^T * G over n rows.  grid (chunks, K tiles of 64, N tiles of 64).  Each block
// streams its row chunk 32 rows at a time through shared memory and keeps a 64 x NT tile of
// partial sums in registers: unit u = (k = u % 64, 4 columns jb = u / 64).
constexpr int kTnKT = 64;
constexpr int kTnNT = 64;
constexpr int kTnRB = 32;

__global__ void __launch_bounds__(256) gemm_tn_partial_kernel(const float* __restrict__ H, int64_t ldh,
                                                              const float* __restrict__ G, int64_t ldg, int64_t n,
                                                              int K, int N, int64_t rows_per_chunk,
                                                              float* __restrict__ ws) {
  __shared__ float Hs[kTnRB][kTnKT];
  __shared__ __align__(16) float Gs[kTnRB][kTnNT];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int k0 = blockIdx.y * kTnKT, n0 = blockIdx.z * kTnNT;
  const int64_t r_begin = static_cast<int64_t>(blockIdx.x) * rows_per_chunk;
  const int64_t r_end = min(n, r_begin + rows_per_chunk);
  const int nt = min(kTnNT, N - n0);        // live columns of this tile
  const int nb = (nt + 3) / 4;              // 4-column groups
  const int units = kTnKT * nb;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  // 32 rows of H (64 columns) and G (up to 64 columns) per step: 8 + 8 values per thread, fetched into registers
  // one step ahead of the multiply.
  float hv[8], gv[8];
  auto fetch = [&](int64_t r0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * u;
      const int r = idx / kTnKT, k = idx % kTnKT;
      hv[u] = (r0 + r < r_end && k0 + k < K) ? __ldg(H + (r0 + r) * ldh + k0 + k) : 0.f;
      const int j = idx % kTnNT;
      gv[u] = (r0 + r < r_end && j < nt) ? __ldg(G + (r0 + r) * ldg + n0 + j) : 0.f;
    }
  };
  if (r_begin < r_end) fetch(r_begin);
  for (int64_t r0 = r_begin; r0 < r_end; r0 += kTnRB) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * u;
      Hs[idx / kTnKT][idx % kTnKT] = hv[u];
      Gs[idx / kTnNT][idx % kTnNT] = gv[u];
    }
    __syncthreads();
    if (r0 + kTnRB < r_end) fetch(r0 + kTnRB);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int u = tid + 256 * i;
      if (u < units) {
        const int k = u % kTnKT, jb = u / kTnKT;
#pragma unroll 8
        for (int r = 0; r < kTnRB; ++r) {
          const float h = Hs[r][k];
          const float4 g = *reinterpret_cast<const float4*>(&Gs[r][jb * 4]);
          acc[i][0] = fmaf(h, g.x, acc[i][0]);
          acc[i][1] = fmaf(h, g.y, acc[i][1]);
          acc[i][2] = fmaf(h, g.z, acc[i][2]);
          acc[i][3] = fmaf(h, g.w, acc[i][3]);
        }
      }
    }
    __syncthreads();
  }
  float* wp = ws + static_cast<int64_t>(blockIdx.x) * K * N;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int u = tid + 256 * i;
    if (u < units) {
      const int k = k0 + u % kTnKT, jb = u / kTnKT;
      if (k < K) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = n0 + jb * 4 + j;
          if (c < N) wp[static_cast<int64_t>(k) * N + c] = acc[i][j];
        }
      }
    }
  }
}

// The same product for N <= 16 (the weight gradients of the 602 x 16 layer: H is the 233K x 602 feature matrix,
// G has 16 columns).  There the kernel above spends two shared-memory reads on four FMAs, prefetches one step
// ahead and runs at 1.4 TB/s of H with its warps waiting on the loads.  Here
//   * a thread owns 4 consecutive k and all 16 columns (64 accumulators) for one sixteenth of the rows of a step:
//     one 128-bit read of H and four of G feed 64 FMAs;
//   * the tiles of the next three steps are already on their way: 16-byte cp.async copies into a four-stage ring
//     of shared-memory tiles (64 rows x 64 columns of H and 64 x 16 of G per stage), out-of-range rows and
//     columns zero-filled by the copy's source size.
// Threads that share their k columns (same tid % 16) are summed at the end, first by a shuffle inside each warp,
// then over the 8 warps in warp order.  Needs 16-byte aligned rows of H and G.
constexpr int kTnSmallRB = 64;       // rows per step
constexpr int kTnSmallStages = 4;
constexpr int kTnSmallStageFloats = kTnSmallRB * kTnKT + kTnSmallRB * 16;
constexpr int kTnSmallSmemBytes = kTnSmallStages * kTnSmallStageFloats * 4;     // 80 KB; also holds the 32 KB of sums

__device__ __forceinline__ void cp_async16(float* smem_dst, const float* gmem_src, int src_bytes) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem_src), "r"(src_bytes) : "memory");
}

struct TnSmallArgs {
  const float *H, *G;
  float* ws;
  int64_t ldh, ldg, rows_per_chunk;
  int K, N, chunks, ktiles;            // chunks * ktiles blocks
};
// One product, or both weight gradients of a small epoch at a time (the blocks of the second behind those of the first: each fills a
// fraction of the chip, and a launch costs as much as either, 5 us at 16 K vertices).
__global__ void __launch_bounds__(256, 2) gemm_tn_small_kernel(TnSmallArgs first, TnSmallArgs second, int64_t n) {
  extern __shared__ __align__(16) float tn_smem[];
  pdl_trigger();
  pdl_wait();
  const bool other = blockIdx.x >= first.chunks * first.ktiles;
  const TnSmallArgs& a = other ? second : first;
  const int blk = blockIdx.x - (other ? first.chunks * first.ktiles : 0);
  const float *__restrict__ H = a.H, *__restrict__ G = a.G;
  float* __restrict__ ws = a.ws;
  const int64_t ldh = a.ldh, ldg = a.ldg, rows_per_chunk = a.rows_per_chunk;
  const int K = a.K, N = a.N, chunk = blk % a.chunks;
  const int tid = threadIdx.x;
  const int kq = tid & 15, rs = tid >> 4;
  const int k0 = blk / a.chunks * kTnKT;
  const int64_t r_begin = static_cast<int64_t>(chunk) * rows_per_chunk;
  const int64_t r_end = min(n, r_begin + rows_per_chunk);
  const int steps = static_cast<int>((r_end - r_begin + kTnSmallRB - 1) / kTnSmallRB);

  // copies of one step: 4 float4 of H and 1 float4 of G per thread
  auto issue = [&](int step) {
    if (step < steps) {
      float* hs = tn_smem + (step % kTnSmallStages) * kTnSmallStageFloats;
      float* gs = hs + kTnSmallRB * kTnKT;
      const int64_t r0 = r_begin + static_cast<int64_t>(step) * kTnSmallRB;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int idx = tid + 256 * u;             // float4 index in the H tile
        const int r = idx >> 4, c = (idx & 15) * 4;
        const int k = k0 + c;
        int bytes = (r0 + r < r_end) ? (K - k) * 4 : 0;
        bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
        const float* src = bytes ? H + (r0 + r) * ldh + k : H;
        cp_async16(hs + r * kTnKT + c, src, bytes);
      }
      const int r = tid >> 2, j = (tid & 3) * 4;
      int bytes = (r0 + r < r_end) ? (N - j) * 4 : 0;
      bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
      const float* src = bytes ? G + (r0 + r) * ldg + j : G;
      cp_async16(gs + r * 16 + j, src, bytes);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");     // an empty group keeps the count in step
  };

  float acc[4][16];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[i][j] = 0.f;

#pragma unroll
  for (int s = 0; s < kTnSmallStages - 1; ++s) issue(s);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kTnSmallStages - 2) : "memory");   // this step's tiles have landed
    __syncthreads();                     // ... for every thread, and everyone is done with the stage refilled next
    issue(step + kTnSmallStages - 1);
    const float* hs = tn_smem + (step % kTnSmallStages) * kTnSmallStageFloats;
    const float* gs = hs + kTnSmallRB * kTnKT;
#pragma unroll
    for (int q = 0; q < kTnSmallRB / 16; ++q) {
      const int r = rs + 16 * q;
      const float4 h4 = *reinterpret_cast<const float4*>(hs + r * kTnKT + kq * 4);
      const float h[4] = {h4.x, h4.y, h4.z, h4.w};
      float g[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 g4 = *reinterpret_cast<const float4*>(gs + r * 16 + c * 4);
        g[4 * c + 0] = g4.x; g[4 * c + 1] = g4.y; g[4 * c + 2] = g4.z; g[4 * c + 3] = g4.w;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[i][j] = fmaf(h[i], g[j], acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                       // the ring is free: it now holds the partial sums of the 8 warps
  float (*red)[16][64] = reinterpret_cast<float (*)[16][64]>(tn_smem);
  // lanes l and l + 16 of a warp hold the same k columns for two row subsets
  const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[i][j] += __shfl_down_sync(0xffffffffu, acc[i][j], 16);
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<float4*>(&red[warp][lane][i * 16 + j]) =
            make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  }
  __syncthreads();
  float* wp = ws + static_cast<int64_t>(chunk) * K * N;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int e = tid + 256 * u;                  // element of the 64 x 16 tile: k = e / 16, column j = e % 16
    const int kk = e >> 4, j = e & 15;
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += red[w][kk >> 2][(kk & 3) * 16 + j];
    if (k0 + kk < K && j < N) wp[static_cast<int64_t>(k0 + kk) * N + j] = sum;
  }
}

// Sum over the row chunks of 32 neighbouring elements of their partial products, for the threads of a block: warp w adds chunks
// w, w + 8, ... of all 32 (whole 128-byte reads), the eight sums are added in warp order -- the same order on every run.
// The sum of element idx is valid in the first warp.
__device__ __forceinline__ float tn_sum(const float* __restrict__ ws, int chunks, int total, int idx, float (&red)[8][32]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float s = 0.f;
  if (idx < total) {
#pragma unroll 4
    for (int c = warp; c < chunks; c += 8) s += __ldg(ws + static_cast<int64_t>(c) * total + idx);
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) s += red[w][lane];
  }
  return s;
}

// out[k, j] (+)= sum of the partial products.
__global__ void __launch_bounds__(256)
gemm_tn_reduce_kernel(const float* __restrict__ ws, int chunks, int K, int N, float* __restrict__ out, int64_t ldo,
                      float beta, int transposed) {
  __shared__ float red[8][32];
  pdl_trigger();
  pdl_wait();
  const int idx = blockIdx.x * 32 + (threadIdx.x & 31);
  const float s = tn_sum(ws, chunks, K * N, idx, red);
  if (threadIdx.x >= 32 || idx >= K * N) return;
  // transposed: the partials are those of G^T * H (K and N as passed here); out is (H^T * G)[N x K]
  float* o = transposed ? out + static_cast<int64_t>(idx % N) * ldo + idx / N : out + static_cast<int64_t>(idx / N) * ldo + idx % N;
  *o = (beta != 0.f) ? s + *o : s;
}

struct TnShape {
  int chunks;
  int64_t rows_per_chunk;
  int ktiles, ntiles;
};

static TnShape tn_shape(int64_t n, int K, int N) {
  TnShape s;
  s.ktiles = (K + kTnKT - 1) / kTnKT;
  s.ntiles = (N + kTnNT - 1) / kTnNT;
  int64_t target = (4 * kNumSMs) / (static_cast<int64_t>(s.ktiles) * s.ntiles);
  if (target < 1) target = 1;
  const int64_t max_chunks = (n + 255) / 256;
  int64_t chunks = target < max_chunks ? target : max_chunks;
  if (chunks < 1) chunks = 1;
  int64_t rows = (n + chunks - 1) / chunks;
  rows = (rows + kTnRB - 1) / kTnRB * kTnRB;
  if (rows < kTnRB) rows = kTnRB;
  s.rows_per_chunk = rows;
  s.chunks = static_cast<int>((n + rows - 1) / rows);
  if (s.chunks < 1) s.chunks = 1;
  return s;
}

// ------------------------------------------------------------------------------------------------
// Element (row, group of 4 columns) of a thread's grid-stride step; 32-bit division where the count allows it.
__device__ __forceinline__ void vec_index(int64_t i, int64_t total, int vecs, int64_t& r, int& c) {
  r = total <= INT_MAX ? static_cast<int>(i) / vecs : i / vecs;
  c = static_cast<int>(i - r * vecs) * 4;
}
__device__ __forceinline__ float4 load4_upto(const float* p, int live, int vec4) {
  if (vec4 && live >= 4) return *reinterpret_cast<const float4*>(p);
  float4 v = make_float4(p[0], 0.f, 0.f, 0.f);
  if (live > 1) v.y = p[1];
  if (live > 2) v.z = p[2];
  if (live > 3) v.w = p[3];
  return v;
}
__device__ __forceinline__ void store4_upto(float* p, float4 v, int live, int vec4) {
  if (vec4 && live >= 4) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    p[0] = v.x;
    if (live > 1) p[1] = v.y;
    if (live > 2) p[2] = v.z;
    if (live > 3) p[3] = v.w;
  }
}

// One 16-byte read (two for the gradient) and write per thread and step; z and h may be the same matrix.
__global__ void __launch_bounds__(256) relu_fwd_kernel(const float* z, int64_t ldz, float* h, int64_t ldh, int64_t n, int N, int vecs,
                                                       int vec4) {
  pdl_trigger();
  pdl_wait();
  const int64_t total = n * vecs;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t r;
    int c;
    vec_index(i, total, vecs, r, c);
    const float4 v = load4_upto(z + r * ldz + c, N - c, vec4);
    store4_upto(h + r * ldh + c, make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f)), N - c, vec4);
  }
}

__global__ void __launch_bounds__(256) relu_bwd_kernel(const float* __restrict__ h, int64_t ldh, const float* g, int64_t ldg, float* dz,
                                                       int64_t lddz, int64_t n, int N, int vecs, int vec4) {
  pdl_trigger();
  pdl_wait();
  const int64_t total = n * vecs;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t r;
    int c;
    vec_index(i, total, vecs, r, c);
    const float4 v = load4_upto(h + r * ldh + c, N - c, vec4), q = load4_upto(g + r * ldg + c, N - c, vec4);
    store4_upto(dz + r * lddz + c, make_float4(v.x > 0.f ? q.x : 0.f, v.y > 0.f ? q.y : 0.f, v.z > 0.f ? q.z : 0.f, v.w > 0.f ? q.w : 0.f),
                N - c, vec4);
  }
}

// LR lanes per row, NV groups of 4 columns per lane (column 4 lane + 4 LR v): the row is read once into registers (16-byte
// loads), reduced by shuffles and written back; z and out may be the same matrix.  (One warp per row walking it three
// times took 87 us for 300K x 47 and 243 us for 700K x 256.)
template <int LR, int NV>
__global__ void __launch_bounds__(256) log_softmax_fwd_kernel(const float* z, int64_t ldz, float* out, int64_t ldo, int64_t n, int N,
                                                              int vec4) {
  pdl_trigger();
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / LR) + threadIdx.x / LR;
  const int l = threadIdx.x % LR;
  const bool have = row < n;
  float v[NV * 4];
  bool live[NV * 4];
#pragma unroll
  for (int w = 0; w < NV; ++w) {
    const int c = (l + LR * w) * 4;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (have && c < N) t = load4_upto(z + row * ldz + c, N - c, vec4);
    v[4 * w] = t.x; v[4 * w + 1] = t.y; v[4 * w + 2] = t.z; v[4 * w + 3] = t.w;
#pragma unroll
    for (int j = 0; j < 4; ++j) live[4 * w + j] = c + j < N;
  }
  const float lse = row_lse<LR, NV * 4>(v, live);
  if (!have) return;
#pragma unroll
  for (int w = 0; w < NV; ++w) {
    const int c = (l + LR * w) * 4;
    if (c < N) store4_upto(out + row * ldo + c, make_float4(v[4 * w] - lse, v[4 * w + 1] - lse, v[4 * w + 2] - lse, v[4 * w + 3] - lse), N - c, vec4);
  }
}

// wider rows: one warp per row
__global__ void log_softmax_fwd_wide_kernel(const float* z, int64_t ldz, float* out, int64_t ldo, int64_t n, int N) {
  pdl_trigger();
  pdl_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  const float* zp = z + row * ldz;
  float mx = -INFINITY;
  for (int c = lane; c < N; c += 32) mx = fmaxf(mx, zp[c]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  float sum = 0.f;
  for (int c = lane; c < N; c += 32) sum += expf(zp[c] - mx);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  const float lse = mx + logf(sum);
  for (int c = lane; c < N; c += 32) out[row * ldo + c] = zp[c] - lse;
}

__global__ void log_softmax_bwd_kernel(const float* __restrict__ logp, int64_t ldl, const float* __restrict__ g,
                                       int64_t ldg, float* __restrict__ dz, int64_t lddz, int64_t n, int N) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  float sum = 0.f;
  for (int c = lane; c < N; c += 32) sum += g[row * ldg + c];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  for (int c = lane; c < N; c += 32) dz[row * lddz + c] = g[row * ldg + c] - expf(logp[row * ldl + c]) * sum;
}

// Pieces of a log-softmax whose rows are split over several processes: every process reduces its own
// columns, the per-row scalars are combined by a collective, then applied.   mode: 0 max, 1 sum,
// 2 sum of exp(z - ref[row]).  One warp per row.
__global__ void row_reduce_kernel(const float* __restrict__ z, int64_t ldz, int64_t n, int N, int mode,
                                  const float* __restrict__ ref, float* __restrict__ out) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  const float* zp = z + row * ldz;
  float acc = (mode == 0) ? -INFINITY : 0.f;
  const float r = (mode == 2) ? ref[row] : 0.f;
  for (int c = lane; c < N; c += 32) {
    const float v = zp[c];
    if (mode == 0) acc = fmaxf(acc, v);
    else if (mode == 1) acc += v;
    else acc += expf(v - r);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_xor_sync(0xffffffffu, acc, off);
    acc = (mode == 0) ? fmaxf(acc, o) : acc + o;
  }
  if (lane == 0) out[row] = acc;
}

// mode 0: out = z - a[row] - log(b[row])        (log-softmax from the global row max a and sum b)
// mode 1: out = g - exp(z) * a[row]             (its backward from log-probabilities z and the global row sum a of g)
__global__ void row_apply_kernel(const float* __restrict__ z, int64_t ldz, const float* __restrict__ g, int64_t ldg,
                                 const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out,
                                 int64_t ldo, int64_t n, int N, int mode) {
  const int64_t total = n * N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / N;
    const int c = static_cast<int>(i - r * N);
    if (mode == 0) out[r * ldo + c] = z[r * ldz + c] - a[r] - logf(b[r]);
    else out[r * ldo + c] = g[r * ldg + c] - expf(z[r * ldz + c]) * a[r];
  }
}

// ------------------------------------------------------------------------------------------------
constexpr int kNllBlocks = 1024;

__global__ void __launch_bounds__(256) nll_partial_kernel(const float* __restrict__ logp, int64_t ldl,
                                                          const int64_t* __restrict__ y,
                                                          const uint8_t* __restrict__ mask, int64_t n, int N, int cls_lo,
                                                          int cls_hi, float gval, float* __restrict__ grad, int64_t ldg,
                                                          float* __restrict__ partial) {
  __shared__ float red[256];
  float s = 0.f;
  const int64_t total = n * N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / N;
    const int c = static_cast<int>(i - r * N);
    const int64_t label = y[r];
    const bool hit = mask[r] && label >= cls_lo && label < cls_hi && (label - cls_lo) == c;
    if (hit) s += logp[r * ldl + c];
    if (grad) grad[r * ldg + c] = hit ? gval : 0.f;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void nll_final_kernel(const float* __restrict__ partial, int blocks, float count, float* __restrict__ loss) {
  __shared__ float red[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < blocks; i += 256) s += partial[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = -red[0] / count;
}

// Loss and gradient of a masked NLL on log-probabilities, taken straight to the gradient before the log-softmax:
//   dz[i, j] = (row i is trained on) ? (exp(logp[i, j]) - [j == y_i]) / count : 0,     partial sums of -logp[i, y_i]
// which is log_softmax_bwd of nll's one-hot gradient without writing, scaling and reading that n x N matrix (four passes
// over it: 0.70M rows x 256 classes 0.47 + 0.46 + 0.32 ms).  One thread per four columns: one 16-byte read and write.
__global__ void __launch_bounds__(256) nll_softmax_bwd_kernel(const float* __restrict__ logp, int64_t ldl,
                                                              const int64_t* __restrict__ y, const uint8_t* __restrict__ mask,
                                                              int64_t n, int N, int vecs, int cls_lo, int cls_hi, float inv_count,
                                                              float* __restrict__ dz, int64_t lddz, float* __restrict__ partial,
                                                              int vec4) {
  __shared__ float red[8];
  pdl_trigger();
  pdl_wait();
  float s = 0.f;
  const int64_t total = n * vecs;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = total <= INT_MAX ? static_cast<int>(i) / vecs : i / vecs;
    const int c = static_cast<int>(i - r * vecs) * 4;
    const int64_t label = __ldg(y + r);
    const bool hit = __ldg(mask + r) && label >= cls_lo && label < cls_hi;
    const int at = hit ? static_cast<int>(label - cls_lo) - c : -1;      // the label's place among these four columns
    float g[4] = {0.f, 0.f, 0.f, 0.f};
    const int live = min(4, N - c);
    if (hit) {
      float l[4] = {0.f, 0.f, 0.f, 0.f};
      if (vec4 && live == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(logp + r * ldl + c));
        l[0] = t.x; l[1] = t.y; l[2] = t.z; l[3] = t.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < live) l[j] = __ldg(logp + r * ldl + c + j);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // g - exp(logp) * rowsum(g) with g = -1 / count at the label, 0 elsewhere
        g[j] = (j == at ? -inv_count : 0.f) + expf(l[j]) * inv_count;
        if (j == at) s += l[j];
      }
    }
    float* o = dz + r * lddz + c;
    if (vec4 && live == 4) {
      *reinterpret_cast<float4*>(o) = make_float4(g[0], g[1], g[2], g[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < live) o[j] = g[j];
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// log_softmax_fwd_kernel followed by nll_softmax_bwd_kernel on its result, in one pass over z (300K x 47: 45 + 31 us for the two, which
// read z, write and read logp and write dz; 26 us of HBM time are left).
template <int LR, int NV>
__global__ void __launch_bounds__(256) log_softmax_nll_kernel(const float* z, int64_t ldz, float* out, int64_t ldo, const int64_t* __restrict__ y,
                                                              const uint8_t* __restrict__ mask, int64_t n, int N, int cls_lo, int cls_hi,
                                                              float inv_count, float* __restrict__ dz, int64_t lddz,
                                                              float* __restrict__ partial, int vec4) {
  __shared__ float red[8];
  pdl_trigger();
  pdl_wait();
  const int l = threadIdx.x % LR;
  float picked = 0.f;
  for (int64_t row0 = static_cast<int64_t>(blockIdx.x) * (256 / LR); row0 < n; row0 += static_cast<int64_t>(gridDim.x) * (256 / LR)) {
    const int64_t row = row0 + threadIdx.x / LR;
    const bool have = row < n;
    int at = -1;
    if (have && __ldg(mask + row)) {
      const int64_t label = __ldg(y + row);
      if (label >= cls_lo && label < cls_hi) at = static_cast<int>(label - cls_lo);
    }
    float v[NV * 4];
    bool live[NV * 4];
#pragma unroll
    for (int w = 0; w < NV; ++w) {
      const int c = (l + LR * w) * 4;
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (have && c < N) t = load4_upto(z + row * ldz + c, N - c, vec4);
      v[4 * w] = t.x; v[4 * w + 1] = t.y; v[4 * w + 2] = t.z; v[4 * w + 3] = t.w;
#pragma unroll
      for (int j = 0; j < 4; ++j) live[4 * w + j] = c + j < N;
    }
    const float lse = row_lse<LR, NV * 4>(v, live);
    if (!have) continue;
#pragma unroll
    for (int w = 0; w < NV; ++w) {
      const int c = (l + LR * w) * 4;
      float g[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[4 * w + j] -= lse;
        if (at >= 0) g[j] = (c + j == at ? -inv_count : 0.f) + expf(v[4 * w + j]) * inv_count;
        if (c + j == at) picked += v[4 * w + j];
      }
      if (c < N) {
        store4_upto(out + row * ldo + c, make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]), N - c, vec4);
        store4_upto(dz + row * lddz + c, make_float4(g[0], g[1], g[2], g[3]), N - c, vec4);
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) picked += __shfl_xor_sync(0xffffffffu, picked, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = picked;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// The end of an epoch in one launch (4 launches of 2 - 4 us before): the two weight gradients from their partial products, Adam on
// both weights (torch.optim.Adam with its default options: the same operations in the same order), and the loss from its
// partial sums, loss = -sum / count.  Blocks of 32 gradient elements, then one block for the loss.
struct EpochTailTensor {
  const float* ws;                   // partial products, `chunks` of K x N
  int chunks, K, N, transposed;      // transposed: of the gradient's transpose
  float *g, *p, *m, *v;              // gradient; weight and moments (p null: no optimizer step)
};
struct EpochTailArgs {
  EpochTailTensor t[2];
  float beta1, beta2, eps, step_size, bias2_sqrt;
  const float* partial;
  int parts;
  float count;
  float* loss;
};
__global__ void __launch_bounds__(256) epoch_tail_kernel(EpochTailArgs a) {
  __shared__ float red[8][32];
  pdl_trigger();
  pdl_wait();
  const int b0 = (a.t[0].K * a.t[0].N + 31) / 32, b1 = (a.t[1].K * a.t[1].N + 31) / 32;
  const int blk = blockIdx.x;
  if (blk < b0 + b1) {
    const EpochTailTensor& t = a.t[blk < b0 ? 0 : 1];
    const int idx = (blk < b0 ? blk : blk - b0) * 32 + (threadIdx.x & 31);
    const float g = tn_sum(t.ws, t.chunks, t.K * t.N, idx, red);
    if (threadIdx.x >= 32 || idx >= t.K * t.N) return;
    const int k = t.transposed ? idx % t.N * t.K + idx / t.N : idx;
    t.g[k] = g;
    if (!t.p) return;
    float m = t.m[k], v = t.v[k];
    m += (1.f - a.beta1) * (g - m);
    v = v * a.beta2 + (1.f - a.beta2) * g * g;
    t.m[k] = m;
    t.v[k] = v;
    t.p[k] -= a.step_size * (m / (sqrtf(v) / a.bias2_sqrt + a.eps));
    return;
  }
  __shared__ float sums[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < a.parts; i += 256) s += a.partial[i];
  sums[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sums[threadIdx.x] += sums[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *a.loss = -sums[0] / a.count;
}

static int elementwise_blocks(int64_t total) {
  int64_t b = (total + 255) / 256;
  const int64_t cap = 32 * kNumSMs;
  return static_cast<int>(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace cagnet

using namespace cagnet;

// Row tiles are as tall as W is narrow (8 rows per thread); below about two tiles per SM, with a K worth splitting, the warps of
// a block share its rows and split K instead.
static bool gemm_splits_k(int64_t n, int K, int N, int epilogue) {
  return N <= 64 && K >= 64 && n < 40000 && epilogue != CAGNET_EPI_LOG_SOFTMAX_256;
}
static int gemm_fma_rows(int64_t n, int N) {
  if (N <= 16) return n < 20000 ? 64 : n < 160000 ? 128 : 256;
  if (N <= 32) return n < 80000 ? 32 : 128;
  return N <= 64 ? 128 : 64;
}
template <bool NLL>
static cudaError_t launch_gemm_fma(const GemmArgs& a, cudaStream_t s) {
  const int64_t n = a.n;
  const int N = a.N;
  auto rows = [&](int bm) { return dim3(static_cast<unsigned>((n + bm - 1) / bm), 1); };
  if constexpr (!NLL) {
    if (gemm_splits_k(n, a.K, N, a.epilogue)) {
      if (N <= 16) return launch_pdl(gemm_nn_splitk_kernel<4, 2>, rows(16), dim3(256), 0, s, a);
      if (N <= 32) return launch_pdl(gemm_nn_splitk_kernel<8, 4>, rows(16), dim3(256), 0, s, a);
      return launch_pdl(gemm_nn_splitk_kernel<16, 8>, rows(16), dim3(256), 0, s, a);
    }
  }
  const int bm = gemm_fma_rows(n, N);
  if (N <= 16) {
    if (bm == 64) return launch_pdl(gemm_nn_kernel<4, 1, 2, 4, 32, NLL>, rows(bm), dim3(128), 0, s, a);
    if (bm == 128) return launch_pdl(gemm_nn_kernel<4, 1, 4, 4, 32, NLL>, rows(bm), dim3(128), 0, s, a);
    return launch_pdl(gemm_nn_kernel<4, 1, 8, 4, 16, NLL>, rows(bm), dim3(128), 0, s, a);
  }
  if (N <= 32) {
    if (bm == 32) return launch_pdl(gemm_nn_kernel<8, 1, 2, 4, 32, NLL>, rows(bm), dim3(128), 0, s, a);
    return launch_pdl(gemm_nn_kernel<8, 1, 8, 4, 32, NLL>, rows(bm), dim3(128), 0, s, a);
  }
  if (N <= 64) return launch_pdl(gemm_nn_kernel<16, 1, 8, 8, 32, NLL>, rows(bm), dim3(256), 0, s, a);
  if (N <= 128) return launch_pdl(gemm_nn_kernel<32, 1, 8, 8, 16, NLL>, rows(bm), dim3(256), 0, s, a);
  dim3 grid = rows(bm);
  grid.y = (N + 255) / 256;
  return launch_pdl(gemm_nn_kernel<32, 2, 8, 8, 16, NLL>, grid, dim3(256), 0, s, a);
}

extern "C" int cagnet_gemm_nn_f32(const float* X, int64_t ldx, const float* W, int64_t ldw, int32_t transW, float* Z,
                                  int64_t ldz, int64_t n, int32_t K, int32_t N, int32_t epilogue, const float* aux,
                                  int64_t ldaux, void* stream) {
  if (n < 0 || K < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!X || !W || !Z) return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: null pointer");
  if (epilogue < 0 || epilogue > 5) return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: unknown epilogue");
  if (epilogue == CAGNET_EPI_RELU_MASK && (!aux || ldaux < N))
    return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: the ReLU-mask epilogue needs aux (n x N)");
  if (epilogue == CAGNET_EPI_LOG_SOFTMAX && N > 64)
    return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: fused log-softmax supports N <= 64 (got %s%lld)", "", N);
  if (epilogue == CAGNET_EPI_LOG_SOFTMAX_256 && N > 256)
    return fail(CAGNET_E_ARG, "cagnet_gemm_nn_f32: fused log-softmax supports N <= 256 (got %s%lld)", "", N);
  if (ldx < K || ldz < N || ldw < (transW ? K : N))
    return fail(CAGNET_E_ALIGN, "cagnet_gemm_nn_f32: leading dimension smaller than the row width");
  if ((n + 15) / 16 > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_gemm_nn_f32: too many rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (gemm_nn_tc_applies(X, ldx, n, K, N, epilogue)) return gemm_nn_tc(X, ldx, W, ldw, transW, Z, ldz, n, K, N, epilogue, aux, ldaux, s);
  GemmArgs a;
  a.X = X; a.W = W; a.aux = aux; a.Z = Z;
  a.ldx = ldx; a.ldw = ldw; a.ldz = ldz; a.ldaux = ldaux; a.n = n;
  a.transW = transW; a.K = K; a.N = N; a.epilogue = epilogue;
  a.x_vec4 = (ldx % 4 == 0 && aligned(X, 16)) ? 1 : 0;
  a.z_vec4 = (ldz % 4 == 0 && aligned(Z, 16)) ? 1 : 0;
  const cudaError_t e = launch_gemm_fma<false>(a, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_nn_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

extern "C" size_t cagnet_gemm_tn_workspace_bytes(int64_t n, int32_t K, int32_t N) {
  if (n < 0 || K <= 0 || N <= 0) return 0;
  const int chunks = max(max(tn_shape(n, K, N).chunks, tn_shape(n, N, K).chunks), kNumSMs);     // either operand order, either kernel
  return sizeof(float) * static_cast<size_t>(chunks) * K * N;
}

// The small-N kernel needs 80 KB of dynamic shared memory: opt in once per device.
static int tn_small_opt_in() {
  static bool opted_in[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !opted_in[dev]) {
    if (cudaFuncSetAttribute(gemm_tn_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTnSmallSmemBytes) !=
        cudaSuccess)
      return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: cannot reserve shared memory for the small-N kernel");
    opted_in[dev] = true;
  }
  return CAGNET_OK;
}

static int launch_tn_small(const TnSmallArgs& a, const TnSmallArgs& b, int64_t n, cudaStream_t s) {
  if (int rc = tn_small_opt_in()) return rc;
  const cudaError_t e = launch_pdl(gemm_tn_small_kernel, dim3(a.chunks * a.ktiles + b.chunks * b.ktiles), dim3(256), kTnSmallSmemBytes, s, a, b, n);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

// The partial products of H^T * G in ws, and what it takes to add them up.  With `later` the narrow kernel is not launched but
// its arguments are left there (later->chunks stays 0 where another kernel ran).
static int tn_partials(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int32_t K, int32_t N, void* ws,
                       size_t ws_bytes, cagnet_tn_sum* sum, cudaStream_t s, TnSmallArgs* later = nullptr) {
  if (!ws || (n > 0 && (!H || !G))) return fail(CAGNET_E_ARG, "cagnet_gemm_tn_f32: null pointer");
  if (ldh < K || ldg < N) return fail(CAGNET_E_ALIGN, "cagnet_gemm_tn_f32: leading dimension too small");
  if (static_cast<int64_t>(K) * N > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_gemm_tn_f32: K*N exceeds int32");
  if (ws_bytes < cagnet_gemm_tn_workspace_bytes(n, K, N))
    return fail(CAGNET_E_WORKSPACE, "cagnet_gemm_tn_f32: workspace of %s%lld bytes is too small (need %lld)", "",
                (long long)ws_bytes, (long long)cagnet_gemm_tn_workspace_bytes(n, K, N));
  float* partials = static_cast<float*>(ws);
  sum->partials = partials;
  if (gemm_tn_tc_applies(H, ldh, G, ldg, n, K, N)) {
    sum->chunks = gemm_tn_tc_blocks(n, K, N);
    sum->K = max(K, N); sum->N = min(K, N);
    sum->transposed = K < N ? 1 : 0;
    return gemm_tn_tc(H, ldh, G, ldg, n, K, N, partials, s);
  }
  const bool rows_aligned = ldh % 4 == 0 && ldg % 4 == 0 && aligned(H, 16) && aligned(G, 16);
  // a narrow H against a wider G (the 16 x 41 weight gradient): the small-N kernel computes G^T * H
  const bool small = (N <= 16 || K <= 16) && rows_aligned, swap = small && N > 16;
  if (swap) {
    const float* h = H; H = G; G = h;
    const int64_t l = ldh; ldh = ldg; ldg = l;
    const int32_t k = K; K = N; N = k;
  }
  const TnShape sh = tn_shape(n, K, N);
  sum->chunks = sh.chunks;
  sum->K = K; sum->N = N;
  sum->transposed = swap ? 1 : 0;
  cudaError_t e;
  if (small) {
    const TnSmallArgs a{H, G, partials, ldh, ldg, sh.rows_per_chunk, K, N, sh.chunks, sh.ktiles};
    if (later) {
      *later = a;
      return CAGNET_OK;
    }
    return launch_tn_small(a, TnSmallArgs{}, n, s);
  }
  e = launch_pdl(gemm_tn_partial_kernel, dim3(sh.chunks, sh.ktiles, sh.ntiles), dim3(256), 0, s, H, ldh, G, ldg, n, K, N,
                 sh.rows_per_chunk, partials);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

extern "C" int cagnet_gemm_tn_f32(const float* H, int64_t ldh, const float* G, int64_t ldg, float* out, int64_t ldo,
                                  int64_t n, int32_t K, int32_t N, float beta, void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || K < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_gemm_tn_f32: negative size");
  if (K == 0 || N == 0) return CAGNET_OK;
  if (beta != 0.f && beta != 1.f) return fail(CAGNET_E_ARG, "cagnet_gemm_tn_f32: beta must be 0 or 1");
  if (!out) return fail(CAGNET_E_ARG, "cagnet_gemm_tn_f32: null pointer");
  if (ldo < N) return fail(CAGNET_E_ALIGN, "cagnet_gemm_tn_f32: leading dimension too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cagnet_tn_sum sum;
  if (int rc = tn_partials(H, ldh, G, ldg, n, K, N, ws, ws_bytes, &sum, s)) return rc;
  launch_pdl(gemm_tn_reduce_kernel, dim3((K * N + 31) / 32), dim3(256), 0, s, sum.partials, sum.chunks, sum.K, sum.N, out, ldo, beta,
             sum.transposed);
  return check_launch("cagnet_gemm_tn_f32");
}

extern "C" int cagnet_gemm_tn_partials_f32(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int32_t K, int32_t N,
                                           void* ws, size_t ws_bytes, cagnet_tn_sum* sum, void* stream) {
  if (n < 0 || K <= 0 || N <= 0 || !sum) return fail(CAGNET_E_ARG, "cagnet_gemm_tn_partials_f32: bad argument");
  return tn_partials(H, ldh, G, ldg, n, K, N, ws, ws_bytes, sum, static_cast<cudaStream_t>(stream));
}

extern "C" int cagnet_gemm_tn_partials2_f32(const cagnet_tn_product* p, cagnet_tn_sum* sum, int64_t n, int32_t* launches, void* stream) {
  if (n < 0 || !p || !sum || !launches || p[0].K <= 0 || p[0].N <= 0 || p[1].K <= 0 || p[1].N <= 0)
    return fail(CAGNET_E_ARG, "cagnet_gemm_tn_partials2_f32: bad argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  TnSmallArgs later[2] = {};
  *launches = 0;
  for (int i = 0; i < 2; ++i) {
    if (int rc = tn_partials(p[i].H, p[i].ldh, p[i].G, p[i].ldg, n, p[i].K, p[i].N, p[i].ws, p[i].ws_bytes, sum + i, s, later + i)) return rc;
    *launches += later[i].chunks == 0;
  }
  if (later[0].chunks == 0 && later[1].chunks == 0) return CAGNET_OK;
  ++*launches;
  return later[0].chunks ? launch_tn_small(later[0], later[1], n, s) : launch_tn_small(later[1], TnSmallArgs{}, n, s);
}

extern "C" int cagnet_relu_fwd_f32(const float* z, int64_t ldz, float* h, int64_t ldh, int64_t n, int32_t N,
                                   void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_relu_fwd_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!z || !h || ldz < N || ldh < N) return fail(CAGNET_E_ARG, "cagnet_relu_fwd_f32: bad argument");
  const int vecs = (N + 3) / 4, vec4 = (ldz % 4 == 0 && ldh % 4 == 0 && aligned(z, 16) && aligned(h, 16)) ? 1 : 0;
  launch_pdl(relu_fwd_kernel, dim3(elementwise_blocks(n * vecs)), dim3(256), 0, static_cast<cudaStream_t>(stream), z, ldz, h, ldh, n, N, vecs, vec4);
  return check_launch("cagnet_relu_fwd_f32");
}

extern "C" int cagnet_relu_bwd_f32(const float* h, int64_t ldh, const float* g, int64_t ldg, float* dz, int64_t lddz,
                                   int64_t n, int32_t N, void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_relu_bwd_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!h || !g || !dz || ldh < N || ldg < N || lddz < N) return fail(CAGNET_E_ARG, "cagnet_relu_bwd_f32: bad argument");
  const int vecs = (N + 3) / 4;
  const int vec4 = (ldh % 4 == 0 && ldg % 4 == 0 && lddz % 4 == 0 && aligned(h, 16) && aligned(g, 16) && aligned(dz, 16)) ? 1 : 0;
  launch_pdl(relu_bwd_kernel, dim3(elementwise_blocks(n * vecs)), dim3(256), 0, static_cast<cudaStream_t>(stream), h, ldh, g, ldg, dz, lddz, n, N,
             vecs, vec4);
  return check_launch("cagnet_relu_bwd_f32");
}

extern "C" int cagnet_log_softmax_fwd_f32(const float* z, int64_t ldz, float* logp, int64_t ldl, int64_t n, int32_t N,
                                          void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_log_softmax_fwd_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!z || !logp || ldz < N || ldl < N) return fail(CAGNET_E_ARG, "cagnet_log_softmax_fwd_f32: bad argument");
  if ((n + 7) / 8 > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_log_softmax_fwd_f32: too many rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int vec4 = (ldz % 4 == 0 && ldl % 4 == 0 && aligned(z, 16) && aligned(logp, 16)) ? 1 : 0;
  const int vecs = (N + 3) / 4;
  auto rows = [&](int lanes) { return dim3(static_cast<unsigned>((n + 256 / lanes - 1) / (256 / lanes))); };
  if (vecs <= 4) launch_pdl(log_softmax_fwd_kernel<4, 1>, rows(4), dim3(256), 0, s, z, ldz, logp, ldl, n, N, vec4);
  else if (vecs <= 8) launch_pdl(log_softmax_fwd_kernel<8, 1>, rows(8), dim3(256), 0, s, z, ldz, logp, ldl, n, N, vec4);
  else if (vecs <= 16) launch_pdl(log_softmax_fwd_kernel<8, 2>, rows(8), dim3(256), 0, s, z, ldz, logp, ldl, n, N, vec4);
  else if (vecs <= 32) launch_pdl(log_softmax_fwd_kernel<16, 2>, rows(16), dim3(256), 0, s, z, ldz, logp, ldl, n, N, vec4);
  else if (vecs <= 64) launch_pdl(log_softmax_fwd_kernel<32, 2>, rows(32), dim3(256), 0, s, z, ldz, logp, ldl, n, N, vec4);
  else launch_pdl(log_softmax_fwd_wide_kernel, rows(32), dim3(256), 0, s, z, ldz, logp, ldl, n, N);
  return check_launch("cagnet_log_softmax_fwd_f32");
}

extern "C" int cagnet_log_softmax_bwd_f32(const float* logp, int64_t ldl, const float* g, int64_t ldg, float* dz,
                                          int64_t lddz, int64_t n, int32_t N, void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_log_softmax_bwd_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!logp || !g || !dz || ldl < N || ldg < N || lddz < N)
    return fail(CAGNET_E_ARG, "cagnet_log_softmax_bwd_f32: bad argument");
  if ((n + 7) / 8 > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_log_softmax_bwd_f32: too many rows");
  log_softmax_bwd_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      logp, ldl, g, ldg, dz, lddz, n, N);
  return check_launch("cagnet_log_softmax_bwd_f32");
}

extern "C" int cagnet_row_reduce_f32(const float* z, int64_t ldz, int64_t n, int32_t N, int32_t mode, const float* ref,
                                     float* out, void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_row_reduce_f32: negative size");
  if (n == 0) return CAGNET_OK;
  if (mode < 0 || mode > 2 || !out || (N > 0 && !z) || (mode == 2 && !ref) || ldz < N)
    return fail(CAGNET_E_ARG, "cagnet_row_reduce_f32: bad argument");
  if ((n + 7) / 8 > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_row_reduce_f32: too many rows");
  row_reduce_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(z, ldz, n, N, mode,
                                                                                                     ref, out);
  return check_launch("cagnet_row_reduce_f32");
}

extern "C" int cagnet_log_softmax_apply_f32(const float* z, int64_t ldz, const float* row_max, const float* row_sum,
                                            float* logp, int64_t ldl, int64_t n, int32_t N, void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_log_softmax_apply_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!z || !row_max || !row_sum || !logp || ldz < N || ldl < N)
    return fail(CAGNET_E_ARG, "cagnet_log_softmax_apply_f32: bad argument");
  row_apply_kernel<<<elementwise_blocks(n * N), 256, 0, static_cast<cudaStream_t>(stream)>>>(z, ldz, nullptr, 0, row_max,
                                                                                           row_sum, logp, ldl, n, N, 0);
  return check_launch("cagnet_log_softmax_apply_f32");
}

extern "C" int cagnet_log_softmax_bwd_apply_f32(const float* logp, int64_t ldl, const float* g, int64_t ldg,
                                                const float* row_sum_g, float* dz, int64_t lddz, int64_t n, int32_t N,
                                                void* stream) {
  if (n < 0 || N < 0) return fail(CAGNET_E_ARG, "cagnet_log_softmax_bwd_apply_f32: negative size");
  if (n == 0 || N == 0) return CAGNET_OK;
  if (!logp || !g || !row_sum_g || !dz || ldl < N || ldg < N || lddz < N)
    return fail(CAGNET_E_ARG, "cagnet_log_softmax_bwd_apply_f32: bad argument");
  row_apply_kernel<<<elementwise_blocks(n * N), 256, 0, static_cast<cudaStream_t>(stream)>>>(logp, ldl, g, ldg, row_sum_g,
                                                                                           nullptr, dz, lddz, n, N, 1);
  return check_launch("cagnet_log_softmax_bwd_apply_f32");
}

extern "C" size_t cagnet_nll_workspace_bytes(int64_t n) {
  (void)n;
  return sizeof(float) * (kNllBlocks > kTcLossParts ? kNllBlocks : kTcLossParts);
}

extern "C" int cagnet_nll_masked_f32(const float* logp, int64_t ldl, const int64_t* y, const uint8_t* mask, int64_t n,
                                     int32_t N, int32_t cls_lo, int32_t cls_hi, float count, float scale,
                                     float* loss_dev, float* grad, int64_t ldg, void* ws, size_t ws_bytes,
                                     void* stream) {
  if (n < 0 || N <= 0) return fail(CAGNET_E_ARG, "cagnet_nll_masked_f32: bad size");
  if (!loss_dev || !ws || (n > 0 && (!logp || !y || !mask))) return fail(CAGNET_E_ARG, "cagnet_nll_masked_f32: null pointer");
  if (ldl < N || (grad && ldg < N)) return fail(CAGNET_E_ALIGN, "cagnet_nll_masked_f32: leading dimension too small");
  if (ws_bytes < cagnet_nll_workspace_bytes(n)) return fail(CAGNET_E_WORKSPACE, "cagnet_nll_masked_f32: workspace too small");
  if (!(count > 0.f)) return fail(CAGNET_E_ARG, "cagnet_nll_masked_f32: count must be positive");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int blocks = elementwise_blocks(n * N);
  if (blocks > kNllBlocks) blocks = kNllBlocks;
  nll_partial_kernel<<<blocks, 256, 0, s>>>(logp, ldl, y, mask, n, N, cls_lo, cls_hi, -scale / count, grad, ldg,
                                            static_cast<float*>(ws));
  nll_final_kernel<<<1, 256, 0, s>>>(static_cast<const float*>(ws), blocks, count, loss_dev);
  return check_launch("cagnet_nll_masked_f32");
}

// Blocks of the loss kernel = partial sums it leaves in ws (cagnet_nll_workspace_bytes).
static int nll_blocks(int64_t n, int vecs) {
  const int b = elementwise_blocks(n * vecs);
  return b > kNllBlocks ? kNllBlocks : b;
}

extern "C" int cagnet_nll_softmax_bwd_f32(const float* logp, int64_t ldl, const int64_t* y, const uint8_t* mask, int64_t n,
                                          int32_t N, int32_t cls_lo, int32_t cls_hi, float count, float* dz, int64_t lddz,
                                          int32_t* parts, void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || N <= 0) return fail(CAGNET_E_ARG, "cagnet_nll_softmax_bwd_f32: bad size");
  if (!parts || !ws || (n > 0 && (!logp || !y || !mask || !dz))) return fail(CAGNET_E_ARG, "cagnet_nll_softmax_bwd_f32: null pointer");
  if (ldl < N || lddz < N) return fail(CAGNET_E_ALIGN, "cagnet_nll_softmax_bwd_f32: leading dimension too small");
  if (ws_bytes < cagnet_nll_workspace_bytes(n)) return fail(CAGNET_E_WORKSPACE, "cagnet_nll_softmax_bwd_f32: workspace too small");
  if (!(count > 0.f)) return fail(CAGNET_E_ARG, "cagnet_nll_softmax_bwd_f32: count must be positive");
  const int vecs = (N + 3) / 4;
  const int vec4 = (ldl % 4 == 0 && lddz % 4 == 0 && aligned(logp, 16) && aligned(dz, 16)) ? 1 : 0;
  *parts = nll_blocks(n, vecs);
  launch_pdl(nll_softmax_bwd_kernel, dim3(*parts), dim3(256), 0, static_cast<cudaStream_t>(stream), logp, ldl, y, mask, n, N, vecs,
             cls_lo, cls_hi, 1.f / count, dz, lddz, static_cast<float*>(ws), vec4);
  return check_launch("cagnet_nll_softmax_bwd_f32");
}

extern "C" int cagnet_log_softmax_nll_f32(const float* z, int64_t ldz, int64_t n, int32_t N, const int64_t* y, const uint8_t* mask,
                                          int32_t cls_lo, int32_t cls_hi, float count, float* logp, int64_t ldl, float* dz, int64_t lddz,
                                          int32_t* parts, void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || N <= 0 || N > 256) return fail(CAGNET_E_ARG, "cagnet_log_softmax_nll_f32: bad size");
  if (!parts || !ws || (n > 0 && (!z || !logp || !y || !mask || !dz))) return fail(CAGNET_E_ARG, "cagnet_log_softmax_nll_f32: null pointer");
  if (ldz < N || ldl < N || lddz < N) return fail(CAGNET_E_ALIGN, "cagnet_log_softmax_nll_f32: leading dimension too small");
  if (ws_bytes < cagnet_nll_workspace_bytes(n)) return fail(CAGNET_E_WORKSPACE, "cagnet_log_softmax_nll_f32: workspace too small");
  if (!(count > 0.f)) return fail(CAGNET_E_ARG, "cagnet_log_softmax_nll_f32: count must be positive");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int vec4 = (ldz % 4 == 0 && ldl % 4 == 0 && lddz % 4 == 0 && aligned(z, 16) && aligned(logp, 16) && aligned(dz, 16)) ? 1 : 0;
  const int vecs = (N + 3) / 4;
  auto run = [&](auto kernel, int lanes) {
    const int64_t blocks = max(static_cast<int64_t>(1), (n + 256 / lanes - 1) / (256 / lanes));
    *parts = static_cast<int32_t>(min(blocks, static_cast<int64_t>(kTcLossParts)));
    launch_pdl(kernel, dim3(*parts), dim3(256), 0, s, z, ldz, logp, ldl, y, mask, n, N, cls_lo, cls_hi, 1.f / count, dz, lddz,
               static_cast<float*>(ws), vec4);
  };
  if (vecs <= 4) run(log_softmax_nll_kernel<4, 1>, 4);
  else if (vecs <= 8) run(log_softmax_nll_kernel<8, 1>, 8);
  else if (vecs <= 16) run(log_softmax_nll_kernel<8, 2>, 8);
  else if (vecs <= 32) run(log_softmax_nll_kernel<16, 2>, 16);
  else run(log_softmax_nll_kernel<32, 2>, 32);
  return check_launch("cagnet_log_softmax_nll_f32");
}

// One launch where one block has whole rows (on the tensor cores the epilogue has every row's log-probabilities at hand: 700K x 256 classes
// 596 us for the two, of which 110 us to read them back), two where K is split.
extern "C" int cagnet_gemm_nll_f32(const float* X, int64_t ldx, const float* W, int64_t ldw, int64_t n, int32_t K, int32_t N,
                                   const int64_t* y, const uint8_t* mask, int32_t cls_lo, int32_t cls_hi, float count, float* logp,
                                   int64_t ldl, float* dz, int64_t lddz, int32_t* parts, int32_t* launches, void* ws, size_t ws_bytes,
                                   void* stream) {
  if (n < 0 || K < 0 || N <= 0 || N > 256) return fail(CAGNET_E_ARG, "cagnet_gemm_nll_f32: bad size");
  if (!parts || !launches || !ws || (n > 0 && (!X || !W || !logp || !y || !mask || !dz))) return fail(CAGNET_E_ARG, "cagnet_gemm_nll_f32: null pointer");
  if (ldx < K || ldw < N || ldl < N || lddz < N) return fail(CAGNET_E_ALIGN, "cagnet_gemm_nll_f32: leading dimension too small");
  if (ws_bytes < cagnet_nll_workspace_bytes(n)) return fail(CAGNET_E_WORKSPACE, "cagnet_gemm_nll_f32: workspace too small");
  if (!(count > 0.f)) return fail(CAGNET_E_ARG, "cagnet_gemm_nll_f32: count must be positive");
  const int epilogue = N <= 64 ? CAGNET_EPI_LOG_SOFTMAX : CAGNET_EPI_LOG_SOFTMAX_256;
  if (gemm_nn_tc_applies(X, ldx, n, K, N, epilogue)) {
    *launches = 1;
    const TcLoss loss{y, mask, dz, static_cast<float*>(ws), lddz, cls_lo, cls_hi, 1.f / count};
    return gemm_nn_tc_nll(X, ldx, W, ldw, logp, ldl, n, K, N, loss, parts, static_cast<cudaStream_t>(stream));
  }
  const int64_t blocks = (n + gemm_fma_rows(n, N) - 1) / gemm_fma_rows(n, N);
  if (n > 0 && blocks <= kTcLossParts && !gemm_splits_k(n, K, N, epilogue)) {
    GemmArgs a = {};
    a.X = X; a.W = W; a.Z = logp;
    a.ldx = ldx; a.ldw = ldw; a.ldz = ldl; a.n = n;
    a.K = K; a.N = N; a.epilogue = epilogue;
    a.x_vec4 = (ldx % 4 == 0 && aligned(X, 16)) ? 1 : 0;
    a.z_vec4 = (ldl % 4 == 0 && lddz % 4 == 0 && aligned(logp, 16) && aligned(dz, 16)) ? 1 : 0;
    a.loss = TcLoss{y, mask, dz, static_cast<float*>(ws), lddz, cls_lo, cls_hi, 1.f / count};
    *launches = 1;
    *parts = static_cast<int32_t>(blocks);
    if (launch_gemm_fma<true>(a, static_cast<cudaStream_t>(stream)) != cudaSuccess) return check_launch("cagnet_gemm_nll_f32");
    return CAGNET_OK;
  }
  *launches = 2;
  if (int rc = cagnet_gemm_nn_f32(X, ldx, W, ldw, 0, logp, ldl, n, K, N, epilogue, nullptr, 0, stream)) return rc;
  return cagnet_nll_softmax_bwd_f32(logp, ldl, y, mask, n, N, cls_lo, cls_hi, count, dz, lddz, parts, ws, ws_bytes, stream);
}

extern "C" int cagnet_epoch_tail_f32(const cagnet_tn_sum* s1, float* g1, float* p1, float* m1, float* v1, const cagnet_tn_sum* s2,
                                     float* g2, float* p2, float* m2, float* v2, double lr, double beta1, double beta2, double eps,
                                     int64_t step, const float* loss_parts, int32_t parts, float count, float* loss, void* stream) {
  if (!s1 || !s2 || !g1 || !g2 || step < 1 || parts < 0 || (loss && (!loss_parts || !(count > 0.f))) ||
      (p1 && (!m1 || !v1)) || (p2 && (!m2 || !v2)))
    return fail(CAGNET_E_ARG, "cagnet_epoch_tail_f32: bad argument");
  const double bias1 = 1.0 - pow(beta1, static_cast<double>(step)), bias2 = 1.0 - pow(beta2, static_cast<double>(step));
  EpochTailArgs a;
  a.t[0] = EpochTailTensor{s1->partials, s1->chunks, s1->K, s1->N, s1->transposed, g1, p1, m1, v1};
  a.t[1] = EpochTailTensor{s2->partials, s2->chunks, s2->K, s2->N, s2->transposed, g2, p2, m2, v2};
  a.beta1 = static_cast<float>(beta1); a.beta2 = static_cast<float>(beta2); a.eps = static_cast<float>(eps);
  a.step_size = static_cast<float>(lr / bias1); a.bias2_sqrt = static_cast<float>(sqrt(bias2));
  a.partial = loss_parts; a.parts = parts; a.count = count; a.loss = loss;
  const int64_t blocks = (static_cast<int64_t>(s1->K) * s1->N + 31) / 32 + (static_cast<int64_t>(s2->K) * s2->N + 31) / 32 + (loss ? 1 : 0);
  launch_pdl(epoch_tail_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream), a);
  return check_launch("cagnet_epoch_tail_f32");
}
