// Tall-skinny fp32 products of the GCN layers on the tensor cores (tcgen05, sm_100a), fp32 in and out.
//
// Z = epilogue(X . W) with X n x K (n large) and W K x N small has 2 N flops per 4-byte element of X: on the FMA pipe it is
// bound by FMA issue and shared-memory reads from N = 16 on (233K x 602 x 16: 213 us against 88 us of HBM time; 700K x 16 x 256:
// 435 us against 116).  Here every element of X and W is cut into three bf16 terms (24 significant bits between them) and
// the six products that matter, x1 w1, x1 w2, x2 w1, x1 w3, x2 w2, x3 w1, go to the tensor pipe with fp32 sums; what is
// dropped is below 2^-25 of a product.  Error against fp64: as the FMA kernels' (1e-7 of the norm).
//   warp 0        TMA boxes of 128 rows x 32 columns of X into a ring of stages (128-byte swizzle; rows and columns outside
//                 the matrix arrive as zeros)
//   warps 12 - 27 four groups take the boxes in turn: a thread reads its row's 128 bytes, splits them and stores the three
//                 terms to TENSOR memory, where the multiply takes its A operand from (K <= 64: warps 20 - 27, two groups)
//   warp 1        tcgen05.mma kind::f16, M = 128, against W's terms, which stay in shared memory (K-major, 128-byte swizzle) for
//                 the block's whole run
//   warps 4 - 11  sums out of tensor memory (K <= 64: warps 4 - 19), epilogue, whole row segments to Z through a shared-memory
//                 exchange; the sums are given back to warp 1 as soon as they are read, before they are stored
// Blocks are persistent over row tiles.  With K <= 64 a tile has two boxes at most and the time is the epilogue's, which is
// why it gets twice the warps there (300K x 47 x 64 with the ReLU mask: 138 us with 8 storing warps that asked for the mask
// after the sums were there and kept the sums until everything was stored).
#include <cuda.h>
#include <limits.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "tc.cuh"

namespace cagnet {

constexpr int kXStageBytes = 128 * 128;           // 128 rows x 32 floats
constexpr int kTcThreads = 896;
constexpr int kTcMaxStages = 8;
constexpr int kTcSmem = 226 * 1024;
constexpr int kTcMaxW = 124 * 1024;               // W's terms
constexpr int kTcMaxBuffers = 4;                  // operand buffers of 3 terms x 16 tensor-memory columns
constexpr int kTcBufferCols = 48;
constexpr int kTcLightK = 64;
constexpr int kTcSlots = 4;                       // row tiles whose sums are kept at a time, at most

// Storing warps of a block, and columns that one takes at a time (an exchange of 32 rows, padded by 4 floats).
__host__ __device__ constexpr int tc_storing_warps(int sets) { return sets == 0 ? 16 : 8; }
__host__ __device__ constexpr bool tc_reads_old(int epilogue) { return epilogue == CAGNET_EPI_RELU_MASK || epilogue == CAGNET_EPI_ACCUMULATE; }
__host__ __device__ constexpr int tc_piece(bool old) { return old ? 16 : 32; }        // (32 columns of old values in flight spill: 620 bytes)
__host__ __device__ constexpr int tc_exchange_bytes(int sets, bool old) { return tc_storing_warps(sets) * 32 * (tc_piece(old) + 4) * 4; }
constexpr int kEpiNll = 6;                        // log-softmax, its masked NLL and the gradient before the log-softmax

struct TcArgs {
  const float* W;
  const float* aux;
  float* Z;
  int64_t ldw, ldz, ldaux, n;
  int transW, K, N, NP, z_vec4, aux_vec4, stages, tiles;
  TcLoss loss;
};

__device__ int g_gemm_error;

// 16 columns of this thread's row: the three sums of each in SETS sets, or (SETS = 0) a single sum.
template <int SETS>
__device__ __forceinline__ void load_sums(unsigned at, int NP, float (&v)[16]) {
  unsigned x[16];
  tmem_ld16(at, x);
  if constexpr (SETS > 0) {
    unsigned y[16], z[16];
    tmem_ld16(at + NP, y);
    tmem_ld16(at + 2 * NP, z);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(x[i]) + (__uint_as_float(y[i]) + __uint_as_float(z[i]));
    if constexpr (SETS == 2) {
      tmem_ld16(at + 3 * NP, x);
      tmem_ld16(at + 4 * NP, y);
      tmem_ld16(at + 5 * NP, z);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(x[i]) + (__uint_as_float(y[i]) + __uint_as_float(z[i]));
    }
  } else {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(x[i]);
  }
}

// Barrier of the `threads` threads that share `id`, and whether `ok` holds for all of them.
__device__ __forceinline__ bool group_and(bool ok, int id, int threads) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1u : 0u), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}

// SETS > 0: the terms of W side by side, three sums of NP columns (x1 w1 | x1 w2 + x2 w1 | x1 w3 + x2 w2 + x3 w1) that three
// products of N = 3 NP, 2 NP, NP per k step fill; SETS = 0 (K <= 64): all products into one sum, which leaves room for more
// row tiles in tensor memory and a third of it to read.  An addition in tensor memory drops what does not fit (1.7e-8 of
// the sum on average, always towards zero), so the number of additions to a full-sized sum is kept at the size of fp32
// rounding: SETS = 0 adds the five small products of all k first, K > 320 alternates between two sets of sums.
template <int SETS, int EPI>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_nn_tc_kernel(const __grid_constant__ CUtensorMap map, TcArgs a) {
  constexpr bool LIGHT = SETS == 0;
  constexpr int STORING = tc_storing_warps(SETS), EXPAND = 4 + STORING, GROUPS = (kTcThreads / 32 - EXPAND) / 4;
  extern __shared__ __align__(1024) char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * kTcMaxStages + 2 * kTcMaxBuffers + 2 * kTcSlots + 1];
  __shared__ unsigned tmem_base_s;
  __shared__ int dead_s;
  char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = a.stages, NP = a.NP;
  const int BUF = LIGHT && S < kTcMaxBuffers ? 2 : kTcMaxBuffers;       // a power of two, not above S (see the expanding warps)
  const int kblocks = (a.K + 63) / 64, ksteps = (a.K + 31) / 32;
  const int wtile = 3 * NP * 128;                 // W's terms for 64 k
  char* wsm = smem + S * kXStageBytes;
  float* xch_all = reinterpret_cast<float*>(wsm + kblocks * wtile);
  const int sums = SETS > 0 ? 3 * NP * SETS : NP;   // tensor-memory columns of a row tile's sums
  // Row tiles whose sums fit at a time.  LIGHT: as many tiles are stored side by side, by PARTS warps per 32 rows each, as one
  // tile's epilogue is a chain of waits (233K x 16 x 41, log-softmax: 38 us with one tile at a time); else all warps take every
  // tile.
  const int room = 512 - BUF * kTcBufferCols;
  const int AS = LIGHT && kTcSlots * sums <= room ? kTcSlots : 2 * sums <= room ? 2 : 1;
  const int PARTS = LIGHT ? STORING / 4 / AS : STORING / 4;
  const unsigned bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8 * s; };
  auto empty = [&](int s) { return bar0 + 8 * (kTcMaxStages + s); };
  auto a_full = [&](int b) { return bar0 + 8 * (2 * kTcMaxStages + b); };
  auto a_empty = [&](int b) { return bar0 + 8 * (2 * kTcMaxStages + BUF + b); };
  auto acc_full = [&](int c) { return bar0 + 8 * (2 * kTcMaxStages + 2 * BUF + c); };
  auto acc_empty = [&](int c) { return bar0 + 8 * (2 * kTcMaxStages + 2 * BUF + kTcSlots + c); };
  const unsigned drain = bar0 + 8 * (2 * kTcMaxStages + 2 * BUF + 2 * kTcSlots);
  volatile int* dead = &dead_s;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 4);        // one arrival per warp of the group that read the stage
    }
    for (int b = 0; b < BUF; ++b) {
      mbar_init(a_full(b), 4);
      mbar_init(a_empty(b), 1);
    }
    for (int c = 0; c < AS; ++c) {
      mbar_init(acc_full(c), 1);
      mbar_init(acc_empty(c), 4 * PARTS);
    }
    mbar_init(drain, 1);
    dead_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_trigger();
  pdl_wait();
  // W's terms: row (term NP + j) of k block q holds W[64 q .., j], 16-byte pieces permuted by the row
  const int n0 = blockIdx.y * NP;
  for (int i = threadIdx.x; i < kblocks * 8 * NP; i += blockDim.x) {
    const int j = i % NP, c = i / NP % 8, q = i / (8 * NP);
    __align__(16) unsigned short y[3][8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int k = q * 64 + c * 8 + t, col = n0 + j;
      float w = 0.f;
      if (k < a.K && col < a.N) w = __ldg(a.W + (a.transW ? static_cast<int64_t>(col) * a.ldw + k : static_cast<int64_t>(k) * a.ldw + col));
      split3(w, y[0][t], y[1][t], y[2][t]);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int row = p * NP + j;
      *reinterpret_cast<uint4*>(wsm + q * wtile + row * 128 + ((c ^ (row & 7)) << 4)) = *reinterpret_cast<const uint4*>(y[p]);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base_s;
  const unsigned a_col = 512 - BUF * kTcBufferCols;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0, issued = 0;
      unsigned ph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x) {
        for (int k = 0; k < ksteps && ok; ++k) {
          ok = mbar_wait(empty(s), ph ^ 1, dead);
          if (!ok) break;
          mbar_expect(full(s), kXStageBytes);
          tma_load_2d(smem_u32(smem + s * kXStageBytes), &map, k * 32, t * 128, full(s));
          ++issued;
          if (++s == S) { s = 0; ph ^= 1; }
        }
      }
      if (*dead) {        // a wait ran out: the copies in flight still write into this block's shared memory
        for (int k = max(0, issued - S); k < issued; ++k)
          for (int i = 0; i < kWaitLimit && !mbar_try(full(k % S), (k / S) & 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const unsigned base = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);      // D fp32, A and B bf16, K-major, M = 128
      auto idesc = [&](int N) { return base | (static_cast<unsigned>(N >> 3) << 17); };
      const unsigned i3 = idesc(3 * NP), i2 = idesc(2 * NP), i1 = idesc(NP);
      const unsigned term = static_cast<unsigned>(NP * 128) >> 4;
      int b = 0, c = 0;
      unsigned aph = 0, cph = 0;
      if constexpr (LIGHT) {
        bool ok = true;
        for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x) {
          const unsigned d = tmem + c * sums;
          const int b1 = (b + 1) & (BUF - 1);
          const unsigned aph1 = b1 ? aph : aph ^ 1;
          auto multiply = [&](int k, int buffer, bool large) {
            const unsigned long long w = smem_desc(smem_u32(wsm) + k * 64);
            const unsigned at = tmem + a_col + buffer * kTcBufferCols;
            for (int ks = 0; ks < 2 && k * 32 + ks * 16 < a.K; ++ks) {
              const unsigned x1 = at + ks * 8, x2 = x1 + 16, x3 = x1 + 32;
              const unsigned long long w1 = w + ks * 2, w2 = w1 + term, w3 = w2 + term;
              if (large) {
                tc_mma_ts(d, x1, w1, i1, 1u);
              } else {
                tc_mma_ts(d, x3, w1, i1, k + ks > 0 ? 1u : 0u);
                tc_mma_ts(d, x2, w2, i1, 1u);
                tc_mma_ts(d, x1, w3, i1, 1u);
                tc_mma_ts(d, x2, w1, i1, 1u);
                tc_mma_ts(d, x1, w2, i1, 1u);
              }
            }
          };
          ok = mbar_wait(acc_empty(c), cph ^ 1, dead) && mbar_wait(a_full(b), aph, dead);
          if (!ok) break;
          tc_fence_after();
          multiply(0, b, false);
          if (ksteps == 2) {
            ok = mbar_wait(a_full(b1), aph1, dead);
            if (!ok) break;
            tc_fence_after();
            multiply(1, b1, false);
          }
          multiply(0, b, true);
          tc_commit(a_empty(b));
          b = b1;
          aph = aph1;
          if (ksteps == 2) {
            multiply(1, b, true);
            tc_commit(a_empty(b));
            b = (b + 1) & (BUF - 1);
            aph = b ? aph : aph ^ 1;
          }
          tc_commit(acc_full(c));
          if (++c == AS) { c = 0; cph ^= 1; }
        }
      } else {
        bool ok = blockIdx.x >= a.tiles || mbar_wait(a_full(0), 0, dead);
        for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x) {
          ok = mbar_wait(acc_empty(c), cph ^ 1, dead);
          for (int k = 0; k < ksteps && ok; ++k) {
            const int set = SETS == 2 ? k & 1 : 0;
            const unsigned d = tmem + c * sums + set * 3 * NP;
            const unsigned long long w = smem_desc(smem_u32(wsm + (k >> 1) * wtile) + (k & 1) * 64);
            const unsigned at = tmem + a_col + b * kTcBufferCols;
            const int nb = b + 1 == BUF ? 0 : b + 1;
            const unsigned naph = nb ? aph : aph ^ 1;
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              if (ks == 1 && k * 32 + 16 >= a.K) break;          // nothing but zeros
              const unsigned first = k >= max(SETS, 1) || ks > 0 ? 1u : 0u;
              tc_mma_ts(d, at + ks * 8, w + ks * 2, i3, first);
              tc_mma_ts(d + NP, at + 16 + ks * 8, w + ks * 2, i2, 1u);
              tc_mma_ts(d + 2 * NP, at + 32 + ks * 8, w + ks * 2, i1, 1u);
              // the wait for the next box stands between the two halves of this one, whose products run meanwhile
              if (ks == 0 && (k + 1 < ksteps || t + static_cast<int>(gridDim.x) < a.tiles)) ok = mbar_wait(a_full(nb), naph, dead);
            }
            tc_commit(a_empty(b));
            b = nb;
            aph = naph;
          }
          if (ok) tc_commit(acc_full(c));
          if (++c == AS) { c = 0; cph ^= 1; }
        }
      }
      if (*dead) {        // products in flight still use the tensor memory
        tc_commit(drain);
        for (int i = 0; i < kWaitLimit && !mbar_try(drain, 0); ++i) {}
      }
    }
  } else if (warp >= EXPAND) {
    const int grp = (warp - EXPAND) >> 2;
    const int quad = (warp & 3) * 32, row = quad + lane;
    const unsigned dst0 = tmem + (static_cast<unsigned>(quad) << 16) + a_col;
    const int mine = (a.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    const int count = max(0, mine) * ksteps;
    int s = grp % S;
    unsigned ph = static_cast<unsigned>(grp / S) & 1, bph = 1;
    int b = grp;
    for (int i = grp; i < count; i += GROUPS) {
      // a stage's phase is known by its parity alone: its previous box (i - S, S >= BUF) must have been multiplied first
      if (!mbar_wait(a_empty(b), bph, dead)) break;
      if (!mbar_wait(full(s), ph, dead)) break;
      tc_fence_after();
      const unsigned dst = dst0 + b * kTcBufferCols;
      const char* src = smem + s * kXStageBytes + row * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        unsigned y[3][8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 v = *reinterpret_cast<const float4*>(src + (((h * 4 + q) ^ (row & 7)) << 4));
          split3_pair(v.x, v.y, y[0][2 * q], y[1][2 * q], y[2][2 * q]);
          split3_pair(v.z, v.w, y[0][2 * q + 1], y[1][2 * q + 1], y[2][2 * q + 1]);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st8(dst + p * 16 + h * 8, y[p]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(s));
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full(b));
      s += GROUPS;
      while (s >= S) { s -= S; ph ^= 1; }
      b += GROUPS;
      if (b >= BUF) { b -= BUF; bph ^= 1; }
    }
  } else if (warp >= 4) {
    // PARTS warps per 32 rows take their column pieces in turn
    constexpr bool OLD = tc_reads_old(EPI);
    constexpr int PIECE = tc_piece(OLD);
    constexpr bool SOFTMAX = EPI == CAGNET_EPI_LOG_SOFTMAX || EPI == kEpiNll;
    const int slot = LIGHT ? ((warp - 4) >> 2) / PARTS : 0, part = ((warp - 4) >> 2) - slot * PARTS, quad = (warp & 3) * 32;
    const int group_id = 1 + slot * 4 + (warp & 3), every = static_cast<int>(gridDim.x) * (LIGHT ? AS : 1);
    const unsigned lane_base = static_cast<unsigned>(quad) << 16;
    float* xch = xch_all + (warp - 4) * (32 * (PIECE + 4));
    const int width = min(NP, a.N - n0);
    const bool vec = a.z_vec4 != 0;
    int c = slot;
    unsigned cph = 0;
    [[maybe_unused]] float picked = 0.f;            // log-probabilities of the labels that this thread wrote
    for (int t = blockIdx.x + slot * gridDim.x; t < a.tiles; t += every) {
      const int64_t row0 = static_cast<int64_t>(t) * 128 + quad;
      const int rows = static_cast<int>(min(static_cast<int64_t>(32), a.n - row0));       // may be <= 0
      // a piece of COLS columns: LR lanes per row, 32 / LR rows per step
      [[maybe_unused]] float4 old[OLD ? PIECE / 4 : 1];
      [[maybe_unused]] auto ask = [&](auto cols_tag, int j0) {
        constexpr int LR = decltype(cols_tag)::value / 4, RS = 32 / LR;
        const int jj = j0 + (lane % LR) * 4, r0 = lane / LR, live = width - jj;
        const float* m = EPI == CAGNET_EPI_RELU_MASK ? a.aux + (row0 + r0) * a.ldaux + n0 + jj : a.Z + (row0 + r0) * a.ldz + n0 + jj;
        const int64_t step = (EPI == CAGNET_EPI_RELU_MASK ? a.ldaux : a.ldz) * RS;
#pragma unroll
        for (int i = 0; i < LR; ++i) {
          old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (live > 0 && r0 + i * RS < rows) {
            if (live >= 4 && a.aux_vec4) {
              old[i] = __ldcg(reinterpret_cast<const float4*>(m + i * step));
            } else {
              old[i].x = __ldcg(m + i * step);
              if (live > 1) old[i].y = __ldcg(m + i * step + 1);
              if (live > 2) old[i].z = __ldcg(m + i * step + 2);
              if (live > 3) old[i].w = __ldcg(m + i * step + 3);
            }
          }
        }
      };
      [[maybe_unused]] int label = -1;              // of row row0 + lane, where the loss has it
      if constexpr (EPI == kEpiNll) {
        if (lane < rows && a.loss.mask[row0 + lane]) {
          const int64_t l = a.loss.y[row0 + lane];
          if (l >= a.loss.cls_lo && l < a.loss.cls_hi) label = static_cast<int>(l - a.loss.cls_lo);
        }
      }
      auto piece = [&](auto cols_tag, int j0, unsigned acc, float lse) {
        constexpr int COLS = decltype(cols_tag)::value, LR = COLS / 4, RS = 32 / LR, STRIDE = COLS + 4;
        const int jj = j0 + (lane % LR) * 4, r0 = lane / LR, live = width - jj;
#pragma unroll
        for (int h = 0; h < COLS / 16; ++h) {
          float v[16];
          load_sums<SETS>(acc + j0 + 16 * h, NP, v);
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            *reinterpret_cast<float4*>(xch + lane * STRIDE + 16 * h + i) = make_float4(v[i] - lse, v[i + 1] - lse, v[i + 2] - lse, v[i + 3] - lse);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && j0 + PIECE * PARTS >= NP) mbar_arrive(acc_empty(c));        // the last that this warp reads of this tile
#pragma unroll
        for (int i = 0; i < LR; ++i) {
          const int r = r0 + i * RS;
          float4 v = *reinterpret_cast<const float4*>(xch + r * STRIDE + (lane % LR) * 4);
          [[maybe_unused]] float4 g;
          if constexpr (EPI == CAGNET_EPI_RELU) {
            v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
          } else if constexpr (EPI == CAGNET_EPI_RELU_MASK) {
            v = make_float4(old[i].x > 0.f ? v.x : 0.f, old[i].y > 0.f ? v.y : 0.f, old[i].z > 0.f ? v.z : 0.f, old[i].w > 0.f ? v.w : 0.f);
          } else if constexpr (EPI == CAGNET_EPI_ACCUMULATE) {
            v = make_float4(v.x + old[i].x, v.y + old[i].y, v.z + old[i].z, v.w + old[i].w);
          } else if constexpr (EPI == kEpiNll) {
            const int at = __shfl_sync(0xffffffffu, label, r), d = at - jj;
            g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (at >= 0) {
              const float w = a.loss.inv_count;
              g = make_float4((d == 0 ? -w : 0.f) + expf(v.x) * w, (d == 1 ? -w : 0.f) + expf(v.y) * w, (d == 2 ? -w : 0.f) + expf(v.z) * w,
                              (d == 3 ? -w : 0.f) + expf(v.w) * w);
              if (d >= 0 && d < 4) picked += d == 0 ? v.x : d == 1 ? v.y : d == 2 ? v.z : v.w;
            }
          }
          if (r < rows && live > 0) {
            auto store = [&](float* p, const float4& x) {
              if (live >= 4 && vec) {
                *reinterpret_cast<float4*>(p) = x;
              } else {
                p[0] = x.x;
                if (live > 1) p[1] = x.y;
                if (live > 2) p[2] = x.z;
                if (live > 3) p[3] = x.w;
              }
            };
            store(a.Z + (row0 + r) * a.ldz + n0 + jj, v);
            if constexpr (EPI == kEpiNll) store(a.loss.dz + (row0 + r) * a.loss.lddz + jj, g);
          }
        }
        __syncwarp();
      };
      // with a piece of PIECE columns or, at the end of an NP that is no multiple of it, of 16
      auto sized = [&](int j0, auto&& what) {
        if (PIECE == 16 || NP - j0 < PIECE) what(std::integral_constant<int, 16>{});
        else what(std::integral_constant<int, PIECE>{});
      };
      if constexpr (OLD) {                          // asked for before the sums are waited for
        if (PIECE * part < NP) sized(PIECE * part, [&](auto tag) { ask(tag, PIECE * part); });
      }
      bool ready = mbar_wait(acc_full(c), cph, dead);
      if (SOFTMAX && PARTS > 1) ready = group_and(ready, group_id, 32 * PARTS);        // they leave together
      if (!ready) break;
      tc_fence_after();
      const unsigned acc = tmem + lane_base + c * sums;
      float lse = 0.f;
      if constexpr (SOFTMAX) {
        // this thread's row, 16 columns at a time; the warps of a row take them in turn and exchange what they found.
        // (Columns that do not exist count as -infinity: a branch per column would keep the exponentials from overlapping.)
        float mx = -INFINITY, sum = 0.f;
        for (int j = 16 * part; j < width; j += 16 * PARTS) {
          float v[16];
          load_sums<SETS>(acc + j, NP, v);
          float m = mx;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            v[i] = j + i < width ? v[i] : -INFINITY;
            m = fmaxf(m, v[i]);
          }
          float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 16; ++i) e[i & 3] += expf(v[i] - m);
          sum = (mx == -INFINITY ? 0.f : sum * expf(mx - m)) + ((e[0] + e[1]) + (e[2] + e[3]));
          mx = m;
        }
        if (PARTS > 1) {
          reinterpret_cast<float2*>(xch)[lane] = make_float2(mx, sum);
          group_and(true, group_id, 32 * PARTS);
          const float* others = xch_all + (slot * PARTS * 4 + (warp & 3)) * (32 * (PIECE + 4));
          auto of = [&](int p) { return reinterpret_cast<const float2*>(others + 4 * p * (32 * (PIECE + 4)))[lane]; };
          for (int p = 0; p < PARTS; ++p) mx = fmaxf(mx, of(p).x);
          sum = 0.f;                                // in the same order in every warp
          for (int p = 0; p < PARTS; ++p) sum += of(p).x == -INFINITY ? 0.f : of(p).y * expf(of(p).x - mx);
          group_and(true, group_id, 32 * PARTS);
        }
        lse = mx + logf(sum);
      }
      for (int j0 = PIECE * part; j0 < NP; j0 += PIECE * PARTS) {
        if constexpr (OLD) {
          if (j0 != PIECE * part) sized(j0, [&](auto tag) { ask(tag, j0); });
        }
        sized(j0, [&](auto tag) { piece(tag, j0, acc, lse); });
      }
      if (PIECE * part >= NP) {                     // no piece of its own
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(c));
      }
      if (LIGHT || ++c == AS) { c = slot; cph ^= 1; }
    }
    if constexpr (EPI == kEpiNll) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) picked += __shfl_xor_sync(0xffffffffu, picked, off);
      if (lane == 0) a.loss.parts[blockIdx.x * STORING + warp - 4] = picked;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && dead_s) g_gemm_error = 1;
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---------------------------------------------------------------------------------------------- transposed product
// Partial sums of A^T . B over a share of the rows, A n x M (the wider operand), B n x N: the weight gradients.
// Here the rows are what is summed over, so a thread of an expanding warp owns a COLUMN of A: it reads 32 rows of it from a
// TMA box (consecutive lanes, consecutive words), splits them and stores them as its lane's operand row; B's rows arrive
// the same way and are turned into K-major shared-memory tiles by four warps.  Sums of all of A's 128-column tiles stay in
// tensor memory (MT tiles of 3 NP columns) for kTnRun steps and are then added to fp32 sums in shared memory: additions in
// tensor memory drop what does not fit, and over a block's 4,700 rows that was 5e-6 of the result (2.7e-7 with runs of 4
// steps = 16 additions, what the FMA kernels' sums have).  Each block leaves one M x N partial.
constexpr int kTnRun = 4;
constexpr int kTnRows = 64;                        // rows per step
constexpr int kTnBox = kTnRows * 128;              // a box: 64 rows x 32 floats
constexpr int kTnSlot = 4 * kTnBox;                // 128 columns of A
constexpr int kTnMaxSlots = 6;
constexpr int kTnThreads = 768;                    // warp 0 loads, 1 multiplies, 4 - 7 lay B out and store sums, 8 - 23 expand A

struct TnTcArgs {
  float* part;                                     // [blocks][M][N]
  int64_t steps;                                   // ceil(n / 64)
  int M, N, NP, MT, slots, parts;                  // MT: 128-column tiles of A per block (of blockIdx.y)
};

__global__ void __launch_bounds__(kTnThreads, 1) gemm_tn_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                                                                   TnTcArgs a) {
  extern __shared__ __align__(1024) char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * kTnMaxSlots + 2 * kTcMaxBuffers + 11];
  __shared__ unsigned tmem_base_s;
  __shared__ int dead_s;
  char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = a.slots, NP = a.NP;
  const int m0 = blockIdx.y * a.MT * 128;                            // this block's first column of A
  const int boxes = min(a.MT * 4, (a.M - m0 + 31) / 32);             // boxes of A per step
  const int MT = (boxes + 3) / 4;
  const int gboxes = (NP + 31) / 32;
  const int bbytes = 3 * NP * 128;
  char* gsm = smem + S * kTnSlot;                                    // two raw steps of B
  char* bsm = gsm + 2 * gboxes * kTnBox;                             // two operand tiles of B
  float* sum_s = reinterpret_cast<float*>(bsm + 2 * bbytes);         // [MT * NP][128]
  const unsigned bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8 * s; };
  auto empty = [&](int s) { return bar0 + 8 * (kTnMaxSlots + s); };
  auto a_full = [&](int b) { return bar0 + 8 * (2 * kTnMaxSlots + b); };
  auto a_empty = [&](int b) { return bar0 + 8 * (2 * kTnMaxSlots + kTcMaxBuffers + b); };
  const unsigned rest0 = bar0 + 8 * (2 * kTnMaxSlots + 2 * kTcMaxBuffers);
  auto g_full = [&](int b) { return rest0 + 8 * b; };
  auto g_empty = [&](int b) { return rest0 + 8 * (2 + b); };
  auto b_full = [&](int b) { return rest0 + 8 * (4 + b); };
  auto b_empty = [&](int b) { return rest0 + 8 * (6 + b); };
  const unsigned acc_full = rest0 + 64, acc_empty = rest0 + 72, drain = rest0 + 80;
  volatile int* dead = &dead_s;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 8);        // four warps for each half of the step
    }
    for (int b = 0; b < kTcMaxBuffers; ++b) {
      mbar_init(a_full(b), 4);
      mbar_init(a_empty(b), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(g_full(b), 1);
      mbar_init(g_empty(b), 4);
      mbar_init(b_full(b), 4);
      mbar_init(b_empty(b), 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 4);
    mbar_init(drain, 1);
    dead_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base_s;
  const unsigned a_col = 512 - kTcMaxBuffers * kTcBufferCols;
  pdl_trigger();
  pdl_wait();
  const int s0 = static_cast<int>(a.steps * blockIdx.x / gridDim.x), s1 = static_cast<int>(a.steps * (blockIdx.x + 1) / gridDim.x);
  const int n0 = blockIdx.z * NP;
  const int count = s1 - s0;                       // >= 1: there are at least as many steps as blocks

  if (warp == 0) {
    if (lane == 0) {
      int q = 0;                                   // slots issued
      bool ok = true;
      for (int i = 0; i < count && ok; ++i) {
        const int row = (s0 + i) * kTnRows;
        ok = mbar_wait(g_empty(i & 1), ((i >> 1) & 1) ^ 1, dead);
        if (!ok) break;
        mbar_expect(g_full(i & 1), gboxes * kTnBox);
        for (int x = 0; x < gboxes; ++x) tma_load_2d(smem_u32(gsm + ((i & 1) * gboxes + x) * kTnBox), &mapB, n0 + x * 32, row, g_full(i & 1));
        for (int mt = 0; mt < MT; ++mt, ++q) {
          const int s = q % S;
          ok = mbar_wait(empty(s), ((q / S) & 1) ^ 1, dead);
          if (!ok) break;
          const int nb = min(4, boxes - mt * 4);
          mbar_expect(full(s), nb * kTnBox);
          for (int x = 0; x < nb; ++x) tma_load_2d(smem_u32(smem + s * kTnSlot + x * kTnBox), &mapA, m0 + mt * 128 + x * 32, row, full(s));
        }
      }
      if (*dead) {        // a wait ran out: the copies in flight still write into this block's shared memory
        for (int k = max(0, q - S); k < q; ++k)
          for (int i = 0; i < kWaitLimit && !mbar_try(full(k % S), (k / S) & 1); ++i) {}
        for (int b = 0; b < 2; ++b)
          for (int i = 0; i < kWaitLimit && !mbar_try(g_full(b), 0) && !mbar_try(g_full(b), 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const unsigned base = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);      // D fp32, A and B bf16, K-major, M = 128
      auto idesc = [&](int N) { return base | (static_cast<unsigned>(N >> 3) << 17); };
      const unsigned i3 = idesc(3 * NP), i2 = idesc(2 * NP), i1 = idesc(NP);
      int b = 0;
      unsigned aph = 0;
      bool ok = true;
      for (int i = 0; i < count && ok; ++i) {
        ok = mbar_wait(b_full(i & 1), (i >> 1) & 1, dead);
        const int run = i % kTnRun;
        if (ok && run == 0 && i > 0) ok = mbar_wait(acc_empty, (i / kTnRun - 1) & 1, dead);
        const unsigned long long w0 = smem_desc(smem_u32(bsm + (i & 1) * bbytes));
        for (int u = 0; u < 2 * MT && ok; ++u) {
          ok = mbar_wait(a_full(b), aph, dead);
          if (!ok) break;
          tc_fence_after();
          const unsigned d = tmem + (u >> 1) * 3 * NP, at = tmem + a_col + b * kTcBufferCols;
          const unsigned long long w = w0 + (u & 1) * 4;
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            tc_mma_ts(d, at + ks * 8, w + ks * 2, i3, run + (u & 1) + ks > 0 ? 1u : 0u);
            tc_mma_ts(d + NP, at + 16 + ks * 8, w + ks * 2, i2, 1u);
            tc_mma_ts(d + 2 * NP, at + 32 + ks * 8, w + ks * 2, i1, 1u);
          }
          tc_commit(a_empty(b));
          if (++b == kTcMaxBuffers) { b = 0; aph ^= 1; }
        }
        if (ok) tc_commit(b_empty(i & 1));
        if (ok && (run + 1 == kTnRun || i + 1 == count)) tc_commit(acc_full);
      }
      if (*dead) {        // products in flight still use the tensor memory
        tc_commit(drain);
        for (int i = 0; i < kWaitLimit && !mbar_try(drain, 0); ++i) {}
      }
    }
  } else if (warp >= 8) {
    const int grp = (warp - 8) >> 2, quad = warp & 3;
    const unsigned dst = tmem + (static_cast<unsigned>(quad * 32) << 16) + a_col + grp * kTcBufferCols;
    const int units = count * 2 * MT;
    unsigned bph = 1;
    for (int u = grp; u < units; u += kTcMaxBuffers) {
      const int q = u >> 1, s = q % S;
      // (a slot's phase is known by its parity alone: the slots before it must have been multiplied, S >= 2)
      if (!mbar_wait(a_empty(grp), bph, dead)) break;
      bph ^= 1;
      if (!mbar_wait(full(s), (q / S) & 1, dead)) break;
      tc_fence_after();
      if (q % MT * 4 + quad < boxes) {             // the last tile may end earlier: those lanes' sums are never read
        const float* src = reinterpret_cast<const float*>(smem + s * kTnSlot + quad * kTnBox) + (u & 1) * 32 * 32 + lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned y[3][8];
#pragma unroll
          for (int r = 0; r < 8; ++r)
            split3_pair(src[(h * 16 + 2 * r) * 32], src[(h * 16 + 2 * r + 1) * 32], y[0][r], y[1][r], y[2][r]);
#pragma unroll
          for (int p = 0; p < 3; ++p) tmem_st8(dst + p * 16 + h * 8, y[p]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(s));
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full(grp));
    }
  } else if (warp >= 4) {
    const int quad = (warp & 3) * 32;
    bool ok = true;
    // B's operand tile of a step: one task is 8 rows of one column, as 16-byte pieces of the three terms' rows
    auto lay_out = [&](int i) {
      if (!mbar_wait(g_full(i & 1), (i >> 1) & 1, dead) || !mbar_wait(b_empty(i & 1), ((i >> 1) & 1) ^ 1, dead)) return false;
      const char* raw = gsm + (i & 1) * gboxes * kTnBox;
      char* tile = bsm + (i & 1) * bbytes;
      for (int t = (warp - 4) * 32 + lane; t < NP * 8; t += 128) {
        const int j = t % NP, c = t / NP;
        const float* src = reinterpret_cast<const float*>(raw + (j >> 5) * kTnBox) + c * 8 * 32 + (j & 31);
        unsigned y[3][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) split3_pair(src[2 * r * 32], src[(2 * r + 1) * 32], y[0][r], y[1][r], y[2][r]);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const int row = p * NP + j;
          *reinterpret_cast<uint4*>(tile + row * 128 + ((c ^ (row & 7)) << 4)) = make_uint4(y[p][0], y[p][1], y[p][2], y[p][3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(g_empty(i & 1));
        mbar_arrive(b_full(i & 1));
      }
      return true;
    };
    // a run's sums out of tensor memory, onto this thread's column of the shared sums
    auto promote = [&](int run) {
      if (!mbar_wait(acc_full, run & 1, dead)) return false;
      tc_fence_after();
      for (int j = 0; j < MT * NP; j += 16) {
        float v[16];
        load_sums<1>(tmem + (static_cast<unsigned>(quad) << 16) + j / NP * 3 * NP + j % NP, NP, v);
        float* d = sum_s + j * 128 + quad + lane;
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i * 128] = run ? d[i * 128] + v[i] : v[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      return true;
    };
    // one step of B ahead of the promotion of the run before it, so that the multiply does not wait for both
    for (int i = 0; i < count && ok; ++i) {
      ok = lay_out(i);
      if (ok && i % kTnRun == 0 && i > 0) ok = promote(i / kTnRun - 1);
    }
    if (ok && promote((count - 1) / kTnRun)) {
      float* out = a.part + static_cast<int64_t>(blockIdx.x) * a.M * a.N;
      for (int mt = 0; mt < MT; ++mt) {
        const int m = m0 + mt * 128 + quad + lane;
        if (m < a.M)
          for (int j = 0; j < NP && n0 + j < a.N; ++j) out[static_cast<int64_t>(m) * a.N + n0 + j] = sum_s[(mt * NP + j) * 128 + quad + lane];
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && dead_s) g_gemm_error = 1;
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---------------------------------------------------------------------------------------------- host side
// Tensor map of an n x K fp32 matrix with rows ld apart, boxes of `rows` rows x 32 columns.
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<EncodeFn>(p);
  }();
  return fn;
}

static bool encode_rows(CUtensorMap* map, const float* X, int64_t n, int K, int64_t ld, int rows, bool swizzle) {
  EncodeFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(n)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 4};
  const cuuint32_t box[2] = {32, static_cast<cuuint32_t>(rows)}, elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(X), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Columns of W a block keeps in shared memory (a multiple of 16), 0 where the kernel does not apply.
static int tc_columns(int K, int N, int epilogue) {
  const int fit = kTcMaxW / ((K + 63) / 64 * 3 * 128) / 16 * 16;
  int np = (N + 15) / 16 * 16;
  if (epilogue == CAGNET_EPI_LOG_SOFTMAX || epilogue == CAGNET_EPI_LOG_SOFTMAX_256 || epilogue == kEpiNll)
    return (np <= 80 || (np <= 256 && K <= 64)) && np <= fit && (K <= 320 || np <= 48) ? np : 0;
  const int most = min(fit, K > 320 ? 48 : (K > 64 ? 80 : 160));
  // at most 160 columns, so that two sets of sums fit and one tile's stores run under the next one's products
  const int parts = fit >= 16 ? (np + most - 1) / most : 0;
  if (parts == 0 || parts > 4) return 0;          // every part reads X again
  np = ((N + parts - 1) / parts + 15) / 16 * 16;
  return np <= most ? np : 0;
}

// The FMA kernels keep the unaligned and the small products, where this kernel's 5 us of set-up show (20K x 32 x 30: 5.0 us there,
// 7.6 here; 39K x 100 x 16: 16.4 and 9.6).
bool gemm_nn_tc_applies(const float* X, int64_t ldx, int64_t n, int K, int N, int epilogue) {
  return n >= 64 * kNumSMs && n * (K + N) >= 3000000 && n <= INT_MAX && K >= 8 && N >= 8 && ldx % 4 == 0 && aligned(X, 16) && tc_columns(K, N, epilogue) > 0 &&
         encode_fn() != nullptr;
}

template <int SETS, int EPI>
static cudaError_t launch_tc(dim3 grid, size_t smem, cudaStream_t s, const CUtensorMap& map, const TcArgs& a) {
  static bool opted_in[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !opted_in[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_nn_tc_kernel<SETS, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
    if (e != cudaSuccess) return e;
    opted_in[dev] = true;
  }
  return launch_pdl(gemm_nn_tc_kernel<SETS, EPI>, grid, dim3(kTcThreads), smem, s, map, a);
}

template <int SETS>
static cudaError_t launch_tc_epilogue(int epilogue, dim3 grid, size_t smem, cudaStream_t s, const CUtensorMap& map, const TcArgs& a) {
  switch (epilogue) {
    case CAGNET_EPI_NONE: return launch_tc<SETS, CAGNET_EPI_NONE>(grid, smem, s, map, a);
    case CAGNET_EPI_RELU: return launch_tc<SETS, CAGNET_EPI_RELU>(grid, smem, s, map, a);
    case CAGNET_EPI_RELU_MASK: return launch_tc<SETS, CAGNET_EPI_RELU_MASK>(grid, smem, s, map, a);
    case CAGNET_EPI_ACCUMULATE: return launch_tc<SETS, CAGNET_EPI_ACCUMULATE>(grid, smem, s, map, a);
    case kEpiNll: return launch_tc<SETS, kEpiNll>(grid, smem, s, map, a);
    default: return launch_tc<SETS, CAGNET_EPI_LOG_SOFTMAX>(grid, smem, s, map, a);
  }
}

static int run_nn_tc(const float* X, int64_t ldx, const float* W, int64_t ldw, int transW, float* Z, int64_t ldz, int64_t n, int K, int N,
                     int epilogue, const float* aux, int64_t ldaux, const TcLoss* loss, int32_t* parts, cudaStream_t s) {
  CUtensorMap map;
  if (!encode_rows(&map, X, n, K, ldx, 128, true)) return fail(CAGNET_E_LAUNCH, "cagnet_gemm_nn_f32: cannot describe X to the copy engine");
  TcArgs a;
  a.W = W; a.aux = aux; a.Z = Z;
  a.ldw = ldw; a.ldz = ldz; a.ldaux = ldaux; a.n = n;
  a.transW = transW; a.K = K; a.N = N;
  a.NP = tc_columns(K, N, epilogue);
  a.loss = loss ? *loss : TcLoss{};
  a.z_vec4 = (ldz % 4 == 0 && aligned(Z, 16) && (!loss || (loss->lddz % 4 == 0 && aligned(loss->dz, 16)))) ? 1 : 0;
  a.aux_vec4 = epilogue == CAGNET_EPI_RELU_MASK ? ldaux % 4 == 0 && aligned(aux, 16) : a.z_vec4;
  a.tiles = static_cast<int>((n + 127) / 128);
  const int wbytes = (K + 63) / 64 * 3 * a.NP * 128;
  const int sets = K <= kTcLightK ? 0 : K > 320 ? 2 : 1, exchange = tc_exchange_bytes(sets, tc_reads_old(epilogue));
  a.stages = min(kTcMaxStages, (kTcSmem - 1024 - exchange - wbytes) / kXStageBytes);
  const size_t smem = 1024 + static_cast<size_t>(a.stages) * kXStageBytes + wbytes + exchange;
  const dim3 grid(a.tiles < kNumSMs ? a.tiles : kNumSMs, (N + a.NP - 1) / a.NP);
  if (parts) *parts = static_cast<int32_t>(grid.x) * tc_storing_warps(sets);
  const cudaError_t e = sets == 0   ? launch_tc_epilogue<0>(epilogue, grid, smem, s, map, a)
                        : sets == 2 ? launch_tc_epilogue<2>(epilogue, grid, smem, s, map, a)
                                    : launch_tc_epilogue<1>(epilogue, grid, smem, s, map, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_nn_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

int gemm_nn_tc(const float* X, int64_t ldx, const float* W, int64_t ldw, int transW, float* Z, int64_t ldz, int64_t n, int K, int N,
               int epilogue, const float* aux, int64_t ldaux, cudaStream_t s) {
  return run_nn_tc(X, ldx, W, ldw, transW, Z, ldz, n, K, N, epilogue, aux, ldaux, nullptr, nullptr, s);
}

int gemm_nn_tc_nll(const float* X, int64_t ldx, const float* W, int64_t ldw, float* Z, int64_t ldz, int64_t n, int K, int N, const TcLoss& loss,
                   int32_t* parts, cudaStream_t s) {
  return run_nn_tc(X, ldx, W, ldw, 0, Z, ldz, n, K, N, kEpiNll, nullptr, 0, &loss, parts, s);
}

// Shape of A^T . B on this kernel: NP columns of B per block (three sums each), MT column tiles of A per block.
struct TnTcShape {
  int np, parts, mt, groups, blocks, slots;
};
static int tn_tc_fixed_smem(const TnTcShape& t) { return 2 * ((t.np + 31) / 32) * kTnBox + 2 * 3 * t.np * 128 + t.mt * t.np * 512; }
static TnTcShape tn_tc_shape(int64_t n, int M, int N) {
  TnTcShape t;
  t.parts = (N + 79) / 80;
  t.np = ((N + t.parts - 1) / t.parts + 15) / 16 * 16;
  const int tiles = (M + 127) / 128, most = 96 / t.np;         // 288 tensor-memory columns, 48 KB of shared sums
  t.groups = (tiles + most - 1) / most;
  t.mt = (tiles + t.groups - 1) / t.groups;
  const int64_t steps = (n + kTnRows - 1) / kTnRows;
  t.blocks = static_cast<int>(steps < kNumSMs ? steps : kNumSMs);
  if (t.groups * t.parts > 1) t.blocks = max(1, min(t.blocks, kNumSMs / (t.groups * t.parts)));
  t.slots = min(kTnMaxSlots, (kTcSmem - 1024 - tn_tc_fixed_smem(t)) / kTnSlot);
  return t;
}

// A = the wider of H and G.  Few rows leave most blocks without enough steps to cover their set-up (2.7K x 1,433 x 16 stays on
// the FMA kernel).
bool gemm_tn_tc_applies(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int K, int N) {
  return n >= 64 * kNumSMs && n * (K + N) >= 3000000 && n <= INT_MAX && min(K, N) >= 4 && max(K, N) >= 64 && min(K, N) <= 320 &&
         ldh % 4 == 0 && ldg % 4 == 0 && aligned(H, 16) && aligned(G, 16) && encode_fn() != nullptr;
}

int gemm_tn_tc_blocks(int64_t n, int K, int N) { return tn_tc_shape(n, max(K, N), min(K, N)).blocks; }

// Partial sums of A^T . B per block into part: A = H when K >= N, G otherwise (then the partials are those of the transpose).
int gemm_tn_tc(const float* H, int64_t ldh, const float* G, int64_t ldg, int64_t n, int K, int N, float* part, cudaStream_t s) {
  static bool opted_in[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !opted_in[dev]) {
    if (cudaFuncSetAttribute(gemm_tn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess)
      return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: cannot reserve shared memory");
    opted_in[dev] = true;
  }
  const bool swap = K < N;
  const float *A = swap ? G : H, *B = swap ? H : G;
  const int M = max(K, N), W = min(K, N);
  const TnTcShape t = tn_tc_shape(n, M, W);
  CUtensorMap ma, mb;
  if (!encode_rows(&ma, A, n, M, swap ? ldg : ldh, kTnRows, false) || !encode_rows(&mb, B, n, W, swap ? ldh : ldg, kTnRows, false))
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: cannot describe the operands to the copy engine");
  TnTcArgs a;
  a.part = part;
  a.steps = (n + kTnRows - 1) / kTnRows;
  a.M = M; a.N = W; a.NP = t.np; a.MT = t.mt; a.slots = t.slots; a.parts = t.parts;
  const size_t smem = 1024 + static_cast<size_t>(t.slots) * kTnSlot + tn_tc_fixed_smem(t);
  const cudaError_t e = launch_pdl(gemm_tn_tc_kernel, dim3(t.blocks, t.groups, t.parts), dim3(kTnThreads), smem, s, ma, mb, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_gemm_tn_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

int gemm_tc_error() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return v;
}

}  // namespace cagnet
