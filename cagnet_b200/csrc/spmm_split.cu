// Nonzero-split SpMM for sm_100a:  C = beta*C + A*B,  fp32 values, row-major B and C.
//
// The row kernels of spmm.cu give a row to a lane group, a warp or a block by its length; on a power-law block the
// longest row of a launch is then its tail (100K nonzeros on one block), a 5-nonzero row costs a chain of three
// dependent loads, and every length class needs its own kernel.  Here the NONZEROS are cut into chunks of equal length
// and a lane group (LPN lanes, each LPN-strided vectors of 4 columns) walks one chunk from end to end, whatever rows it
// holds: the last nonzero of every row carries a mark in the sign bit of its column index, and a group that meets one
// writes the finished row and starts the next.  What bounds it is the gather itself: one L1 wavefront per nonzero at
// widths <= 32 (71 % busy at width 16 on a 1 M-vertex / 32 M-nonzero R-MAT graph), L2 misses of the gathered rows beyond.
//   * (column, value) pairs are stored interleaved: 16 bytes per lane bring 2 LPN pairs of the group's chunk into
//     registers one stage ahead, pass through a shared-memory slot and come back as broadcasts;
//   * BATCH gathers of a lane are issued before the first of their multiply-adds (in nonzero order);
//   * a row that crosses chunks leaves its pieces in a workspace: at most one piece ends and one begins in a chunk.  The
//     join kernel adds a row's pieces in chunk order, so results are the same on every run (no atomics).
// Measured against the row kernels (spmm.cu) on one GPU, whole multiply: R-MAT 1 M vertices / 32 M nonzeros width 16
// 0.355 -> 0.23 ms, 41 0.90 -> 0.57, 64 0.88 -> 0.57, 128 1.47 -> 1.18, 602 7.18 -> 6.1; 65 K vertices / 3.2 M nonzeros
// width 16 70 -> 33 us, 128 216 -> 108 us; 5 K vertices / 100 K nonzeros width 16 20 -> 8 us, width 128 148 -> 11 us.
#include <limits.h>

#include "common.cuh"

namespace cagnet {

constexpr int kUnit = 8;                // granularity of the row bookkeeping, nonzeros
constexpr int kSplitWarps = 4;          // warps per block
constexpr unsigned kMid = 0x80000000u;  // first[]: the unit starts inside a row

struct SplitArgs {
  const int2* pairs;       // (column | end-of-row mark, value bits), padded to whole units with (INT_MAX, 0)
  const unsigned* first;   // per unit: position in `rows` of the row its first nonzero belongs to, kMid if it began earlier
  const int* rows;         // rows with nonzeros, ascending; nullptr = all of them
  const int* empty;        // rows without
  const float* B;
  float* C;
  float* part;             // [feature tiles][chunks][ending piece | beginning piece][tile columns]
  int64_t nnz, ldb, ldc;
  int nrows, nempty, f_eff, f, chunk, nchunks, c_vec4;
  // a block given as row-sorted COO for one multiply (spmm_gpu), nothing prepared: instead of pairs, first, rows and empty
  const int *coo_rows, *coo_cols;
  const float* coo_vals;
  const int* status;       // nonzero: the indices are malformed, nothing may be done; nullptr = not checked
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// C[row, this lane's columns] = acc, or += acc: every element gets exactly one addition per multiply, so it is left to the
// memory system (the order cannot matter) instead of a load that the whole warp waits for at every row's end.  Columns >= f
// are never written.
template <int LPN, int NV>
__device__ __forceinline__ void split_store(const SplitArgs& a, int row, int column0, int nvalid, bool add,
                                            const float (&acc)[NV][4]) {
  float* cp = a.C + static_cast<int64_t>(row) * a.ldc + column0;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (k < nvalid) {
      float* p = cp + k * (LPN * 4);
      const int live = a.f - (column0 + k * (LPN * 4));
      if (live >= 4 && a.c_vec4) {
        const float4 v = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
        if (add) red_add4(p, v);
        else *reinterpret_cast<float4*>(p) = v;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < live) {
            if (add) atomicAdd(p + j, acc[k][j]);
            else p[j] = acc[k][j];
          }
        }
      }
    }
  }
}

template <int LPN, int NV>
__device__ __forceinline__ void piece_store(float* p, const float (&acc)[NV][4]) {
#pragma unroll
  for (int w = 0; w < NV; ++w)
    *reinterpret_cast<float4*>(p + w * (LPN * 4)) = make_float4(acc[w][0], acc[w][1], acc[w][2], acc[w][3]);
}

// Blocks of the walk kernel that an SM holds: what the registers of a variant allow (the compiler is held to it), and the
// size of a wave in the choice of the chunk length.
__host__ __device__ constexpr int split_blocks_per_sm(int nv, bool coo) {
  return nv == 4 ? 4 : nv == 3 ? 5 : coo ? 6 : 7;
}

// Row a chunk starts in, and whether it began in an earlier chunk: from the plan, or from the COO rows themselves.
template <bool COO>
__device__ __forceinline__ unsigned chunk_row(const SplitArgs& a, int c, bool& mid) {
  const int64_t at = static_cast<int64_t>(c) * a.chunk;
  if constexpr (COO) {
    const int r = __ldg(a.coo_rows + at);
    mid = at > 0 && __ldg(a.coo_rows + at - 1) == r;
    return static_cast<unsigned>(r);
  } else {
    const unsigned fw = __ldg(a.first + at / kUnit);
    mid = (fw & kMid) != 0;
    return fw & ~kMid;
  }
}

template <int LPN, int NV, int BATCH, bool ADD, bool COO>
__global__ void __launch_bounds__(kSplitWarps * 32, split_blocks_per_sm(NV, COO)) spmm_split_kernel(SplitArgs a) {
  constexpr int G = 32 / LPN;
  constexpr int PL = (2 * LPN >= BATCH) ? 1 : BATCH / (2 * LPN);   // 16-byte loads (2 pairs) per lane and stage
  constexpr int SL = 2 * LPN * PL;                                 // pairs per lane group and stage
  constexpr int TILE = LPN * 4 * NV;
  static_assert(SL % kUnit == 0 && SL % BATCH == 0, "stages and chunks are whole units and batches");
  __shared__ __align__(16) int2 stage_s[kSplitWarps][G][SL];
  __shared__ __align__(8) int stage_rows_s[COO ? kSplitWarps : 1][COO ? G : 1][COO ? SL : 1];
  pdl_trigger();
  pdl_wait();
  if (COO && a.status && *a.status) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPN, l = lane % LPN;
  const int chunk_id = (blockIdx.x * kSplitWarps + warp) * G + sub;
  if ((blockIdx.x * kSplitWarps + warp) * G >= a.nchunks) return;        // whole warps
  const int column0 = blockIdx.y * TILE + l * 4;
  const int nvalid = column0 >= a.f_eff ? 0 : min(NV, (a.f_eff - column0 + LPN * 4 - 1) / (LPN * 4));
  const int64_t start = static_cast<int64_t>(chunk_id) * a.chunk;
  const int len = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(a.chunk), a.nnz - start)));
  const int2* src = COO ? nullptr : a.pairs + start;
  int2* stage = stage_s[warp][sub];
  int* stage_rows = COO ? stage_rows_s[warp][sub] : nullptr;
  bool head = false;                            // the row being summed began in an earlier chunk
  int k = len > 0 ? static_cast<int>(chunk_row<COO>(a, chunk_id, head)) : 0;       // its position in `rows`
  const float* bt = a.B + column0;
  float* piece = a.part + (static_cast<int64_t>(blockIdx.y) * a.nchunks + chunk_id) * (2 * TILE) + l * 4;

  float acc[NV][4];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[v][j] = 0.f;
  bool open = false;      // acc holds terms of a row whose last nonzero has not been met

  int2 nxt_rows[PL];
  auto load_pairs = [&](int at, int4 (&q)[PL]) {
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = at + (i * LPN + l) * 2;
      if constexpr (COO) {
        q[i] = make_int4(INT_MAX, 0, INT_MAX, 0);
        if (e < len) {
          const int64_t g = start + e;
          const int r0 = __ldg(a.coo_rows + g), r1 = g + 1 < a.nnz ? __ldg(a.coo_rows + g + 1) : -1;
          q[i].x = __ldg(a.coo_cols + g) | (r0 != r1 ? INT_MIN : 0);
          q[i].y = __float_as_int(__ldg(a.coo_vals + g));
          nxt_rows[i].x = r0;
          if (e + 1 < len) {
            const int r2 = g + 2 < a.nnz ? __ldg(a.coo_rows + g + 2) : -1;
            q[i].z = __ldg(a.coo_cols + g + 1) | (r1 != r2 ? INT_MIN : 0);
            q[i].w = __float_as_int(__ldg(a.coo_vals + g + 1));
            nxt_rows[i].y = r1;
          }
        }
        continue;
      }
      // the array is padded to whole units: a 16-byte load that starts inside the chunk stays inside the array
      q[i] = e < len ? __ldg(reinterpret_cast<const int4*>(src + e)) : make_int4(INT_MAX, 0, INT_MAX, 0);
    }
  };
  int4 nxt[PL];
  load_pairs(0, nxt);
  const int steps = a.chunk / SL;      // warp-uniform; groups past the end of the matrix run on empty stages
  for (int s = 0; s < steps; ++s) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      *reinterpret_cast<int4*>(stage + (i * LPN + l) * 2) = nxt[i];
      if constexpr (COO) *reinterpret_cast<int2*>(stage_rows + (i * LPN + l) * 2) = nxt_rows[i];
    }
    __syncwarp();
    load_pairs((s + 1) * SL, nxt);
#pragma unroll
    for (int b = 0; b < SL; b += BATCH) {
      int c[BATCH];
      float v[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; i += 2) {
        const int4 q = *reinterpret_cast<const int4*>(stage + b + i);
        c[i] = q.x; v[i] = __int_as_float(q.y);
        c[i + 1] = q.z; v[i + 1] = __int_as_float(q.w);
      }
      float4 x[BATCH][NV];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        const int cc = c[i] & 0x7fffffff;
        const float* bp = bt + static_cast<int64_t>(cc) * a.ldb;
#pragma unroll
        for (int w = 0; w < NV; ++w)
          x[i][w] = (cc != INT_MAX && w < nvalid) ? ld4(bp + w * (LPN * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
#pragma unroll
        for (int w = 0; w < NV; ++w) {
          acc[w][0] = fmaf(v[i], x[i][w].x, acc[w][0]);
          acc[w][1] = fmaf(v[i], x[i][w].y, acc[w][1]);
          acc[w][2] = fmaf(v[i], x[i][w].z, acc[w][2]);
          acc[w][3] = fmaf(v[i], x[i][w].w, acc[w][3]);
        }
        if (c[i] < 0) {          // the last nonzero of a row
          if (head) {
            piece_store<LPN, NV>(piece, acc);
            head = false;
          } else {
            split_store<LPN, NV>(a, COO ? stage_rows[b + i] : (a.rows ? __ldg(a.rows + k) : k), column0, nvalid, ADD, acc);
          }
          ++k;
#pragma unroll
          for (int w = 0; w < NV; ++w)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[w][j] = 0.f;
        }
      }
      open = c[BATCH - 1] >= 0;
    }
  }
  if (open && len > 0) piece_store<LPN, NV>(piece + TILE, acc);
}

// One warp per chunk in which a row ends that began in an earlier one: the row's pieces added up in chunk order
// (lane group g takes every G-th, the groups are folded by a fixed shuffle tree).  Blocks beyond the chunks clear the
// rows without nonzeros when C is overwritten.
template <int LPN, int NV, bool ADD, bool COO>
__global__ void __launch_bounds__(128) spmm_split_join_kernel(SplitArgs a, int join_blocks) {
  constexpr int G = 32 / LPN;
  constexpr int TILE = LPN * 4 * NV;
  const int lane = threadIdx.x & 31, sub = lane / LPN, l = lane % LPN;
  pdl_trigger();
  if (blockIdx.x >= join_blocks) {
    pdl_wait();
    const int i = (blockIdx.x - join_blocks) * (128 / LPN) + threadIdx.x / LPN;
    if (i >= a.nempty) return;
    const int column0 = blockIdx.y * TILE + l * 4;
    const int nvalid = column0 >= a.f_eff ? 0 : min(NV, (a.f_eff - column0 + LPN * 4 - 1) / (LPN * 4));
    float zero[NV][4];
#pragma unroll
    for (int w = 0; w < NV; ++w)
#pragma unroll
      for (int j = 0; j < 4; ++j) zero[w][j] = 0.f;
    split_store<LPN, NV>(a, __ldg(a.empty + i), column0, nvalid, false, zero);
    return;
  }
  const int e = blockIdx.x * 4 + (threadIdx.x >> 5);
  unsigned row_k = 0;
  int lo = e;                                    // chunks lo .. e start in row row_k
  bool mine = false;
  if (COO) pdl_wait();                           // the rows may be those of the kernel in front, the status is
  if (e < a.nchunks && !(COO && a.status && *a.status)) {
    // the plan is constant: it may be read before the pieces are there
    bool mid, other;
    row_k = chunk_row<COO>(a, e, mid);
    const unsigned next = e + 1 < a.nchunks ? chunk_row<COO>(a, e + 1, other) : static_cast<unsigned>(a.nrows);
    mine = mid && next != row_k;                 // next == row_k: the row runs through this chunk
    while (mine) {                               // first chunk that starts with this row, 32 candidates at a time
      const int c = lo - 1 - lane;
      const bool same = c >= 0 && chunk_row<COO>(a, c, other) == row_k;
      const unsigned m = __ballot_sync(0xffffffffu, same);
      const int run = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
      lo -= run;
      if (run < 32) break;
    }
    if (mine) {
      chunk_row<COO>(a, lo, mid);
      if (mid) --lo;                             // it began inside the chunk before
    }
  }
  if (!COO) pdl_wait();
  if (!mine) return;
  const float* base = a.part + static_cast<int64_t>(blockIdx.y) * a.nchunks * (2 * TILE) + l * 4;
  float acc[NV][4];
#pragma unroll
  for (int w = 0; w < NV; ++w)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[w][j] = 0.f;
#pragma unroll 4
  for (int c = lo + sub; c <= e; c += G) {
    const float* p = base + static_cast<int64_t>(c) * (2 * TILE) + (c == e ? 0 : TILE);
#pragma unroll
    for (int w = 0; w < NV; ++w) {
      const float4 t = *reinterpret_cast<const float4*>(p + w * (LPN * 4));
      acc[w][0] += t.x; acc[w][1] += t.y; acc[w][2] += t.z; acc[w][3] += t.w;
    }
  }
#pragma unroll
  for (int off = LPN; off < 32; off <<= 1)
#pragma unroll
    for (int w = 0; w < NV; ++w)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[w][j] += __shfl_xor_sync(0xffffffffu, acc[w][j], off);
  if (sub != 0) return;
  const int column0 = blockIdx.y * TILE + l * 4;
  const int nvalid = column0 >= a.f_eff ? 0 : min(NV, (a.f_eff - column0 + LPN * 4 - 1) / (LPN * 4));
  split_store<LPN, NV>(a, a.rows ? __ldg(a.rows + row_k) : static_cast<int>(row_k), column0, nvalid, ADD, acc);
}

// ------------------------------------------------------------------------------------------------ plan
__global__ void split_pairs_kernel(const int* __restrict__ col, const float* __restrict__ val, int64_t nnz, int64_t padded,
                                   int2* __restrict__ pairs) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= padded) return;
  pairs[e] = e < nnz ? make_int2(col[e], __float_as_int(val[e])) : make_int2(INT_MAX, 0);
}

__global__ void split_rows_kernel(const int* __restrict__ rowptr, const int* __restrict__ rows, int nrows, int2* pairs,
                                  unsigned* __restrict__ first) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nrows) return;
  const int row = rows ? rows[k] : k;
  const int s = rowptr[row], e = rowptr[row + 1];
  pairs[e - 1].x |= 0x80000000;
  for (int64_t u = (static_cast<int64_t>(s) + kUnit - 1) / kUnit; u * kUnit < e; ++u)
    first[u] = static_cast<unsigned>(k) | (u * kUnit > s ? kMid : 0u);
}

// Rows of B on 16-byte boundaries for the vector loads.
__global__ void __launch_bounds__(256) pad_rows_kernel(const float* __restrict__ B, int64_t ldb, int m, int f, int ld4,
                                                       float4* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const int64_t total = static_cast<int64_t>(m) * ld4;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / ld4;
    const int c = static_cast<int>(i - r * ld4) * 4;
    const float* p = B + r * ldb + c;
    out[i] = make_float4(__ldg(p), c + 1 < f ? __ldg(p + 1) : 0.f, c + 2 < f ? __ldg(p + 2) : 0.f, c + 3 < f ? __ldg(p + 3) : 0.f);
  }
}

// ------------------------------------------------------------------------------------------------ choice of a variant
struct SplitShape {
  int lpn, nv, tiles, chunk;
  int64_t nchunks;
};

// Lane mapping by width (vectors of 4 columns per gathered row), measured on R-MAT graphs of 0.03 - 115 M nonzeros.
// Narrow rows: one vector per lane, as few lanes as the row has vectors (more nonzeros in flight per warp).  From 9 vectors
// on, 8 lanes with 2 to 4 vectors each: every lane has that many independent loads per nonzero, and a nonzero's pair, row
// end test and broadcast are paid once for all of them (22.6 M nonzeros, width 602: 16 lanes x 2 4.7 ms, 8 x 3 4.36;
// width 128: 16 x 2 0.87 ms, 8 x 4 0.84; width 300: 16 x 2 2.47 ms, 8 x 3 2.31).  Which of them: the one that covers
// the width with the least padding, weighed by its time per vector (two vectors 8 % above three, four 6 %).  Two-vector
// tiles are kept out of large multiplies (width 256: 8 x 2 2.20 ms, 8 x 4 1.73: 256-byte pieces of rows that do not stay
// in L2) and four-vector ones out of small ones, which they cannot spread over the chip (0.6 M nonzeros, width 128:
// 33.9 us with 2, 38.8 with 4), unless their rows are even (0.75 M nonzeros in rows of 125, width 200: 45.4 us with 2, 38.9
// with 4).  The smallest take one vector per lane for the same reason (0.1 M nonzeros, width 64:
// 11.8 us with 1, 13.7 with 2; 0.03 M, width 400: 12.5 and 14.2; but 0.09 M, width 1,093: 51.7 and, with 3, 39.4).  COO operands, whose row indices take registers and a second stage, stay with two (4 M
// nonzeros, width 128: 158 us with 2, 230 with 4).
//
// Chunk length: the launch is a whole number of full waves, a wave being what the SMs hold.  All chunks take about as long,
// so a wave that is filled to its last block ends together and one block more costs a whole wave (22.6 M nonzeros, width
// 16: chunks of 512 end in a wave of 6 % at 216 us; chunks of 704, one wave, 174 us; of 600 on seven blocks per SM 162).
// Chunks stay under 704 nonzeros, 1,024 for narrow rows (more waves beyond: 23.6 M nonzeros, width 16: one wave 144 us, two 170) and not under 32 (0.5 M nonzeros, width 16: 15.4 us with 16, 12.5 with
// 32, 13.9 with 48), and are longer only where the pieces would need more than half a gigabyte.  A B beyond L2 takes a wave
// for every 64 MB, at most one per feature tile: waves go tile by tile, so each gathers from columns that stay in L2 (1 M
// nonzeros in even rows, B of 200 MB, 4 tiles: one wave 224 us, four 170).
static SplitShape split_shape(int64_t nnz, int m, int f, bool coo, bool even) {
  SplitShape s;
  const int v = (f + 3) / 4;
  const int longest = v <= 8 ? 1024 : 704, shortest = 32;
  s.lpn = v <= 4 ? 4 : 8;
  s.nv = 1;
  if (v > 8 && (v <= 16 ? nnz >= 500000 : nnz * v >= 5000000)) {
    const bool wide = even || nnz >= 2000000;
    const int few = coo || v <= 16 || !wide ? 2 : 3, many = coo ? 2 : wide ? 4 : 3;
    constexpr int weight[5] = {0, 0, 108, 100, 106};
    for (int nv = few, best = INT_MAX; nv <= many; ++nv) {
      const int cost = (v + 8 * nv - 1) / (8 * nv) * nv * weight[nv];
      if (cost < best) best = cost, s.nv = nv;
    }
  }
  const int tile = s.lpn * s.nv;
  s.tiles = (v + tile - 1) / tile;
  const int unit = 2 * s.lpn, per_block = kSplitWarps * (32 / s.lpn);
  const int64_t slots = static_cast<int64_t>(kNumSMs) * split_blocks_per_sm(s.nv, coo);        // blocks of a wave
  int64_t waves = (nnz * s.tiles + slots * per_block * longest - 1) / (slots * per_block * longest);
  const int64_t parts = (static_cast<int64_t>(m) * f * 4 + (64 << 20) - 1) >> 26;
  waves = max(waves, min(static_cast<int64_t>(s.tiles), parts));
  while (waves * slots < s.tiles) ++waves;
  const int64_t walks = waves * slots / s.tiles * per_block;                                    // chunks of a feature tile
  int64_t chunk = (nnz + walks - 1) / walks;
  chunk = ((chunk < shortest ? shortest : chunk) + unit - 1) / unit * unit;
  while ((nnz + chunk - 1) / chunk * s.tiles * tile * 32 > (512ll << 20)) chunk *= 2;
  s.chunk = static_cast<int>(chunk);
  s.nchunks = (nnz + chunk - 1) / chunk;
  return s;
}

static size_t split_bytes(const SplitShape& s) {
  return static_cast<size_t>(s.nchunks) * s.tiles * s.lpn * s.nv * 32;     // two pieces of 16-byte vectors
}

template <bool COO, int LPN, int NV, int BATCH>
static int launch_split(const SplitArgs& a, int tiles, float beta, cudaStream_t s) {
  constexpr int G = 32 / LPN;
  const int per_block = kSplitWarps * G;
  const dim3 grid(static_cast<unsigned>((a.nchunks + per_block - 1) / per_block), tiles);
  const int join_blocks = (a.nchunks + 3) / 4;
  const int clear_blocks = beta == 0.f ? (a.nempty * LPN + 127) / 128 : 0;
  const dim3 jgrid(join_blocks + clear_blocks, tiles);
  // Large multiplies start on idle SMs: a kernel that is scheduled behind the tile multiply's 226 KB of shared memory keeps
  // that split of the L1 array for its whole run (R-MAT 1 M vertices, width 602, back to back: 5.4 -> 7.5 ms).
  const bool early = a.nnz * tiles <= (1 << 21);
  cudaError_t e;
  if (COO || beta != 0.f) {      // COO is the accumulating operator only
    e = launch_pdl_if(early, spmm_split_kernel<LPN, NV, BATCH, true, COO>, grid, dim3(kSplitWarps * 32), 0, s, a);
    if (e == cudaSuccess) e = launch_pdl(spmm_split_join_kernel<LPN, NV, true, COO>, jgrid, dim3(128), 0, s, a, join_blocks);
  } else if constexpr (!COO) {
    e = launch_pdl_if(early, spmm_split_kernel<LPN, NV, BATCH, false, COO>, grid, dim3(kSplitWarps * 32), 0, s, a);
    if (e == cudaSuccess) e = launch_pdl(spmm_split_join_kernel<LPN, NV, false, COO>, jgrid, dim3(128), 0, s, a, join_blocks);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_spmm_block_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

template <bool COO>
static int dispatch_split(const SplitArgs& a, const SplitShape& sh, float beta, cudaStream_t stream) {
  if (sh.lpn == 4) return launch_split<COO, 4, 1, 8>(a, sh.tiles, beta, stream);
  if (sh.nv == 1) return launch_split<COO, 8, 1, 8>(a, sh.tiles, beta, stream);
  if (COO || sh.nv == 2) return launch_split<COO, 8, 2, 4>(a, sh.tiles, beta, stream);
  if constexpr (!COO) {
    if (sh.nv == 3) return launch_split<false, 8, 3, 4>(a, sh.tiles, beta, stream);
    return launch_split<false, 8, 4, 4>(a, sh.tiles, beta, stream);
  }
}

// Rows about as long as each other, as far as the host knows.
static bool even_rows(const cagnet_block* b) { return b->max_row >= 0 && b->max_row * static_cast<int64_t>(b->n) <= 4 * b->nnz; }

static SplitShape block_shape(const cagnet_block* b, int f) { return split_shape(b->nnz, b->m, f, false, even_rows(b)); }

static int run_split(const cagnet_block* b, const float* B, int64_t ldb, float* C, int64_t ldc, int f, float beta, void* ws,
                     cudaStream_t stream) {
  const SplitShape sh = block_shape(b, f);
  SplitArgs a = {};
  const int64_t padded = (b->nnz + kUnit - 1) / kUnit * kUnit;
  a.pairs = static_cast<const int2*>(b->split);
  a.first = reinterpret_cast<const unsigned*>(a.pairs + padded);
  a.rows = b->rows;
  a.empty = b->empty;
  a.nrows = b->nrows;
  a.nempty = b->nempty;
  a.B = B; a.C = C;
  a.part = static_cast<float*>(ws);
  a.nnz = b->nnz; a.ldb = ldb; a.ldc = ldc;
  a.f = f; a.f_eff = (f + 3) / 4 * 4;
  a.chunk = sh.chunk;
  a.nchunks = static_cast<int>(sh.nchunks);
  a.c_vec4 = (ldc % 4 == 0 && aligned(C, 16)) ? 1 : 0;
  return dispatch_split<false>(a, sh, beta, stream);
}
// The row kernels stay the better choice for small blocks of short rows, one launch instead of two and no pieces (ER, 13.5 K
// nonzeros, width 16: 3.0 us against 6.5; at 280 K nonzeros the two are level, at widths 17 - 32 from 40 K on), and for
// even rows of up to 16 columns until the chip is full (0.75 M nonzeros in rows of 125, width 6: 9.3 us against 12.8; 1 M
// in rows of 20: 16.7 against 18.0; 2 M: 29.0 against 28.2).  So they are for even rows of more than 384 columns in blocks
// that do not fill the chip many times over, if the rows are long or B's rows do not start on cache lines, which tiles of
// columns then cut (width 500: 0.75 M nonzeros in rows of 125 82 us against 86; 2 M in rows of 20, ldb 500, 317 against 348,
// but ldb 512 344 against 307).  At power-law rows the split wins from the smallest block on.
static bool use_split(const cagnet_block* b, int64_t ldb, int f) {
  if (!b->split || b->nnz <= 0 || spmm_forced_tile() != 0) return false;
  if (b->max_row < 0 || b->max_row > 256) return true;
  if (b->max_row <= 64 && b->nnz <= (f > 16 && f <= 32 ? 40000 : 150000)) return false;
  if (!even_rows(b)) return true;
  if (f > 384 && b->nnz <= 3000000) return ldb % 32 == 0 && b->nnz < 64 * static_cast<int64_t>(b->n);
  return f > 16 || b->nnz > 1500000;
}

// Dense tiles pay when the nonzeros they take over outweigh their three launches (tile_work: about 80 M gathered floats,
// 65 K vertices / 1.8 M nonzeros in tiles: width 16 33 -> 48 us, width 41 73 -> 66, width 128 117 -> 107).
static bool use_tiles(const cagnet_block* b, int f) {
  return b->tiles > 0 && b->rest && b->tile_nnz * static_cast<int64_t>(f) >= b->tile_work && spmm_forced_tile() == 0;
}

static bool b_aligned(const float* B, int64_t ldb) { return ldb % 4 == 0 && aligned(B, 16); }

// An unaligned B is copied once into rows of whole vectors when its rows are gathered often enough to pay for the copy.
static bool pad_pays(const cagnet_block* b) { return b->nnz >= 2 * static_cast<int64_t>(b->m); }

static size_t round256(size_t x) { return (x + 255) / 256 * 256; }

// B in rows of whole vectors: itself, or a copy at w (then w, ldb move on).
static const float* pad_rows(const float* B, int64_t& ldb, int m, int f, char*& w, cudaStream_t s) {
  if (b_aligned(B, ldb)) return B;
  const int ld4 = (f + 3) / 4;
  const int64_t total = static_cast<int64_t>(m) * ld4, blocks = (total + 255) / 256;
  float* out = reinterpret_cast<float*>(w);
  launch_pdl(pad_rows_kernel, dim3(static_cast<unsigned>(blocks < 16 * kNumSMs ? blocks : 16 * kNumSMs)), dim3(256), 0, s, B, ldb, m, f,
             ld4, reinterpret_cast<float4*>(out));
  w += round256(static_cast<size_t>(m) * ld4 * 16);
  ldb = ld4 * 4;
  return out;
}

static int split_launches(const cagnet_block* b, int64_t ldb, int32_t f) {
  if (use_tiles(b, f)) return split_launches(b->rest, ldb, f) + 2 + (b->joins > 0);
  if (use_split(b, ldb, f)) return 2;
  return (b->plan && b->hub_rows != 0) ? 2 : 1;
}

}  // namespace cagnet

using namespace cagnet;

extern "C" size_t cagnet_spmm_split_plan_bytes(int64_t nnz) {
  if (nnz <= 0) return 0;
  const size_t units = static_cast<size_t>((nnz + kUnit - 1) / kUnit);
  return units * kUnit * sizeof(int2) + units * sizeof(unsigned);
}

extern "C" int cagnet_spmm_split_plan_i32(const int32_t* rowptr, const int32_t* col, const float* val, const int32_t* rows,
                                          int32_t nrows, int64_t nnz, void* plan, size_t plan_bytes, void* stream) {
  if (nnz < 0 || nrows < 0) return fail(CAGNET_E_ARG, "cagnet_spmm_split_plan_i32: negative size");
  if (nnz == 0) return CAGNET_OK;
  if (!rowptr || !col || !val || !plan) return fail(CAGNET_E_ARG, "cagnet_spmm_split_plan_i32: null pointer");
  if (nnz > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_spmm_split_plan_i32: nnz %s%lld exceeds int32", "", nnz);
  if (plan_bytes < cagnet_spmm_split_plan_bytes(nnz)) return fail(CAGNET_E_WORKSPACE, "cagnet_spmm_split_plan_i32: plan buffer too small");
  if (!aligned(plan, 16)) return fail(CAGNET_E_ALIGN, "cagnet_spmm_split_plan_i32: plan buffer must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t padded = (nnz + kUnit - 1) / kUnit * kUnit;
  int2* pairs = static_cast<int2*>(plan);
  split_pairs_kernel<<<static_cast<unsigned>((padded + 255) / 256), 256, 0, s>>>(col, val, nnz, padded, pairs);
  split_rows_kernel<<<(nrows + 255) / 256, 256, 0, s>>>(rowptr, rows, nrows, pairs, reinterpret_cast<unsigned*>(pairs + padded));
  return check_launch("cagnet_spmm_split_plan_i32");
}

extern "C" size_t cagnet_spmm_block_workspace_bytes(const cagnet_block* b, const float* B, int64_t ldb, int32_t f) {
  if (!b || f <= 0 || b->n <= 0) return 0;
  const bool tiles = use_tiles(b, f);
  const cagnet_block* src = tiles ? b->rest : b;
  size_t bytes = tiles ? round256(cagnet_tile_core_workspace_bytes(b->tile_kbs, b->ctas, f)) : 0;
  if (use_split(src, ldb, f) && (b_aligned(B, ldb) || pad_pays(src))) {
    bytes += round256(split_bytes(block_shape(src, f)));
    if (!b_aligned(B, ldb)) bytes += round256(static_cast<size_t>(b->m) * ((f + 3) / 4) * 16);
  }
  return bytes;
}

extern "C" int cagnet_spmm_block_launches(const cagnet_block* b, int64_t ldb, int32_t f) {
  return b ? split_launches(b, ldb, f) : 0;
}

extern "C" int cagnet_spmm_block_f32(const cagnet_block* b, const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f,
                                     float beta, void* ws, size_t ws_bytes, void* stream) {
  if (!b) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: null block");
  if (ws_bytes < cagnet_spmm_block_workspace_bytes(b, B, ldb, f))
    return fail(CAGNET_E_WORKSPACE, "cagnet_spmm_block_f32: workspace too small");
  const bool tiles = use_tiles(b, f);
  const cagnet_block* src = tiles ? b->rest : b;
  if (!use_split(src, ldb, f) || !(b_aligned(B, ldb) || pad_pays(src)) || f <= 0 || b->n <= 0) {
    const int rc = spmm_rows_f32(src->rowptr, src->col, src->val, src->n, src->m, src->nnz, B, ldb, C, ldc, f, beta, src->plan,
                                 src->hub_rows, stream);
    if (rc != CAGNET_OK || !tiles) return rc;
  } else {
    if (!B || !C || !ws) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: null pointer");
    if (beta != 0.f && beta != 1.f) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: beta must be 0 or 1");
    if (ldb < f || ldc < f) return fail(CAGNET_E_ALIGN, "cagnet_spmm_block_f32: leading dimension smaller than f");
    char* w = static_cast<char*>(ws);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    B = pad_rows(B, ldb, b->m, f, w, s);
    const int rc = run_split(src, B, ldb, C, ldc, f, beta, w, s);
    if (rc != CAGNET_OK) return rc;
    ws = w + round256(split_bytes(block_shape(src, f)));
  }
  if (!tiles) return check_launch("cagnet_spmm_block_f32");
  return cagnet_tile_core_f32(b->tile_bits, b->tile_kb, b->panel_ptr, b->cta_ptr, b->ctas, b->panels, b->join_list, b->joins,
                              b->tile_cols, b->tile_kbs, b->panel_rows, b->panel_scale, b->col_scale, B, ldb, C, ldc, f, ws,
                              cagnet_tile_core_workspace_bytes(b->tile_kbs, b->ctas, f), stream);
}

extern "C" size_t cagnet_spmm_coo_workspace_bytes(int32_t m, int64_t nnz, const float* B, int64_t ldb, int32_t f) {
  if (nnz <= 0 || f <= 0) return 0;
  return round256(split_bytes(split_shape(nnz, m, f, true, false))) + (b_aligned(B, ldb) ? 0 : round256(static_cast<size_t>(m) * ((f + 3) / 4) * 16));
}

extern "C" int cagnet_spmm_coo_f32(const int32_t* rows, const int32_t* cols, const float* vals, int32_t n, int32_t m, int64_t nnz,
                                   const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f, const int32_t* status,
                                   void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || m < 0 || nnz < 0 || f < 0) return fail(CAGNET_E_ARG, "cagnet_spmm_coo_f32: negative size");
  if (n == 0 || nnz == 0 || f == 0) return CAGNET_OK;
  if (!rows || !cols || !vals || !B || !C || !ws) return fail(CAGNET_E_ARG, "cagnet_spmm_coo_f32: null pointer");
  if (nnz > INT_MAX) return fail(CAGNET_E_OVERFLOW, "cagnet_spmm_coo_f32: nnz %s%lld exceeds int32", "", nnz);
  if (ldb < f || ldc < f) return fail(CAGNET_E_ALIGN, "cagnet_spmm_coo_f32: leading dimension smaller than f");
  if (ws_bytes < cagnet_spmm_coo_workspace_bytes(m, nnz, B, ldb, f)) return fail(CAGNET_E_WORKSPACE, "cagnet_spmm_coo_f32: workspace too small");
  char* w = static_cast<char*>(ws);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  B = pad_rows(B, ldb, m, f, w, s);
  const SplitShape sh = split_shape(nnz, m, f, true, false);
  SplitArgs a = {};
  a.coo_rows = rows; a.coo_cols = cols; a.coo_vals = vals; a.status = status;
  a.nrows = n;                 // no chunk starts in row n
  a.B = B; a.C = C;
  a.part = reinterpret_cast<float*>(w);
  a.nnz = nnz; a.ldb = ldb; a.ldc = ldc;
  a.f = f; a.f_eff = (f + 3) / 4 * 4;
  a.chunk = sh.chunk;
  a.nchunks = static_cast<int>(sh.nchunks);
  a.c_vec4 = (ldc % 4 == 0 && aligned(C, 16)) ? 1 : 0;
  return dispatch_split<true>(a, sh, 1.f, s);
}
