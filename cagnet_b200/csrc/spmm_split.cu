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

constexpr int kUnit = 32;               // granularity of the row bookkeeping, nonzeros
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
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// C[row, this lane's columns] = acc (+ the old value); columns >= f are never written.
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
        float4 v = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
        if (add) {
          const float4 o = *reinterpret_cast<const float4*>(p);
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        *reinterpret_cast<float4*>(p) = v;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < live) p[j] = add ? p[j] + acc[k][j] : acc[k][j];
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

template <int LPN, int NV, int BATCH, bool ADD>
__global__ void __launch_bounds__(kSplitWarps * 32) spmm_split_kernel(SplitArgs a) {
  constexpr int G = 32 / LPN;
  constexpr int PL = (2 * LPN >= BATCH) ? 1 : BATCH / (2 * LPN);   // 16-byte loads (2 pairs) per lane and stage
  constexpr int SL = 2 * LPN * PL;                                 // pairs per lane group and stage
  constexpr int TILE = LPN * 4 * NV;
  static_assert(SL <= kUnit && SL % BATCH == 0, "a stage lies inside a unit");
  __shared__ __align__(16) int2 stage_s[kSplitWarps][G][SL];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPN, l = lane % LPN;
  const int chunk_id = (blockIdx.x * kSplitWarps + warp) * G + sub;
  if ((blockIdx.x * kSplitWarps + warp) * G >= a.nchunks) return;        // whole warps
  const int column0 = blockIdx.y * TILE + l * 4;
  const int nvalid = column0 >= a.f_eff ? 0 : min(NV, (a.f_eff - column0 + LPN * 4 - 1) / (LPN * 4));
  const int64_t start = static_cast<int64_t>(chunk_id) * a.chunk;
  const int len = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(a.chunk), a.nnz - start)));
  const int2* src = a.pairs + start;
  int2* stage = stage_s[warp][sub];
  const unsigned fw = len > 0 ? __ldg(a.first + start / kUnit) : 0u;
  int k = static_cast<int>(fw & ~kMid);         // position in `rows` of the row being summed
  bool head = (fw & kMid) != 0;                 // it began in an earlier chunk
  const float* bt = a.B + column0;
  float* piece = a.part + (static_cast<int64_t>(blockIdx.y) * a.nchunks + chunk_id) * (2 * TILE) + l * 4;

  float acc[NV][4];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[v][j] = 0.f;
  bool open = false;      // acc holds terms of a row whose last nonzero has not been met

  auto load_pairs = [&](int at, int4 (&q)[PL]) {
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = at + (i * LPN + l) * 2;
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
    for (int i = 0; i < PL; ++i) *reinterpret_cast<int4*>(stage + (i * LPN + l) * 2) = nxt[i];
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
            split_store<LPN, NV>(a, a.rows ? __ldg(a.rows + k) : k, column0, nvalid, ADD, acc);
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
template <int LPN, int NV, bool ADD>
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
  const int upc = a.chunk / kUnit;
  auto start_of = [&](int c) { return __ldg(a.first + static_cast<int64_t>(c) * upc); };
  unsigned row_k = 0;
  int lo = e;                                    // chunks lo .. e start in row row_k
  bool mine = false;
  if (e < a.nchunks) {
    // the row bookkeeping is constant: it may be read before the pieces are there
    const unsigned fw = start_of(e);
    row_k = fw & ~kMid;
    const unsigned next = e + 1 < a.nchunks ? start_of(e + 1) & ~kMid : static_cast<unsigned>(a.nrows);
    mine = (fw & kMid) && next != row_k;         // next == row_k: the row runs through this chunk
    while (mine) {                               // first chunk that starts with this row, 32 candidates at a time
      const int c = lo - 1 - lane;
      const bool same = c >= 0 && (start_of(c) & ~kMid) == row_k;
      const unsigned m = __ballot_sync(0xffffffffu, same);
      const int run = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
      lo -= run;
      if (run < 32) break;
    }
    if (mine && (start_of(lo) & kMid)) lo -= 1;  // it began inside the chunk before
  }
  pdl_wait();
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

// Lane mapping by width (vectors of 4 columns per gathered row), measured on R-MAT graphs of 0.1 - 115 M nonzeros:
// one group per row segment as narrow as the row allows (more nonzeros in flight per warp), two or three vectors per
// lane from 9 vectors on (fewer broadcasts per byte: width 41 0.67 -> 0.58 ms, width 128 with 16 x 2 lanes 1.18 ms against
// 1.42 with 32 x 1) unless the matrix is so small that it cannot fill the chip (below 1 M nonzeros one vector per lane
// gives twice the warps: width 48, 100 K nonzeros 9.2 against 10.2 us).
// Chunk length: about 26,000 chunk walks per launch (6 resident groups per lane group slot), in [32, 512]; shorter
// chunks start more walks than they fill, longer ones leave a ragged last wave.  Doubled where the pieces would need more
// than half a gigabyte.
static SplitShape split_shape(int64_t nnz, int f) {
  SplitShape s;
  const int v = (f + 3) / 4;
  if (v <= 4) s.lpn = 4, s.nv = 1;
  else if (v <= 8) s.lpn = 8, s.nv = 1;
  else if (v <= 16 && nnz < (1 << 20)) s.lpn = 16, s.nv = 1;
  else if (v <= 16) s.lpn = 8, s.nv = 2;
  else if (v <= 24) s.lpn = 8, s.nv = 3;
  else s.lpn = 16, s.nv = 2;
  const int tile = s.lpn * s.nv;
  s.tiles = (v + tile - 1) / tile;
  s.chunk = kUnit;
  while (s.chunk < 512 && nnz * s.tiles > static_cast<int64_t>(s.chunk) * 37000) s.chunk *= 2;
  while (((nnz + s.chunk - 1) / s.chunk) * s.tiles * tile * 32 > (512ll << 20)) s.chunk *= 2;
  s.nchunks = (nnz + s.chunk - 1) / s.chunk;
  return s;
}

static size_t split_bytes(int64_t nnz, int f) {
  const SplitShape s = split_shape(nnz, f);
  return static_cast<size_t>(s.nchunks) * s.tiles * s.lpn * s.nv * 32;     // two pieces of 16-byte vectors
}

template <int LPN, int NV, int BATCH>
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
  if (beta != 0.f) {
    e = launch_pdl_if(early, spmm_split_kernel<LPN, NV, BATCH, true>, grid, dim3(kSplitWarps * 32), 0, s, a);
    if (e == cudaSuccess) e = launch_pdl(spmm_split_join_kernel<LPN, NV, true>, jgrid, dim3(128), 0, s, a, join_blocks);
  } else {
    e = launch_pdl_if(early, spmm_split_kernel<LPN, NV, BATCH, false>, grid, dim3(kSplitWarps * 32), 0, s, a);
    if (e == cudaSuccess) e = launch_pdl(spmm_split_join_kernel<LPN, NV, false>, jgrid, dim3(128), 0, s, a, join_blocks);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_spmm_block_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

static int run_split(const cagnet_block* b, const float* B, int64_t ldb, float* C, int64_t ldc, int f, float beta, void* ws,
                     cudaStream_t stream) {
  const SplitShape sh = split_shape(b->nnz, f);
  SplitArgs a;
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
  if (sh.lpn == 4) return launch_split<4, 1, 8>(a, sh.tiles, beta, stream);
  if (sh.lpn == 8 && sh.nv == 1) return launch_split<8, 1, 8>(a, sh.tiles, beta, stream);
  if (sh.lpn == 8 && sh.nv == 2) return launch_split<8, 2, 4>(a, sh.tiles, beta, stream);
  if (sh.lpn == 8) return launch_split<8, 3, 4>(a, sh.tiles, beta, stream);
  if (sh.nv == 1) return launch_split<16, 1, 4>(a, sh.tiles, beta, stream);
  return launch_split<16, 2, 4>(a, sh.tiles, beta, stream);
}

// The row kernels stay the better choice for small blocks of short rows: one launch instead of two and no pieces (ER,
// 13.5 K nonzeros, width 16: 3.0 us against 6.5; at 280 K nonzeros the two are level, at power-law rows the split wins
// from the smallest block on).
static bool use_split(const cagnet_block* b) {
  return b->split && b->nnz > 0 && !(b->max_row >= 0 && b->max_row <= 64 && b->nnz <= 150000) && spmm_forced_tile() == 0;
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

int split_launches(const cagnet_block* b, int32_t f) {
  if (use_tiles(b, f)) return split_launches(b->rest, f) + 2 + (b->joins > 0);
  if (use_split(b)) return 2;
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
  if (use_split(src) && (b_aligned(B, ldb) || pad_pays(src))) {
    bytes += round256(split_bytes(src->nnz, f));
    if (!b_aligned(B, ldb)) bytes += round256(static_cast<size_t>(b->m) * ((f + 3) / 4) * 16);
  }
  return bytes;
}

extern "C" int cagnet_spmm_block_launches(const cagnet_block* b, int32_t f) { return b ? split_launches(b, f) : 0; }

extern "C" int cagnet_spmm_block_f32(const cagnet_block* b, const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f,
                                     float beta, void* ws, size_t ws_bytes, void* stream) {
  if (!b) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: null block");
  if (ws_bytes < cagnet_spmm_block_workspace_bytes(b, B, ldb, f))
    return fail(CAGNET_E_WORKSPACE, "cagnet_spmm_block_f32: workspace too small");
  const bool tiles = use_tiles(b, f);
  const cagnet_block* src = tiles ? b->rest : b;
  if (!use_split(src) || !(b_aligned(B, ldb) || pad_pays(src)) || f <= 0 || b->n <= 0) {
    const int rc = spmm_rows_f32(src->rowptr, src->col, src->val, src->n, src->m, src->nnz, B, ldb, C, ldc, f, beta, src->plan,
                                 src->hub_rows, stream);
    if (rc != CAGNET_OK || !tiles) return rc;
  } else {
    if (!B || !C || !ws) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: null pointer");
    if (beta != 0.f && beta != 1.f) return fail(CAGNET_E_ARG, "cagnet_spmm_block_f32: beta must be 0 or 1");
    if (ldb < f || ldc < f) return fail(CAGNET_E_ALIGN, "cagnet_spmm_block_f32: leading dimension smaller than f");
    char* w = static_cast<char*>(ws);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!b_aligned(B, ldb)) {
      const int ld4 = (f + 3) / 4;
      const size_t bytes = round256(static_cast<size_t>(b->m) * ld4 * 16);
      const int64_t total = static_cast<int64_t>(b->m) * ld4;
      const int64_t blocks = (total + 255) / 256;
      launch_pdl(pad_rows_kernel, dim3(static_cast<unsigned>(blocks < 16 * kNumSMs ? blocks : 16 * kNumSMs)), dim3(256), 0, s, B, ldb,
                 b->m, f, ld4, reinterpret_cast<float4*>(w));
      B = reinterpret_cast<const float*>(w);
      ldb = ld4 * 4;
      w += bytes;
    }
    const int rc = run_split(src, B, ldb, C, ldc, f, beta, w, s);
    if (rc != CAGNET_OK) return rc;
    ws = w + round256(split_bytes(src->nnz, f));
  }
  if (!tiles) return check_launch("cagnet_spmm_block_f32");
  return cagnet_tile_core_f32(b->tile_bits, b->tile_kb, b->panel_ptr, b->cta_ptr, b->ctas, b->panels, b->join_list, b->joins,
                              b->tile_cols, b->tile_kbs, b->panel_rows, b->panel_scale, b->col_scale, B, ldb, C, ldc, f, ws,
                              cagnet_tile_core_workspace_bytes(b->tile_kbs, b->ctas, f), stream);
}
