// Dense tiles of a NORMALISED adjacency block as bit matrices on the tensor cores (tcgen05, sm_100a).
//
// With rows and columns in order of degree a power-law block is far from uniformly sparse: on the 233K-vertex /
// 115M-nonzero benchmark graph 80 % of the nonzeros lie in the 58,000 tiles of 256 x 64 cells that are at least 2 % full,
// on a 1 M-vertex R-MAT graph with 31 nonzeros per row 30 % in 7,600.  A normalised value factors, val[r, c] = rs[r] * cs[c]
// for a simple edge (partition.coalesce_block), so a tile is diag(rs) . Bits . diag(cs) with one BIT per cell (2 KB per tile
// against 8 bytes per nonzero: 41 nonzeros' worth of index stream at 2 % density carries 328) and its product with B is
//        rs . ( Bits . Y ),     Y = cs . B cut into three bf16 terms that carry 24 significant bits between them.
// Bits are exact in bf16, products of a bit and a term are exact, sums are fp32 in tensor memory: against fp64 the whole
// product is off by 5e-8 .. 1e-7 of its norm, as fp32 multiply-adds are (1e-7 .. 2e-7); 3e-7 over 1,600 column blocks.
//
//   tile_operand_kernel   Y's terms for the columns that occur in tiles, laid out as the multiply reads them
//   tile_core_kernel      persistent over each block's share of the tiles, sorted by row panel (256 rows):
//       warp 0            bulk copies of the next tiles' operand (3 NT x 64 bf16) and bits (2 KB) into a ring of stages
//       warps 12 - 27     turn a row's 64 bits into 64 packed bf16 values (one shift and one AND per pair of cells: the
//                         bf16 number 2 is a single bit) and store them to TENSOR memory, where the multiply takes its A
//                         operand from: no shared-memory traffic for A, no swizzle, no 16-fold expansion of what L2 delivers
//       warp 1            tcgen05.mma kind::f16, M = 128 twice per tile against the same B (one B tile feeds 256 rows: 32 B/clk
//                         of L2 traffic per SM at the full rate)
//       warps 4 - 11      panel sums out of tensor memory, through a shared-memory exchange into whole C row segments
//   tile_join_kernel      panels cut over several blocks: pieces added in block order
// Widths <= 64 put the three terms side by side (N = 3 NT, one product per k step, NT = width rounded up to 16), wider ones
// add three products of N = NT <= 192 into one sum.  At N >= 128 the steady state runs at the tensor pipe's rate (1,921
// clocks per tile at NT = 160, 1,920 by arithmetic; 1.27 PFLOP/s over the benchmark graph's width-602 product, 92 % of the
// sustained cuBLAS bf16 rate under the power cap); at NT = 16 a tile takes 350 - 450 clocks, the round trip from a finished
// product to the next expanded operand.  Every sum has one order: results are bit-reproducible.
#include <cuda_bf16.h>
#include <limits.h>

#include "common.cuh"
#include "tc.cuh"

namespace cagnet {

constexpr int kTileRows = 256;            // rows of a tile: two M = 128 accumulators
constexpr int kTileCols = 64;             // columns of a tile: one 128-byte swizzled line of bf16 per operand row
constexpr int kTileWords = kTileRows * 2; // 32-bit words of a tile's bit matrix: two per row
constexpr int kTileBitsBytes = kTileWords * 4;
constexpr int kMaxNT = 192;                // widest feature tile: two fp32 sums of 192 columns beside 128 operand columns
constexpr int kTileThreads = 896;         // warp 0 loads, warp 1 multiplies, warps 4-11 store sums, warps 12-27 expand bits
constexpr int kExchangeBytes = 8 * 32 * 36 * 4;   // storing warps: 32 rows x 32 columns each, rows padded to 36 floats
constexpr int kMaxStages = 16;

// ---------------------------------------------------------------------------------------------- plan
// counts[(rank_r / 256) * nkb + rank_c / 64] += 1 over the entries whose ranks lie inside the searched square
__global__ void tile_count_kernel(const int* __restrict__ rowptr, const int* __restrict__ col, int n,
                                  const int* __restrict__ rank_r, const int* __restrict__ rank_c, int lim_r, int lim_c,
                                  int nkb, int* __restrict__ counts) {
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const int rr = rank_r[warp];
  if (rr >= lim_r) return;
  int* c = counts + static_cast<int64_t>(rr / kTileRows) * nkb;
  for (int e = rowptr[warp] + lane; e < rowptr[warp + 1]; e += 32) {
    const int rc = rank_c[col[e]];
    if (rc < lim_c) atomicAdd(c + rc / kTileCols, 1);
  }
}

// The bit of row r, column k of a tile: word 2 r + k / 32; inside a word the columns are ordered so that the pair
// (2 j, 2 j + 1) sits at bits j and j + 16, which is what one shift and one AND turn into a packed bf16 pair.
__device__ __forceinline__ int tile_bit(int k) { return ((k & 31) >> 1) + ((k & 1) << 4); }

// Sets the bits of the entries that belong to a dense tile and whose value is exactly the product of its factors;
// keep[e] = 1 for every other entry.  An entry listed twice keeps its second occurrence outside.
__global__ void tile_fill_kernel(const int* __restrict__ rowptr, const int* __restrict__ col, const float* __restrict__ val,
                                 int n, const int* __restrict__ rank_r, const int* __restrict__ rank_c, int lim_r,
                                 int lim_c, int nkb, const int* __restrict__ tile_of, const float* __restrict__ rs,
                                 const float* __restrict__ cs, unsigned* __restrict__ bits, uint8_t* __restrict__ keep) {
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const int rr = rank_r[warp];
  const float r = rs[warp];
  for (int e = rowptr[warp] + lane; e < rowptr[warp + 1]; e += 32) {
    bool out = true;
    const int c = col[e];
    const int rc = rank_c[c];
    if (rr < lim_r && rc < lim_c) {
      const int t = tile_of[static_cast<int64_t>(rr / kTileRows) * nkb + rc / kTileCols];
      if (t >= 0 && val[e] == __fmul_rn(r, cs[c])) {
        const unsigned bit = 1u << tile_bit(rc % kTileCols);
        unsigned* w = bits + static_cast<int64_t>(t) * kTileWords + (rr % kTileRows) * 2 + (rc % kTileCols) / 32;
        out = (atomicOr(w, bit) & bit) != 0;
      }
    }
    keep[e] = out;
  }
}

// ---------------------------------------------------------------------------------------------- operand
// One block per 64-column block of the core and feature tile: the 64 rows of B it names, scaled by cs, cut into three
// bf16 terms and laid out as the multiply reads them: row (term * NT + j) holds feature j of all 64 columns, 128 bytes
// in the 128-byte-swizzled order.
__global__ void __launch_bounds__(256) tile_operand_kernel(const float* __restrict__ B, int64_t ldb, const int* __restrict__ cols,
                                                           const float* __restrict__ cs, int f, int NT, int b_vec4,
                                                           char* __restrict__ out) {
  extern __shared__ float xs[];            // [64][NT + 1]
  pdl_trigger();
  pdl_wait();
  const int kb = blockIdx.x, ft = blockIdx.y;
  const int f0 = ft * NT;
  const int w = min(NT, f - f0);
  const int ld = NT + 1;
  const int nv = NT / 4;
  for (int i = threadIdx.x; i < kTileCols * nv; i += blockDim.x) {
    const int k = i / nv, j = (i % nv) * 4;
    const int c = __ldg(cols + kb * kTileCols + k);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (c >= 0 && j < w) {
      const float s = __ldg(cs + c);
      const float* p = B + static_cast<int64_t>(c) * ldb + f0 + j;
      if (b_vec4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = q.x * s;
        v[1] = j + 1 < w ? q.y * s : 0.f;
        v[2] = j + 2 < w ? q.z * s : 0.f;
        v[3] = j + 3 < w ? q.w * s : 0.f;
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (j + t < w) v[t] = __ldg(p + t) * s;
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) xs[k * ld + j + t] = v[t];
  }
  __syncthreads();
  char* tile = out + (static_cast<int64_t>(ft) * gridDim.x + kb) * (3 * NT * 128);
  for (int i = threadIdx.x; i < NT * 8; i += blockDim.x) {
    const int j = i % NT, c = i / NT;        // feature, 16-byte piece (8 columns)
    __align__(16) unsigned short y[3][8];
#pragma unroll
    for (int t = 0; t < 8; ++t) split3(xs[(c * 8 + t) * ld + j], y[0][t], y[1][t], y[2][t]);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int row = p * NT + j;
      *reinterpret_cast<uint4*>(tile + row * 128 + ((c ^ (row & 7)) << 4)) = *reinterpret_cast<const uint4*>(y[p]);
    }
  }
}

struct TileArgs {
  const unsigned* bits;        // [T][256][2]
  const int* tile_kb;          // [T] column block of each tile; tiles sorted by row panel
  const int* panel_ptr;        // [panels + 1] first tile of each row panel
  const int* cta_ptr;          // [gridDim.x + 1] first tile of each block's share
  const int* rows;             // [panels * 256] row of C behind each panel row, -1 = none
  const float* rs;             // [panels * 256] row factor of each panel row, 0 = none
  const int4* joins;           // panels cut over several blocks: (panel, first block, last block + 1, 0)
  const char* operand;         // [FT][nkb][3 NT][128 bytes]
  float* C;
  float* part;                 // [2 * gridDim.x][256][NT] per feature tile
  int64_t ldc;
  int panels, nkb, NT, f, stages, c_vec4;
};

// Set when a wait of the multiply ran out (a fault of this library: the block then gave up and its part of C is missing).
__device__ int g_tile_error;

// The panel that holds tile u.
__device__ __forceinline__ int tile_panel(const TileArgs& a, int u) {
  int lo = 0, hi = a.panels - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(a.panel_ptr + mid) <= u) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// WIDE: the three terms are accumulated into one sum by three products of N = NT; otherwise they sit side by side in
// one product of N = 3 NT and are added when the sums are read.
template <bool WIDE>
__global__ void __launch_bounds__(kTileThreads, 1) tile_core_kernel(TileArgs a) {
  extern __shared__ __align__(1024) char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * kMaxStages + 10];
  __shared__ unsigned tmem_base_s;
  __shared__ int dead_s;
  char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int NT = a.NT;
  const int bbytes = 3 * NT * 128;
  const int stage_bytes = bbytes + kTileBitsBytes;
  const int S = a.stages;
  const int N = WIDE ? NT : 3 * NT;
  // Tensor memory: AS sets of sums (two: the next panel's products run under this one's stores) below NB operand
  // buffers of 64 columns (two 128 x 64 bf16 halves) at the top.  Four buffers cover the round trip from a finished
  // product to the next expanded tile where a tile's products are short (N <= 96: 0.2 us).
  const int NB = !WIDE && N <= 96 ? 4 : 2;
  const int AS = 4 * N <= 512 - 64 * NB ? 2 : 1;
  const int a_col = 512 - 64 * NB;
  const unsigned bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8 * s; };
  auto done = [&](int s) { return bar0 + 8 * (kMaxStages + s); };
  auto a_full = [&](int b) { return bar0 + 8 * (2 * kMaxStages + b); };
  auto acc_full = [&](int b) { return bar0 + 8 * (2 * kMaxStages + 4 + b); };
  auto acc_empty = [&](int b) { return bar0 + 8 * (2 * kMaxStages + 6 + b); };
  auto acc_at = [&](int set, int half) { return static_cast<unsigned>((set * 2 + half) * N); };
  const unsigned drain = bar0 + 8 * (2 * kMaxStages + 8);
  volatile int* dead = &dead_s;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(done(s), 1);         // the products that read the stage are complete
    }
    for (int b = 0; b < 4; ++b) mbar_init(a_full(b), 8);       // one arrival per expanding warp of the buffer's group
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), 8);    // one arrival per storing warp
    }
    mbar_init(drain, 1);
    dead_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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
  const int u0 = __ldg(a.cta_ptr + blockIdx.x), u1 = __ldg(a.cta_ptr + blockIdx.x + 1);
  const int ft = blockIdx.y;
  const int count = u1 - u0;

  pdl_trigger();
  pdl_wait();
  if (count <= 0) {
    // nothing: a block may get no tile when there are few
  } else if (warp == 0) {
    int s = 0, issued = 0;
    unsigned ph = 0;
    bool ok = true;
    const char* operand = a.operand + static_cast<int64_t>(ft) * a.nkb * bbytes;
    for (int base = 0; base < count && ok; base += 32) {
      // the next 32 tiles' column blocks in one load
      const int info = base + lane < count ? __ldg(a.tile_kb + u0 + base + lane) : 0;
      const int live = min(32, count - base);
      for (int i = 0; i < live; ++i) {
        const int kb = __shfl_sync(0xffffffffu, info, i);
        if (lane == 0) {
          ok = mbar_wait(done(s), ph ^ 1, dead);
          if (ok) {
            const unsigned dst = smem_u32(smem + s * stage_bytes);
            mbar_expect(full(s), stage_bytes);
            bulk_load(dst, operand + static_cast<int64_t>(kb) * bbytes, bbytes, full(s));
            bulk_load(dst + bbytes, a.bits + static_cast<int64_t>(u0 + base + i) * kTileWords, kTileBitsBytes, full(s));
            ++issued;
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
    if (lane == 0 && *dead) {        // a wait ran out: the copies in flight still write into this block's shared memory
      for (int k = max(0, issued - S); k < issued; ++k)
        for (int i = 0; i < kWaitLimit && !mbar_try(full(k % S), (k / S) & 1); ++i) {}
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // kind::f16: D fp32, A and B bf16, both K-major
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned>(N >> 3) << 17) | (8u << 24);
      const unsigned term = static_cast<unsigned>(NT * 128) >> 4;
      int s = 0, b = 0, c = 0;
      unsigned aph = 0, cph = 0;
      int panel = tile_panel(a, u0);
      int end = min(u1, __ldg(a.panel_ptr + panel + 1));
      // An operand buffer is announced by warps that have seen its stage arrive, so it is the only thing to wait for;
      // the wait for tile u + 1 stands between the two halves of tile u, whose products run meanwhile.
      bool ok = mbar_wait(a_full(0), 0, dead);
      for (int u = u0; u < u1 && ok; ++panel) {
        const int next_end = end < u1 ? min(u1, __ldg(a.panel_ptr + panel + 2)) : end;
        ok = mbar_wait(acc_empty(c), cph ^ 1, dead);
        unsigned accumulate = 0;
        for (; u < end && ok; ++u) {
          const unsigned long long desc = smem_desc(smem_u32(smem + s * stage_bytes));
          tc_fence_after();
          const int nb = b + 1 == NB ? 0 : b + 1;
          const unsigned naph = nb ? aph : aph ^ 1;
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            const unsigned d = tmem + acc_at(c, p);
            const unsigned at = tmem + a_col + (b * 2 + p) * 32;
#pragma unroll
            for (int t = 0; t < (WIDE ? 3 : 1); ++t)
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)
                tc_mma_ts(d, at + ks * 8, desc + t * term + ks * 2, idesc, (t == 0 && ks == 0) ? accumulate : 1u);
            if (p == 0 && u + 1 < u1) ok = mbar_wait(a_full(nb), naph, dead);
          }
          accumulate = 1;
          tc_commit(done(s));
          if (++s == S) s = 0;
          b = nb;
          aph = naph;
        }
        if (ok) tc_commit(acc_full(c));
        if (++c == AS) { c = 0; cph ^= 1; }
        end = next_end;
      }
      if (*dead) {        // products in flight still use the tensor memory
        tc_commit(drain);
        for (int i = 0; i < kWaitLimit && !mbar_try(drain, 0); ++i) {}
      }
    }
  } else if (warp >= 12) {
    // two groups of eight warps expand every other tile, each into its own operand buffer
    const int grp = (warp - 12) >> 3, p = ((warp - 12) >> 2) & 1;
    const int quad = (warp & 3) * 32;              // TMEM lanes this warp can reach
    const int prow = p * 128 + quad + lane;        // row inside the 256-row tile
    const unsigned dst = tmem + (static_cast<unsigned>(quad) << 16) + a_col + p * 32;
    int s = grp % S, ds = s, b = grp;              // ds, dph: stage and phase of the tile NB before, whose products free the buffer
    unsigned ph = static_cast<unsigned>(grp / S) & 1, dph = ph;
    // A stage's phase is known by its parity alone, so a tile may only be waited for once the stage's previous tile has
    // been consumed.  Narrow products have at least NB + 2 stages: the tile two before, which this warp has expanded,
    // was preceded by the end of tile i - 2 - NB >= i - S.  Wide ones wait for the products first.
    auto buffer_free = [&](int i) {
      if (i < NB) return true;
      if (!mbar_wait(done(ds), dph, dead)) return false;
      ds += 2;
      if (ds >= S) { ds -= S; dph ^= 1; }
      return true;
    };
    for (int i = grp; i < count; i += 2) {
      if (WIDE && !buffer_free(i)) break;
      if (!mbar_wait(full(s), ph, dead)) break;
      const uint2 w = *reinterpret_cast<const uint2*>(smem + s * stage_bytes + bbytes + prow * 8);
      unsigned r[32];
#pragma unroll
      for (int j = 0; j < 15; ++j) {
        r[14 - j] = (w.x << j) & 0x40004000u;      // bf16 2.0 where the bit is set
        r[30 - j] = (w.y << j) & 0x40004000u;
      }
      r[15] = (w.x >> 1) & 0x40004000u;
      r[31] = (w.y >> 1) & 0x40004000u;
      if (!WIDE && !buffer_free(i)) break;
      tc_fence_after();
      tmem_st32(dst + b * 64, r);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full(b));
      b = b + 2 >= NB ? grp : b + 2;
      s += 2;
      if (s >= S) { s -= S; ph ^= 1; }
    }
  } else if (warp >= 4) {
    const int p = (warp - 4) >> 2;                 // panel half
    const int quad = (warp & 3) * 32;
    const unsigned lane_base = static_cast<unsigned>(quad) << 16;
    const int prow = p * 128 + quad + lane;
    float* xch = reinterpret_cast<float*>(smem + S * stage_bytes) + (warp - 4) * (32 * 36);     // 32 rows x 32 columns, padded
    const int f0 = ft * NT;
    const int width = min(NT, a.f - f0);
    int c = 0;
    unsigned cph = 0;
    int panel = tile_panel(a, u0);
    int first = __ldg(a.panel_ptr + panel), next = __ldg(a.panel_ptr + panel + 1);
    int row = __ldg(a.rows + static_cast<int64_t>(panel) * kTileRows + prow);
    float rscale = __ldg(a.rs + static_cast<int64_t>(panel) * kTileRows + prow);
    for (int u = u0; u < u1; ++panel) {
      const bool partial = first < u0 || next > u1;
      const int slot = (ft * gridDim.x + blockIdx.x) * 2 + (first < u0 ? 0 : 1);
      float* piece = a.part + (static_cast<int64_t>(slot) * kTileRows + p * 128 + quad) * NT;
      const float scale = partial ? 0.5f : 0.5f * rscale;      // a set bit is the bf16 number 2
      // the following panel's rows travel while this one's products run
      int next2 = next, row2 = -1;
      float rscale2 = 0.f;
      if (next < u1) {
        next2 = __ldg(a.panel_ptr + panel + 2);
        row2 = __ldg(a.rows + static_cast<int64_t>(panel + 1) * kTileRows + prow);
        rscale2 = __ldg(a.rs + static_cast<int64_t>(panel + 1) * kTileRows + prow);
      }
      // Eight lanes per row, 128 contiguous bytes each.  The old values of a piece of 32 columns are asked for before
      // the sums are there (wide products) or added by the memory system (narrow ones: every element of C gets exactly
      // one addition from this kernel, so the order of the additions does not matter).
      const int lj = (lane & 7) * 4;
      float4 old[WIDE ? 8 : 1];
      auto load_old = [&](int j0) {
        if constexpr (WIDE) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int crow = __shfl_sync(0xffffffffu, row, i * 4 + (lane >> 3));
            old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!partial && crow >= 0 && j0 + lj + 4 <= width && a.c_vec4)
              old[i] = __ldcg(reinterpret_cast<const float4*>(a.C + static_cast<int64_t>(crow) * a.ldc + f0 + j0 + lj));
          }
        }
      };
      load_old(0);
      if (!mbar_wait(acc_full(c), cph, dead)) break;
      tc_fence_after();
      const unsigned acc = lane_base + tmem + acc_at(c, p);
      for (int j0 = 0; j0 < NT; j0 += 32) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int j = j0 + 16 * h;
          if (j < NT) {
            unsigned x[16];
            tmem_ld16(acc + j, x);
            if constexpr (!WIDE) {
              unsigned y[16], z[16];
              tmem_ld16(acc + NT + j, y);
              tmem_ld16(acc + 2 * NT + j, z);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int t = 0; t < 16; ++t)
                x[t] = __float_as_uint(scale * (__uint_as_float(x[t]) + (__uint_as_float(y[t]) + __uint_as_float(z[t]))));
            } else {
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int t = 0; t < 16; ++t) x[t] = __float_as_uint(scale * __uint_as_float(x[t]));
            }
#pragma unroll
            for (int t = 0; t < 16; t += 4)
              *reinterpret_cast<uint4*>(xch + lane * 36 + 16 * h + t) = make_uint4(x[t], x[t + 1], x[t + 2], x[t + 3]);
          }
        }
        __syncwarp();
        const int jj = j0 + lj;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          const int crow = __shfl_sync(0xffffffffu, row, r);
          float4 v = *reinterpret_cast<const float4*>(xch + r * 36 + lj);
          if (jj < NT) {
            if (partial) {
              *reinterpret_cast<float4*>(piece + static_cast<int64_t>(r) * NT + jj) = v;
            } else if (crow >= 0) {
              float* cp = a.C + static_cast<int64_t>(crow) * a.ldc + f0 + jj;
              if (jj + 4 <= width && a.c_vec4) {
                if constexpr (WIDE) {
                  v.x += old[i].x; v.y += old[i].y; v.z += old[i].z; v.w += old[i].w;
                  *reinterpret_cast<float4*>(cp) = v;
                } else {
                  red_add4(cp, v);
                }
              } else {
                if (jj + 0 < width) atomicAdd(cp + 0, v.x);
                if (jj + 1 < width) atomicAdd(cp + 1, v.y);
                if (jj + 2 < width) atomicAdd(cp + 2, v.z);
                if (jj + 3 < width) atomicAdd(cp + 3, v.w);
              }
            }
          }
        }
        __syncwarp();
        if (j0 + 32 < NT) load_old(j0 + 32);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(c));
      if (++c == AS) { c = 0; cph ^= 1; }
      u = next;
      first = next;
      next = next2;
      row = row2;
      rscale = rscale2;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && dead_s) g_tile_error = 1;
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// Panels cut over several blocks: their pieces added in block order, scaled and added into C.  One thread per four
// columns of a panel row; block (i, y, ft): cut panel, group of rows, feature tile.
__global__ void __launch_bounds__(256) tile_join_kernel(TileArgs a, int ctas) {
  pdl_trigger();
  pdl_wait();
  const int4 cut = __ldg(a.joins + blockIdx.x);
  const int ft = blockIdx.z, vecs = a.NT / 4;
  const int e = blockIdx.y * 256 + threadIdx.x;
  const int pr = e / vecs, j = (e - pr * vecs) * 4;
  if (pr >= kTileRows) return;
  const int row = __ldg(a.rows + static_cast<int64_t>(cut.x) * kTileRows + pr);
  const float scale = __ldg(a.rs + static_cast<int64_t>(cut.x) * kTileRows + pr);
  const int f0 = ft * a.NT, width = min(a.NT, a.f - f0);
  if (row < 0 || j >= width) return;
  const int64_t slot = static_cast<int64_t>(kTileRows) * a.NT;
  const float* p = a.part + static_cast<int64_t>(ft) * ctas * 2 * slot + static_cast<int64_t>(pr) * a.NT + j;
  float4 sum = *reinterpret_cast<const float4*>(p + (2 * cut.y + 1) * slot);      // the first block's last piece
#pragma unroll 8
  for (int c = cut.y + 1; c < cut.z; ++c) {
    const float4 t = *reinterpret_cast<const float4*>(p + 2 * c * slot);
    sum.x += t.x; sum.y += t.y; sum.z += t.z; sum.w += t.w;
  }
  float* cp = a.C + static_cast<int64_t>(row) * a.ldc + f0 + j;
  if (j + 4 <= width && a.c_vec4) {
    float4 o = *reinterpret_cast<const float4*>(cp);
    o.x += scale * sum.x; o.y += scale * sum.y; o.z += scale * sum.z; o.w += scale * sum.w;
    *reinterpret_cast<float4*>(cp) = o;
  } else {
    const float v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (j + t < width) cp[t] += scale * v[t];
  }
}

struct TileShape {
  int nt, ft;
  bool wide;
};

static TileShape tile_shape(int f) {
  TileShape t;
  t.wide = f > 64;
  t.ft = t.wide ? (f + kMaxNT - 1) / kMaxNT : 1;
  t.nt = ((f + t.ft - 1) / t.ft + 15) / 16 * 16;
  return t;
}

static size_t operand_bytes(const TileShape& t, int nkb) { return static_cast<size_t>(t.ft) * nkb * 3 * t.nt * 128; }

// The kernels need more than the default dynamic shared memory: opt in once per device.
constexpr int kTileSmem = 226 * 1024;
static int tile_opt_in() {
  static bool opted_in[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !opted_in[dev]) {
    if (cudaFuncSetAttribute(tile_core_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem) != cudaSuccess ||
        cudaFuncSetAttribute(tile_core_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem) != cudaSuccess ||
        cudaFuncSetAttribute(tile_operand_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileCols * (kMaxNT + 1) * 4) != cudaSuccess)
      return fail(CAGNET_E_LAUNCH, "cagnet_tile_core_f32: cannot reserve shared memory");
    opted_in[dev] = true;
  }
  return CAGNET_OK;
}

}  // namespace cagnet

using namespace cagnet;

extern "C" int cagnet_tile_count_i32(const int32_t* rowptr, const int32_t* col, int32_t n, const int32_t* rank_r,
                                     const int32_t* rank_c, int32_t lim_r, int32_t lim_c, int32_t* counts, void* stream) {
  if (n < 0 || lim_r < 0 || lim_c < 0) return fail(CAGNET_E_ARG, "cagnet_tile_count_i32: negative size");
  if (n == 0) return CAGNET_OK;
  if (!rowptr || !rank_r || !rank_c || !counts) return fail(CAGNET_E_ARG, "cagnet_tile_count_i32: null pointer");
  const int nkb = (lim_c + kTileCols - 1) / kTileCols;
  tile_count_kernel<<<static_cast<unsigned>((static_cast<int64_t>(n) * 32 + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rowptr, col, n, rank_r, rank_c, lim_r, lim_c, nkb, counts);
  return check_launch("cagnet_tile_count_i32");
}

extern "C" int cagnet_tile_fill_i32(const int32_t* rowptr, const int32_t* col, const float* val, int32_t n, const int32_t* rank_r,
                                    const int32_t* rank_c, int32_t lim_r, int32_t lim_c, const int32_t* tile_of,
                                    const float* row_scale, const float* col_scale, void* bits, uint8_t* keep, void* stream) {
  if (n < 0 || lim_r < 0 || lim_c < 0) return fail(CAGNET_E_ARG, "cagnet_tile_fill_i32: negative size");
  if (n == 0) return CAGNET_OK;
  if (!rowptr || !rank_r || !rank_c || !tile_of || !row_scale || !col_scale || !bits || !keep)
    return fail(CAGNET_E_ARG, "cagnet_tile_fill_i32: null pointer");
  const int nkb = (lim_c + kTileCols - 1) / kTileCols;
  tile_fill_kernel<<<static_cast<unsigned>((static_cast<int64_t>(n) * 32 + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      rowptr, col, val, n, rank_r, rank_c, lim_r, lim_c, nkb, tile_of, row_scale, col_scale, static_cast<unsigned*>(bits), keep);
  return check_launch("cagnet_tile_fill_i32");
}

extern "C" size_t cagnet_tile_core_workspace_bytes(int32_t kbs, int32_t ctas, int32_t f) {
  if (kbs <= 0 || ctas <= 0 || f <= 0) return 0;
  const TileShape t = tile_shape(f);
  return operand_bytes(t, kbs) + static_cast<size_t>(t.ft) * 2 * ctas * kTileRows * t.nt * 4;
}

extern "C" int cagnet_tile_core_f32(const void* bits, const int32_t* tile_kb, const int32_t* panel_ptr, const int32_t* cta_ptr,
                                    int32_t ctas, int32_t panels, const void* join_list, int32_t joins, const int32_t* tile_cols,
                                    int32_t kbs, const int32_t* panel_rows, const float* panel_scale, const float* col_scale,
                                    const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f, void* ws, size_t ws_bytes,
                                    void* stream) {
  if (ctas < 0 || panels < 0 || joins < 0 || kbs < 0 || f < 0) return fail(CAGNET_E_ARG, "cagnet_tile_core_f32: negative size");
  if (ctas == 0 || panels == 0 || kbs == 0 || f == 0) return CAGNET_OK;
  if (!bits || !tile_kb || !panel_ptr || !cta_ptr || (joins > 0 && !join_list) || !tile_cols || !panel_rows || !panel_scale ||
      !col_scale || !B || !C || !ws)
    return fail(CAGNET_E_ARG, "cagnet_tile_core_f32: null pointer");
  if (ldb < f || ldc < f) return fail(CAGNET_E_ALIGN, "cagnet_tile_core_f32: leading dimension smaller than f");
  if (ws_bytes < cagnet_tile_core_workspace_bytes(kbs, ctas, f)) return fail(CAGNET_E_WORKSPACE, "cagnet_tile_core_f32: workspace too small");
  if (!aligned(ws, 128) || !aligned(bits, 16)) return fail(CAGNET_E_ALIGN, "cagnet_tile_core_f32: workspace and bits must be aligned");
  if (int rc = tile_opt_in()) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const TileShape t = tile_shape(f);
  TileArgs a;
  a.bits = static_cast<const unsigned*>(bits);
  a.tile_kb = tile_kb; a.panel_ptr = panel_ptr; a.cta_ptr = cta_ptr;
  a.rows = panel_rows; a.rs = panel_scale;
  a.joins = static_cast<const int4*>(join_list);
  a.operand = static_cast<const char*>(ws);
  a.C = C;
  a.part = reinterpret_cast<float*>(static_cast<char*>(ws) + operand_bytes(t, kbs));
  a.ldc = ldc;
  a.panels = panels; a.nkb = kbs; a.NT = t.nt; a.f = f;
  a.c_vec4 = (ldc % 4 == 0 && aligned(C, 16)) ? 1 : 0;
  const int stage = 3 * t.nt * 128 + kTileBitsBytes;
  a.stages = min(kMaxStages, (kTileSmem - 1024 - kExchangeBytes) / stage);
  const size_t smem = static_cast<size_t>(a.stages) * stage + 1024 + kExchangeBytes;
  const int b_vec4 = (ldb % 4 == 0 && aligned(B, 16)) ? 1 : 0;
  cudaError_t e = launch_pdl(tile_operand_kernel, dim3(kbs, t.ft), dim3(256), kTileCols * (t.nt + 1) * 4, s, B, ldb, tile_cols,
                             col_scale, f, t.nt, b_vec4, static_cast<char*>(ws));
  if (e == cudaSuccess)
    e = launch_pdl(t.wide ? tile_core_kernel<true> : tile_core_kernel<false>, dim3(ctas, t.ft), dim3(kTileThreads), smem, s, a);
  if (e == cudaSuccess && joins > 0)
    e = launch_pdl(tile_join_kernel, dim3(joins, (kTileRows * (t.nt / 4) + 255) / 256, t.ft), dim3(256), 0, s, a, static_cast<int>(ctas));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CAGNET_E_LAUNCH, "cagnet_tile_core_f32: CUDA launch failed: %s", cudaGetErrorString(e));
  }
  return CAGNET_OK;
}

extern "C" int cagnet_tile_core_error(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tile_error, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return v | gemm_tc_error();
}
