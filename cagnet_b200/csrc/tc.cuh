// tcgen05 / mbarrier / bulk-copy instructions as the tensor-core kernels of this library use them (one CTA, no cluster).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace cagnet {

constexpr int kWaitLimit = 1 << 22;       // tries of one mbarrier wait before a kernel gives up

// x = a + b + c up to 2^-24 relative: successive bf16 roundings of the remainder (each subtraction is exact).
__device__ __forceinline__ void split3(float x, unsigned short& a, unsigned short& b, unsigned short& c) {
  const __nv_bfloat16 h1 = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(h1);
  const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(h2);
  a = __bfloat16_as_ushort(h1);
  b = __bfloat16_as_ushort(h2);
  c = __bfloat16_as_ushort(__float2bfloat16_rn(r2));
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for a phase, with a limit: a wait that runs out sets the block's `dead` flag, which ends every other wait too.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int* dead) {
  for (int i = 0; i < kWaitLimit; ++i) {
    if (mbar_try(bar, parity)) return true;
    if ((i & 63) == 63 && *dead) return false;
  }
  *dead = 1;
  return false;
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// True in one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}
// One box of a 2-D tensor map into shared memory, its first element at column x, row y.
__device__ __forceinline__ void tma_load_2d(unsigned dst, const void* map, int x, int y, unsigned bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// Two fp32 values as the three packed bf16 pairs of their exact split.
__device__ __forceinline__ void split3_pair(float x, float y, unsigned& a, unsigned& b, unsigned& c) {
  auto pack = [](float lo, float hi) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
  };
  a = pack(x, y);
  x -= __uint_as_float(a << 16);
  y -= __uint_as_float(a & 0xffff0000u);
  b = pack(x, y);
  x -= __uint_as_float(b << 16);
  y -= __uint_as_float(b & 0xffff0000u);
  c = pack(x, y);
}
__device__ __forceinline__ void tc_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem], M = 128, K = 16, bf16 in, fp32 accumulation
__device__ __forceinline__ void tc_mma_ts(unsigned d, unsigned a, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// shared-memory operand descriptor: K-major, 128-byte swizzle, 8-row groups 1,024 bytes apart
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
  return (static_cast<unsigned long long>((addr >> 4) & 0x3fff)) | (1ull << 16) | (static_cast<unsigned long long>(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
#define R8(x, o) "=r"(x[o]), "=r"(x[o + 1]), "=r"(x[o + 2]), "=r"(x[o + 3]), "=r"(x[o + 4]), "=r"(x[o + 5]), "=r"(x[o + 6]), "=r"(x[o + 7])
__device__ __forceinline__ void tmem_ld16(unsigned addr, unsigned (&x)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : R8(x, 0), R8(x, 8)
      : "r"(addr));
}
#undef R8
#define S8(x, o) "r"(x[o]), "r"(x[o + 1]), "r"(x[o + 2]), "r"(x[o + 3]), "r"(x[o + 4]), "r"(x[o + 5]), "r"(x[o + 6]), "r"(x[o + 7])
__device__ __forceinline__ void tmem_st32(unsigned addr, const unsigned (&x)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
      S8(x, 0), S8(x, 8), S8(x, 16), S8(x, 24)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(unsigned addr, const unsigned (&x)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), S8(x, 0) : "memory");
}
#undef S8

}  // namespace cagnet
