// tc05.cuh -- the fifth-generation tensor core operations that the exact
// split products use, as inline PTX: mbarriers, bulk and 16-byte asynchronous
// copies, tensor-memory allocation, tcgen05.mma (kind::f16, FP16 operands in
// shared memory, FP32 sums in tensor memory) and tcgen05.ld.
//
// Operands are small integers stored as FP16 (exact up to 2048) and the sums
// stay below 2^24, so every product and sum is an exact integer: measured,
// the FP32 accumulators of M = 128, N = 16..256 products return the integer
// sums unchanged up to 2^24.
//
// Both operands are K-major without swizzle: element (row r, k) of an
// operand of R rows sits at (k / 8) * 16 R + (r / 8) * 128 + (r % 8) * 16 +
// (k % 8) * 2 bytes, i.e. 16-byte pieces of eight k, row after row.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace vpmg {
namespace tc05 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits with a limit; once a wait has run out, `dead` stays set and every later
// wait of the thread returns at once.  The caller spreads `dead` over its CTA,
// waits for what is in flight and reports.
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, bool& dead, int polls) {
  if (dead) return;
  for (int i = 0; i < polls; ++i)
    if (bar_try(bar, parity)) return;
  dead = true;
}
constexpr int kPolls = 1 << 20;  // about a second

// 16 bytes, zero-filled when !ok (src is not read then)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// contiguous bulk copy (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// generic-proxy writes to shared memory become visible to the tensor core
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// one whole warp
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}

// shared-memory descriptor: address, bytes between 16-byte columns (lbo) and
// between groups of eight rows (128)
__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 | (uint64_t)(128 >> 4) << 32 |
         1ull << 46;
}
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {  // D FP32, A and B FP16, both K-major
  return (1u << 4) | (uint32_t)(n >> 3) << 17 | (uint32_t)(m >> 4) << 24;
}
// D[tmem] = A B^T (+ D), K = 16; one thread
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// bar gets an arrival when the MMAs issued so far by this thread are done
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// eight consecutive columns of this warp's 32 lanes (not complete before ld_wait)
__device__ __forceinline__ void ld8(uint32_t addr, uint32_t v[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}
__device__ __forceinline__ void ld4(uint32_t addr, uint32_t v[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The integer round(v 2^55 / 2^(emax - 1022)) for |v| < 2^(emax - 1022), emax
// the biased exponent of the scale; |result| <= 2^55.
__device__ __forceinline__ long long fixed55(double v, int emax) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7FF);
  const unsigned long long m = ((b & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull)) << 2;
  const int sh = emax - (e ? e : 1);
  unsigned long long u = 0;
  if (sh <= 0) u = m << min(-sh, 1);  // an average of a list may round to one step above its maximum
  else if (sh < 57) u = (m + (1ull << (sh - 1))) >> sh;
  return (long long)b < 0 ? -(long long)u : (long long)u;
}
// Biased exponent that scales a list whose largest magnitude has this high word.
__device__ __forceinline__ int scale_exp(unsigned hi) { return max((int)(hi >> 20), 1); }

// The seven balanced base-256 digits of two integers |x| <= 2^56 each,
// x = sum_j d_j 256^(6-j), |d_j| <= 128 but for the top one (<= 256), as FP16
// pairs (the first integer's digit in the low half).  A biased digit u < 1024
// or-ed into the FP16 1024 is 1024 + u; 1024 + bias is taken off exactly.
__device__ __forceinline__ unsigned hadd2(unsigned a, unsigned b) {
  unsigned r;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void digits256x2(long long x0, long long x1, unsigned d[7]) {
  const unsigned long long y0 = (unsigned long long)(x0 + 0x0200808080808080ll);  // + 512 on top, 128 below
  const unsigned long long y1 = (unsigned long long)(x1 + 0x0200808080808080ll);
  const unsigned l0 = (unsigned)y0, h0 = (unsigned)(y0 >> 32), l1 = (unsigned)y1, h1 = (unsigned)(y1 >> 32);
  d[0] = hadd2(__byte_perm(h0, h1, 0x7632) | 0x64006400u, 0xE600E600u);                    // bits 48.., - 1536
  d[1] = hadd2((__byte_perm(h0, h1, 0x0501) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);    // - 1152
  d[2] = hadd2((__byte_perm(h0, h1, 0x0400) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);
  d[3] = hadd2((__byte_perm(l0, l1, 0x0703) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);
  d[4] = hadd2((__byte_perm(l0, l1, 0x0602) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);
  d[5] = hadd2((__byte_perm(l0, l1, 0x0501) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);
  d[6] = hadd2((__byte_perm(l0, l1, 0x0400) & 0x00FF00FFu) | 0x64006400u, 0xE480E480u);
}
// one integer's digits
__device__ __forceinline__ void digits256(long long x, unsigned short d[7]) {
  unsigned p[7];
  digits256x2(x, 0, p);
#pragma unroll
  for (int j = 0; j < 7; ++j) d[j] = (unsigned short)p[j];
}

}  // namespace tc05
}  // namespace vpmg
