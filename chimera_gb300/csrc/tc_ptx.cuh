// Inline-PTX helpers of the tcgen05 product kernels: mbarriers, bulk-copy
// TMA, shared-memory and instruction descriptors, MMA issue and commit.
#pragma once
#include <stdint.h>

namespace chm {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait for the phase with parity `parity` to complete
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long limit) {
  const uint32_t a = smem_u32(bar);
  for (long long it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// shared-memory matrix descriptor (SWIZZLE_NONE, K-major core matrices of 8
// rows x 16 bytes: LBO = 128 B between K groups, SBO = 16 K B between row
// groups for a K-wide block); the start address sits in bits 0..13 (address
// >> 4), so adding (offset >> 4) to a descriptor moves it by offset bytes
template <int K>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(128u >> 4) << 16;
  d |= (uint64_t)(((K / 8) * 128u) >> 4) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for tcgen05
  return d;
}

// instruction descriptor: kind::f16, BF16 x BF16 -> F32, K-major A and B
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4)                          // D format F32
         | (1u << 7)                        // A format BF16
         | (1u << 10)                       // B format BF16
         | ((uint32_t)(N >> 3) << 17)       // N / 8
         | ((uint32_t)(M >> 4) << 24);      // M / 16
}

// What an MMA does with the collector buffer that holds its A operand: read A
// and drop it, read and keep it for the next MMA, or take the kept one (and
// keep it on, or drop it).  Consecutive MMAs on one A so read it from shared
// memory once.
enum Collect { kDiscard, kFill, kUse, kLastUse };

// MMA with both operands in shared memory; the descriptors as their low words
// (address, LBO) and a common high word (SBO, version), which halves the
// registers of an unrolled issue loop
template <int C>
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi,
                                          uint32_t idesc, uint32_t accumulate) {
#define CHM_UMMA(COLLECT)                                                         \
  asm volatile(                                                                   \
      "{\n"                                                                       \
      ".reg .pred p;\n"                                                           \
      ".reg .b64 a, b;\n"                                                         \
      "mov.b64 a, {%1, %3};\n"                                                    \
      "mov.b64 b, {%2, %3};\n"                                                    \
      "setp.ne.b32 p, %5, 0;\n"                                                   \
      "tcgen05.mma.cta_group::1.kind::f16.collector::a::" COLLECT " [%0], a, b, %4, p;\n" \
      "}\n" ::"r"(tmem_d),                                                        \
      "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate)                    \
      : "memory")
  if (C == kFill) CHM_UMMA("fill");
  else if (C == kUse) CHM_UMMA("use");
  else if (C == kLastUse) CHM_UMMA("lastuse");
  else CHM_UMMA("discard");
#undef CHM_UMMA
}

// whether the phase with parity `parity` has completed, without waiting (a
// try_wait may suspend the thread for a while)
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace chm
