// PTX helpers of the tensor-core GEMM kernels (oz.cu, crt.cu, nl_tc.cu): shared-memory operand descriptors,
// kind::i8 products, bounded mbarrier waits, bulk copies and tensor-memory reads.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cpwb {
namespace mma8 {

constexpr unsigned long long kWaitNs = 2000000000ull;   // 2 s per mbarrier wait at most

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major operand tile, 128-byte swizzle: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);               // start address
  d |= (uint64_t)1 << 16;                               // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((1024 >> 4) & 0x3FFF) << 32;          // stride byte offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;                               // descriptor version
  d |= (uint64_t)2 << 61;                               // 128-byte swizzle
  return d;
}

// kind::i8 instruction descriptor: D S32, A and B signed 8-bit, both K-major
__device__ __forceinline__ uint32_t instr_desc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t mbar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(mbar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// wait bounded in time (limit_ns); gives up early once another role has recorded a failure.
// The hand-offs between the roles use the caller's limit (GemmArgs::wait_ns, 2 s unless a
// failure-detection test shortens it); the waits for copies and MMAs already issued, before the
// CTA exits, always use kWaitNs: those complete on their own.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, const volatile int* failed,
                                          unsigned long long limit_ns = kWaitNs) {
  // a phase that is already complete costs no read of the timer (about a microsecond)
  if (mbar_try(mbar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (unsigned it = 0;; ++it) {
    if (mbar_try(mbar, parity)) return true;
    if ((it & 63) == 63) {
      if (failed && *failed) return false;
      if (globaltimer_ns() - t0 > limit_ns) return false;
    }
  }
}

// The same for all lanes of a converged warp, with one answer: a lane that gave up alone would leave the others
// to run the warp-wide tensor-memory loads without it.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t mbar, uint32_t parity, const volatile int* failed,
                                               unsigned long long limit_ns) {
  return __all_sync(0xffffffffu, mbar_wait(mbar, parity, failed, limit_ns));
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar), "r"(bytes) : "memory");
}
// contiguous global -> shared bulk copy (16-byte aligned, size a multiple of 16), no multicast
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

}  // namespace mma8
}  // namespace cpwb
