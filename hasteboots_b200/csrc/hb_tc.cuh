// hb_tc.cuh -- tcgen05 (5th-generation tensor core) primitives for exact byte products: u8 x u8
// operands in shared memory, s32 accumulators in tensor memory (TMEM), one CTA.
//
// Operand tiles are K-major without swizzle: 8 rows x 16 bytes form a 128-byte core matrix (rows 16
// bytes apart); consecutive 8-row groups lie 128 bytes apart (SBO), consecutive 16-byte K chunks LBO
// bytes apart. An instruction multiplies M = 128 rows by N rows over K = 32 bytes (two chunks); row r
// of A lands in TMEM lane r, row c of B in column c, 32 bits each.
#pragma once

#include <cstdint>

#include "hb_sync.cuh"

namespace hb {
namespace tc {

// Descriptor of an operand tile at shared address `addr` (16-byte aligned): start address, LBO and SBO
// in 16-byte units, the fixed version field, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 |
         (uint64_t)((sbo >> 4) & 0x3FFF) << 32 | 1ull << 46;
}

// Instruction descriptor of kind::i8: s32 accumulators, unsigned 8-bit A and B, both K-major.
__host__ __device__ constexpr uint32_t idesc_u8(uint32_t m, uint32_t n) {
  return 2u << 4 | (n >> 3) << 17 | (m >> 4) << 24;
}

// One elected thread: D[tmem] (+)= A B^T over K = 32 bytes.
__device__ __forceinline__ void mma_u8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// Arrive on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// True in one lane of the warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r));
  return r != 0;
}

// One warp: allocate / free `cols` TMEM columns (a power of two >= 32); the address goes to *slot.
__device__ __forceinline__ void alloc(uint32_t *slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void dealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

// Ordering of tcgen05 operations against barriers: before the barrier that hands TMEM or operands
// over, after the one that takes them.
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy writes to shared memory become visible to the tensor core (and TMA).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 consecutive 32-bit columns of the thread's TMEM lane (lane offset in the address's upper half);
// results are valid after ld_wait.
__device__ __forceinline__ void ld16(uint32_t (&r)[16], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}
// Waits for the thread's loads; r is tied in so that no use of it moves above the wait.
__device__ __forceinline__ void ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

}  // namespace tc
}  // namespace hb
