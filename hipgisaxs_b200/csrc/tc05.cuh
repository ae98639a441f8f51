// Inline-PTX helpers for the fifth-generation tensor cores (tcgen05) of sm_100a: TMEM
// allocation, register <-> TMEM moves, and s8 x s8 -> s32 matrix products with A in TMEM and B
// in shared memory.  One CTA (cta_group::1) throughout.
#pragma once
#include <stdint.h>

#include "ptx.cuh"

namespace hgx {

// Allocates `cols` TMEM columns (a power of two >= 32) and writes the base address to *dst
// (shared memory); one whole warp calls it and, later, tmem_free.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Consecutive columns of this warp's 32 lanes (addr: lane in bits 31-16, column in 15-0): thread
// i holds lane i's row.
__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
// The values are valid after tmem_wait_ld.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr)
               : "memory");
}
// Waits for the loads into r[0..N): the registers pass through the statement so that no use of
// them moves above it.
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}

// Instruction descriptor of kind::i8: s32 accumulators, A and B signed 8-bit, both K-major,
// M = 128 rows, N columns.
__host__ __device__ constexpr uint32_t idesc_s8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

// Shared-memory descriptor of a K-major operand without swizzle: 8 x 16-byte core matrices of
// 128 contiguous bytes; lbo: bytes between core matrices along K, sbo: along N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         (1ull << 46);
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t v;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(v));
  return v != 0;
}

// D[128 x N] (+)= A[128 x 32] B[32 x N], one thread; acc = 0 overwrites D.
__device__ __forceinline__ void mma_s8_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// Arrives on the mbarrier when this thread's earlier MMAs are done.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

}  // namespace hgx
