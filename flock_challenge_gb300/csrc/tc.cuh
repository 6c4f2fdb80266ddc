// Tensor-core helpers (tcgen05, sm_103a) for bit matrices over GF(2).
//
// A product of bit matrices is a matrix product of 0/1 integers followed by the
// parity of each count. The operands are fp4 (e2m1) values in shared memory, 64
// bits of the summed index per MMA; the counts are f32 in TMEM, exact up to
// 2^24, so a parity is taken once per accumulation, however long. Nibbles of a
// 32-bit word keep their places: masking every fourth bit of a word of 32 bits
// gives eight e2m1 values at once, and the code point of the bit's place in the
// nibble (0001: 0.5, 0010: 1, 0100: 2) is a power of two that the other operand
// or the parity extraction undoes.
//
// Operand layout (K-major, no swizzle): core matrices of 8 rows x 16 bytes (32
// summed bits), 128 bytes each; consecutive groups of eight rows SBO bytes
// apart, the two halves of an MMA's 64 summed bits LBO bytes apart.
#pragma once
#include <cstdint>

#include "wait_clock.h"

namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// Waits for the completion of phase `parity`; false when it gave up after
// `limit` clocks of waiting (wait_clock.h). Kernels whose limit is zero start as
// if a wait had given up.
//
// A kernel whose wait gave up still owns what it started: before its block
// leaves or its TMEM is freed, the bulk copies it issued have landed and its MMAs
// are done, or they would write shared memory or TMEM that the next block already
// has. Every kernel therefore waits for them with kDrainClocks, whatever its own limit:
// copies and MMAs end by themselves, they need nothing more of the block. (Past that
// limit too, the block leaves all the same, and what its copies and MMAs then
// write is undefined; a second without an end is a broken device.)
constexpr uint32_t kDrainClocks = 1u << 31;
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, uint32_t limit) {
  const uint32_t a = smem_addr(b);
  WaitClock wc;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if (wc.passed((uint32_t)clock(), limit)) return false;
  }
}
// Contiguous copy into shared memory by the copy engine (16-byte aligned both
// sides, a multiple of 16 bytes); its bytes complete b's expected count.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(b))
               : "memory");
}
// Orders this thread's shared-memory stores before later MMA reads.
__device__ __forceinline__ void fence_smem_for_mma() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// TMEM columns (a power of two, at least 32): one warp, all lanes.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// The calling warp's 32 lanes of 32 columns from addr on set to v.
__device__ __forceinline__ void tmem_fill32(uint32_t addr, uint32_t v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(addr),
      "r"(v)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 32 columns of the calling warp's lanes.
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// K-major operand without swizzle at shared address a.
__device__ __forceinline__ uint64_t operand(uint32_t a, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
// Instruction descriptor of kind::mxf4: e2m1 operands, ue8m0 scales, M x N, K = 64.
__host__ __device__ constexpr uint32_t mxf4_desc(int m, int n) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(m >> 4) << 24);
}
// D (+)= A B^T over 64 summed bits; all scales at sf are one (0x7f bytes).
__device__ __forceinline__ void mma_mxf4(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t sfa, uint32_t sfb,
                                         bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(desc), "r"(sfa), "r"(sfb), "r"((uint32_t)accumulate)
      : "memory");
}
// Arrives on b when the MMAs this thread issued so far are done.
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b))
               : "memory");
}

}  // namespace tc
