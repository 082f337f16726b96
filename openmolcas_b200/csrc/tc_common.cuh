// Helpers for the hand-written tcgen05 (5th-generation tensor core) kernels:
// mbarriers with bounded waits, TMA tile loads, shared-memory matrix
// descriptors and MMA issue.  Only single-CTA forms are used (no clusters,
// no multicast).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mg {

// Iterations of a bounded mbarrier wait (a few hundred ms on a B200); a wait
// that runs out makes the kernel give up and report an error.
constexpr long long kTcWaitLimit = 1ll << 24;

__device__ __forceinline__ uint32_t tc_smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tc_mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void tc_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tc_mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool tc_mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase with the given parity; false when it ran out or
// another role of the CTA already gave up (then *abort is set).
__device__ __forceinline__ bool tc_mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
  for (long long i = 0; i < kTcWaitLimit; ++i) {
    if (tc_mbar_test(bar, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  return false;
}

// 5D tiled TMA load into shared memory, completion on an mbarrier.
__device__ __forceinline__ void tc_tma_load5(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                             int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], "
      "[%2];" ::"r"(dst),
      "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

// Shared-memory matrix descriptor (Blackwell version 1), K-major operand,
// 32-byte swizzle: rows of 32 bytes (one K = 32 step of 8-bit operands), 8-row
// atoms of 256 bytes stacked along M/N.
__device__ __forceinline__ uint64_t tc_desc_sw32(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;           // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(256 >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;           // descriptor version
  d |= (uint64_t)6 << 61;  // SWIZZLE_32B
  return d;
}

// Instruction descriptor, M = 128, both operands K-major: 8-bit integers -> S32
// (kind::i8); a_signed / b_signed select S8 (else U8)
__host__ __device__ constexpr uint32_t tc_idesc_i8(int n, bool a_signed, bool b_signed) {
  return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | ((b_signed ? 1u : 0u) << 10) | ((uint32_t)(n >> 3) << 17) |
         ((128u >> 4) << 24);
}

// One lane of a converged warp (1 there, 0 in the others).
__device__ __forceinline__ uint32_t tc_elect() {
  uint32_t el;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(el));
  return el;
}

// Issued by the lanes with el != 0 (one of a converged warp).
__device__ __forceinline__ void tc_mma_i8(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc,
                                          uint32_t el) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %9, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(el));
}

// Arrive on an mbarrier once every tcgen05 operation issued so far by this
// thread has completed (the lanes with el != 0).
__device__ __forceinline__ void tc_commit_if(uint32_t bar, uint32_t el) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
      "r"(el)
      : "memory");
}

// 16 consecutive 32-bit TMEM columns of this thread's lane (warp w reads lanes
// 32 (w % 4) .. +31), without waiting:
// several loads may be in flight; tc_ld_wait() completes them and
// tc_ld_bind() orders every later use of the registers after it.
__device__ __forceinline__ void tc_ld16_async(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld_bind(uint32_t (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(v[i]));
}

}  // namespace mg
