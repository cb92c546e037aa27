// Inline-PTX helpers of the tensor-core (tcgen05) Legendre kernels: bounded
// waits, TMA tile loads, shared-memory and instruction descriptors, MMA
// issue and TMEM reads (internal header).
#pragma once
#include <cuda.h>

#include "mbarrier.cuh"

namespace dccm {
namespace sht {

// Bounded wait: returns false (and records code) if the phase did not
// complete within the limit or another role already gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, int *err, volatile int *abort_flag,
                                          int code, unsigned long long limit_ns) {
  if (mbar_try(b, parity)) return true;
  const unsigned long long t0 = gtimer();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try(b, parity)) return true;
    if ((it & 255) == 0) {
      if (*abort_flag) return false;
      if (gtimer() - t0 > limit_ns) {
        *abort_flag = 1;
        atomicCAS(err, 0, code);
        return false;
      }
    }
  }
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory operand descriptor, 128-byte swizzle, 8-row groups 1024
// bytes apart (stride byte offset).  K-major: the leading byte offset is
// unused.  MN-major: it is the distance between the 64-element (128-byte)
// column blocks along M.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;  // leading byte offset
  d |= (uint64_t)(1024 >> 4) << 32;            // stride byte offset
  d |= (uint64_t)1 << 46;                      // descriptor version (sm_100 family)
  d |= (uint64_t)2 << 61;                      // SWIZZLE_128B
  return d;
}
// kind::f16 instruction descriptor: BF16 x BF16 (bf16 = 1) or FP16 x FP16
// (bf16 = 0; A and B always of one type) -> F32, M = 128, B K-major, A
// K-major (a_mn = 0) or MN-major (a_mn = 1, bit 15).
__device__ __forceinline__ uint32_t idesc_f16kind(int n, int a_mn, int bf16) {
  const uint32_t t = bf16 ? 1u : 0u;
  return (1u << 4) | (t << 7) | (t << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t dtmem, uint64_t da, uint64_t db, uint32_t idesc, int acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(da), "l"(db), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// 16 consecutive TMEM columns of this thread's lane into registers, without
// waiting: several loads are issued, then one tmem_wait_ld before use.
__device__ __forceinline__ void tmem_ld16_nw(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Named barrier of the mixed kernel's epilogue warps (NTHREADS threads from 64 on).
template <int NTHREADS> __device__ __forceinline__ void epi_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
}
// 4 consecutive TMEM columns of this thread's lane, without waiting.
__device__ __forceinline__ void tmem_ld4_nw(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
// 8 consecutive TMEM columns of this thread's lane, without waiting.
__device__ __forceinline__ void tmem_ld8_nw(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_nw(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16_nw(taddr, r); }
__device__ __forceinline__ void tmem_ld_nw(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8_nw(taddr, r); }
__device__ __forceinline__ void tmem_ld_nw(uint32_t taddr, uint32_t (&r)[4]) { tmem_ld4_nw(taddr, r); }

}  // namespace sht
}  // namespace dccm
