// Shared-memory barriers and bulk copies (PTX mbarrier, cp.async.bulk), with bounded waits.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sb {

constexpr long long kSpinCycles = 4000000000LL;  // about 2 s at the B200's clocks

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(b)) : "memory");
}
// One arrival for the calling warp, after all its lanes got here.
__device__ __forceinline__ void warp_arrive(unsigned long long* b) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(b);
}
__device__ __forceinline__ bool mbar_done(unsigned long long* b, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return done != 0;
}
// A bounded wait on phase `parity`: false if it gave up (then *err and sm.abort are set) or if
// another warp gave up first.
template <class Smem>
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, uint32_t parity, Smem& sm,
                                          unsigned* err) {
  if (mbar_done(b, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_done(b, parity)) {
    if (*(volatile int*)&sm.abort) return false;
    if (clock64() - t0 > kSpinCycles) {
      atomicExch(err, 1u);
      *(volatile int*)&sm.abort = 1;
      return false;
    }
  }
  return true;
}
// A bounded wait that ignores the abort flag: the drains of copies and MMAs in flight.
__device__ __forceinline__ void mbar_wait_drain(unsigned long long* b, uint32_t parity,
                                                unsigned* err) {
  const long long t0 = clock64();
  while (!mbar_done(b, parity))
    if (clock64() - t0 > kSpinCycles) {
      atomicExch(err, 1u);
      return;
    }
}
// Bulk copy of `bytes` (a multiple of 16) from global to shared memory, completing on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

}  // namespace sb
