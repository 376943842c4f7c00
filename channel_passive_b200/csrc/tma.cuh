// tma.cuh - mbarrier and bulk-copy helpers (sm_100a), shared by the kernels that stage through
// cp.async.bulk.  Every wait has an iteration limit; a wait that gives up returns false and its
// caller sets the error flag and leaves.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace kmm {

constexpr int kTmaWaitIters = 1 << 20;

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
// bounded wait for the phase of `bar` with this parity; false if it gave up
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity = 0) {
  for (int it = 0; it < kTmaWaitIters; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// untiled copy of `bytes` (a multiple of 16; both addresses 16-byte aligned) completing on `bar`
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

}  // namespace kmm
