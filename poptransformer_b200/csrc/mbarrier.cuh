// Shared-memory barriers and bulk copies that arrive on them.  Every wait is bounded.
#pragma once
#include "common.cuh"

namespace pt {

constexpr int WAIT_LIMIT = 1 << 22;
#ifndef PT_TC_HINT
#define PT_TC_HINT 1000   // suspend-time hint (ns) of the barrier waits; negative: plain polling with test_wait
#endif

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// One look.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// One look that may last as long as the suspend-time hint.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
#if PT_TC_HINT < 0
  return mbar_test(bar, parity);
#else
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity), "r"((uint32_t)PT_TC_HINT)
               : "memory");
  return ok != 0;
#endif
}
// Bounded wait; gives up at once when the CTA has already recorded a failure.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  for (int it = 0; it < WAIT_LIMIT; ++it) {
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  return false;
}
// The same without a way to give up early: for what is still in flight when a block ends after a failure.
__device__ __forceinline__ void mbar_wait_all(uint32_t bar, uint32_t parity) {
  volatile int never = 0;
  mbar_wait(bar, parity, &never);
}
// The last copies that were sent to a ring of S slots, `issued` in all, have landed: the block that asked for them may end.  (Bounded as a whole.)
inline __device__ __noinline__ void mbar_wait_ring(uint32_t full0, int issued, int S) {
  int looks = 0;
  for (int i = max(0, issued - S); i < issued; ++i)
    while (!mbar_try(full0 + i % S * 8, (i / S) & 1))
      if (++looks >= WAIT_LIMIT) return;
}
// The blocks of a cluster send one another sums.  A block whose waits have not run out ends when all that is sent to it has come.  One that has given up
// stays until nobody can send any more: this returns when every thread of the cluster has come here or has ended, which each does in bounded time.
__device__ __forceinline__ void stay_for_cluster() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

}  // namespace pt
