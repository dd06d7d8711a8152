// Inboxes of the respond clusters: mbarriers in shared memory that count the bytes of words arriving from other CTAs.
#pragma once
#include "ig_arith.cuh"

namespace igk {
using namespace ig;

__device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void inbox_init(u32 bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// One thread opens a phase of `bytes`; every thread waits for its end.
__device__ __forceinline__ void inbox_expect(u32 bar, u32 bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity; false when the tries ran out. A try suspends the thread for 4 us at most (as
// measured, whatever hint it is given), so a wait gives up after a second.
constexpr int INBOX_TRIES = 1 << 18;
__device__ __forceinline__ bool inbox_wait(u32 bar, u32 parity) {
  for (int k = 0; k < INBOX_TRIES; k++) {
    u32 done;
    asm volatile("{.reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace igk
