// Device check of a respond cluster's bounded wait (compiled and run by test_gpu_inbox_wait.py): a phase that is
// complete is seen by every thread; one that nothing completes is given up by every thread, after a second or so.
#include <cstdio>

#include "ig_inbox.cuh"

using namespace igk;

__global__ void k_wait(u32 bytes, u32* gave_up, u64* ns) {
  __shared__ __align__(8) u64 inbox;
  const u32 bar = smem_addr(&inbox);
  if (threadIdx.x == 0) {
    inbox_init(bar);
    inbox_expect(bar, bytes);  // no byte ever arrives
  }
  __syncthreads();
  u64 t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  if (!inbox_wait(bar, 0)) atomicAdd(gave_up, 1u);
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
  if (threadIdx.x == 0) *ns = t1 - t0;
}

int main() {
  u32* gave_up;
  u64* ns;
  if (cudaMallocManaged(&gave_up, 4) || cudaMallocManaged(&ns, 8)) return 2;
  for (u32 bytes : {0u, 8u}) {
    *gave_up = 0;
    k_wait<<<1, 256>>>(bytes, gave_up, ns);
    if (cudaDeviceSynchronize()) return 2;
    const double s = 1e-9 * (double)*ns;
    std::printf("%u bytes awaited: %u of 256 threads gave up, %.3f s\n", bytes, *gave_up, s);
    if (*gave_up != (bytes ? 256u : 0u) || s > 3.0) return 1;
  }
  std::printf("ok\n");
  return 0;
}
