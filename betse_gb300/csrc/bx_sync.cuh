// bx_sync.cuh -- the bounded grid barrier of the cooperative step kernels.
#pragma once
#include <cuda_runtime.h>

namespace bx {

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Arrival at the grid barrier: release, so this thread's writes (and those
// it observed, e.g. through the preceding bar.sync) are visible first.
__device__ __forceinline__ void res_arrive(unsigned* ctl) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctl) : "memory");
}

// Thread 0 waits until ctl[0] reaches `target` (acquire), or until another
// CTA raised ctl[1], or until timeout_ns passed (then it raises ctl[1]
// itself); the result is broadcast through *sflag after a bar.sync.
__device__ __forceinline__ bool res_wait(unsigned* ctl, unsigned target, long long timeout_ns, int* sflag) {
  if (threadIdx.x == 0) {
    const unsigned long long t0 = global_ns();
    int ok = 1;
    unsigned n = 0;
    while (true) {
      unsigned v, f;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctl) : "memory");
      if ((int)(v - target) >= 0) break;
      if ((++n & 31u) == 0) {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(ctl + 1) : "memory");
        if (f) { ok = 0; break; }
        if ((long long)(global_ns() - t0) > timeout_ns) {
          atomicExch(ctl + 1, 1u);
          ok = 0;
          break;
        }
      }
    }
    *sflag = ok;
  }
  __syncthreads();
  return *sflag != 0;
}

}  // namespace bx
