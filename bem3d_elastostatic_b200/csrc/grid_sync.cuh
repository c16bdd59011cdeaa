// Release/acquire words and the bounded grid barrier of cooperative launches.
#pragma once

#include "common.cuh"

namespace bem {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add_u32(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier of a cooperative launch (bounded): every thread's earlier writes are
// ordered before the arrival (CTA barrier, then thread 0's release, which is cumulative),
// and the acquire before every thread's later reads by the second CTA barrier; the
// wait gives up after wait_ns or once another CTA recorded an error, and records
// BEM_ERR_TIMEOUT.  Returns false when the launch must stop.
__device__ __forceinline__ bool coop_barrier(unsigned* barrier, unsigned target, int* status,
                                             unsigned long long wait_ns, int* s_abort) {
  __syncthreads();
  if (threadIdx.x == 0) {
    red_release_add_u32(barrier, 1u);
    unsigned long long t0 = 0;
    unsigned spins = 0;
    int abort = 0;
    while (ld_acquire_u32(barrier) < target) {
      if ((++spins & 63u) != 0) continue;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > wait_ns || *((volatile int*)status) != 0) {
        abort = 1;
        break;
      }
    }
    if (abort) atomicCAS(status, 0, BEM_ERR_TIMEOUT);
    *s_abort = abort;
  }
  __syncthreads();
  return *s_abort == 0;
}

}  // namespace bem
