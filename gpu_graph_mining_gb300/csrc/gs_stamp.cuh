// Device time stamps for the per-kernel times of the statistics.  An event
// between two kernels of a stream costs about 3 us of it; a stamp is one store.
#pragma once
#include "gs_device.hpp"

namespace gsgb {

__device__ __forceinline__ unsigned long long now_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// word = the kernel's start
__device__ __forceinline__ void stamp_start(unsigned long long *word)
{
  if(word && blockIdx.x == 0 && threadIdx.x == 0) *word = now_ns();
}

// End of a block of a materialise pass (stamps: kMatStampWords words of the
// context; every thread of the block calls it last).
__device__ __forceinline__ void stamp_mat_end(unsigned long long *stamps)
{
  if(!stamps) return;
  __syncthreads();
  if(threadIdx.x == 0) atomicMax(&stamps[16 * (1 + blockIdx.x % kMatSlots)], now_ns());
}

}  // namespace gsgb
