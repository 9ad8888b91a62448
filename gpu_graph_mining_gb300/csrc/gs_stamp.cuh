// Device helpers of several kernels: time stamps for the per-kernel times of the
// statistics (an event between two kernels of a stream costs about 3 us of it, a
// stamp is one store), the wait of early launches, a bitmap word in use.
#pragma once
#include "gs_device.hpp"

namespace gsgb {

__device__ __forceinline__ unsigned long long now_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// First statement of a kernel that may be launched before the one ahead of it
// has finished (KernelCall::early): what that one wrote is there from here on.
// It must not be read through const __restrict__ pointers or __ldg, whose loads
// may move ahead of the wait; what kernels before that one wrote may.  The
// launch overlaps the last blocks of the kernel ahead: a mine of 42 waves of
// one node 1.42 -> 1.34 ms, 100,000 graphs at 1% 2.31 -> 2.24.  An explicit
// trigger (griddepcontrol.launch_dependents) at the start of each kernel gave 1%
// more in small waves and took 4% in large ones: blocks that only wait keep
// the room that other contexts' kernels would use.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

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

// A bitmap word while other warps set bits of it.
__device__ __forceinline__ uint32_t word_now(const uint32_t *p)
{
  uint32_t x;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p));
  return x;
}

}  // namespace gsgb
