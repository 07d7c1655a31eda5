// stamps.cuh -- phase times of an iteration, taken by its kernels.
#pragma once

#include <cstdint>

namespace cmn {

// In nanoseconds (the counter moves in steps of 32 or more).  An event between
// two kernels of the captured iteration cost 8 us: 38 of the 216 us of an
// iteration with a small pool.
__device__ __forceinline__ uint64_t now_ns()
{
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// When the kernel's first block started.
__device__ __forceinline__ void stamp_first(uint64_t* t)
{
  if (t != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *t = now_ns();
}
// When the last block that had work (`worked`) ended; a thread per warp or
// block calls it.
__device__ __forceinline__ void stamp_last(uint64_t* t, bool worked)
{
  if (t != nullptr && (worked || blockIdx.x == 0)) atomicMax((unsigned long long*)t, (unsigned long long)now_ns());
}

}  // namespace cmn
