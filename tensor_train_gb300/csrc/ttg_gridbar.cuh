// Bounded barrier of the co-resident CTAs of a cooperative launch.
#pragma once

#include <cuda_runtime.h>

#include "ttg_job.h"

namespace ttg
{
namespace
{

// Barrier of the `count` CTAs of a team (the whole grid, or a group of it).
// One counter that only grows: a CTA's arrival number says which barrier it
// is at ((old / count + 1) * count arrivals complete it), so a barrier is
// one atomic and a poll of the same word, with no reset and no second word.
// Returns false once this CTA gave up (after `limit` clock cycles of
// waiting) or saw that another one did; a CTA that leaves never arrives
// again, so every other CTA leaves at its next barrier.
__device__ __forceinline__ bool grid_barrier(GridBar* gb, unsigned int count, long long limit)
{
  __shared__ int ok_sh;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    int ok = 1;
    __threadfence();
    const unsigned int old = atomicAdd(&gb->count, 1u);
    const unsigned int target = (old / count + 1u) * count;
    const volatile unsigned int* cp = &gb->count;
    const volatile int* errp = &gb->err;
    const long long t0 = clock64();
    int polls = 0;
    while (static_cast<int>(*cp - target) < 0)
    {
      if ((++polls & 63) == 0)
      {
        if (*errp)
        {
          ok = 0;
          break;
        }
        if (clock64() - t0 > limit)
        {
          atomicExch(&gb->err, 1);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    ok_sh = ok;
  }
  __syncthreads();
  return ok_sh != 0;
}

}  // namespace
}  // namespace ttg
