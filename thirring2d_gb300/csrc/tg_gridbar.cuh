// tg_gridbar.cuh -- the grid barrier of the persistent solvers (tg_pcg.cu,
// tg_grid_cg.cu).
#pragma once

#include "tg_launch.h"

namespace tg {

// polls of >= 32 ns plus an L2 round trip each: from about half a second to tens
constexpr long long kBarrierSpinLimit = 1LL << 24;

// The number of grid barriers this block has passed in this launch (the arriving
// thread only; every block passes the same sequence of barriers).
__device__ __forceinline__ unsigned& barrier_epoch() {
  __shared__ unsigned epoch;
  return epoch;
}

// Grid barrier on a monotonic arrival count (0 at launch): the k-th barrier is
// passed once the count reaches k * nblocks (the grid's blocks).  Each block
// adds its arrival without waiting for the atomic's result and polls the
// count, so no block has to finish the barrier for the others.  After `limit`
// polls a block gives up.
//
// warp0_grid_wait is the barrier's core, run by one warp (warp 0 in tg_pcg.cu, the
// scalar warp in tg_grid_cg.cu) after a block barrier that follows the block's
// writes; it returns false in every lane if the wait gave up.  prep() runs in lane
// 0 between the arrival and the first poll: the reciprocals that the scalars after
// the sum need (an FP64 division has a latency of 574 clocks) are computed there,
// while the other blocks arrive.  The arrival (lane 0) is a release and each poll
// an acquire at GPU scope: the block's writes, ordered before lane 0 by that block
// barrier, are visible to every block that sees the count complete.  The warp
// barrier hands the acquire on to the other lanes, and the caller's next block
// barrier to the other warps.  Measured 0.35 us faster per barrier than a fence, a
// relaxed atomic and a second fence, with the same 152 blocks.  A one-block grid
// needs no arrival: its block barrier orders its global writes.
struct NoPrep {
  __device__ __forceinline__ void operator()() const {}
};
template <class Prep = NoPrep>
__device__ __forceinline__ bool warp0_grid_wait(const GridBar& b, unsigned nblocks, long long limit, Prep prep = {}) {
  int ok = 1;
  if (nblocks == 1) {
    if ((threadIdx.x & 31) == 0) prep();
  } else if ((threadIdx.x & 31) == 0) {
    const unsigned target = (barrier_epoch() += 1) * nblocks;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.count) : "memory");
    prep();
    long long spins = 0;
    while (true) {
      unsigned c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(b.count) : "memory");
      if ((int)(c - target) >= 0) break;
      if (++spins > limit) {
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

}  // namespace tg
