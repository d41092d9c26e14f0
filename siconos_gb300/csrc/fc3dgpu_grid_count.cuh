// Barrier of a grid whose blocks are all resident (a cooperative launch): a
// counter of arrivals, zero at the launch, that one thread a block polls.  A wait
// ends after `spin` polls: `dead`, the same in the whole block, then ends the
// solve and *fail tells the host; the block's later barriers pass at once, and
// the other blocks' waits for it run out in turn.  arrived, fail and spin come
// with every call, in the kernel's arguments: kept here they would stand in
// registers.  (A flag a block, polled by a warp of every block, took up to 1.4
// times as long between the colours of a 2D sweep of 70,020 contacts.)
#pragma once
#include <cuda_runtime.h>

namespace fc3dgpu {

struct GridCount {
  unsigned target = 0;
  bool dead = false;
  template <typename A>
  __device__ __forceinline__ void give_up(const A& a) {
    *(volatile double*)a.fail = 1.0;
    dead = true;
  }
  template <typename A>
  __device__ __forceinline__ void sync(const A& a) {
    __syncthreads();
    if (gridDim.x == 1) return;
    target += gridDim.x;
    bool ok = true;
    if (threadIdx.x == 0 && !dead) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.arrived) : "memory");
      for (unsigned long long n = 0;; n++) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(a.arrived) : "memory");
        if ((int)(c - target) >= 0) break;
        if (n > a.spin) {
          ok = false;
          break;
        }
        if (n > 256) __nanosleep(32);
      }
    }
    if (__syncthreads_or(!ok)) give_up(a);
  }
};

}  // namespace fc3dgpu
