// Grid-wide barrier for cooperative (co-resident) launches, with a bounded
// wait: a barrier that does not complete within the time limit records
// ECL_ERR_NO_CONVERGENCE in the status block and every block returns, so a
// wait can never hang the GPU.
//
// Cost is round trips to L2, so there are as few as can be: one add (the
// arrivals only count up, and the value it returns says which multiple of the
// grid ends this barrier) and the polls of that same word; another warp looks
// at the status word meanwhile.  With a generation word, acquire polls behind
// naps and the status read after them, a barrier of 148 blocks took about
// 4 us; this one takes about 2 (Boruvka on a 701 x 1031 grid, 31 barriers:
// 0.34 -> 0.29 ms; the sort of 150 k keys, 9 barriers: 80 -> 69 us).
#pragma once

#include "common.cuh"
#include "ecl_b200.h"

namespace ecl {
namespace dev {

struct GridBarrier {
  unsigned count;  // arrivals (zeroed before the first launch; all launches that share it have one grid size)
  unsigned pad[63];
};

constexpr unsigned long long kBarrierNs = 4000000000ull;

// All threads of the block call (at least two warps).  Returns false when the
// barrier timed out or an error was raised; callers then leave the kernel.
// kTimeoutOnly: only when it timed out, for a launch whose output later
// launches index by and that must be whole whatever an earlier launch has
// found in the graph.
template <bool kTimeoutOnly = false>
__device__ __forceinline__ bool grid_sync(GridBarrier* b, Status* status) {
  __shared__ int s_ok[2];
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    if (gridDim.x > 1) {
      __threadfence();
      const unsigned old = fetch_add(&b->count, 1u);
      const unsigned target = (old / gridDim.x + 1) * gridDim.x;
      unsigned long long t0 = 0;
      for (unsigned spins = 1; (int)(ld(&b->count) - target) < 0; spins++) {
        if ((spins & 255u) == 0) {
          unsigned long long t;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
          if (t0 == 0) t0 = t;
          if (t - t0 > kBarrierNs) {
            raise(status, ECL_ERR_NO_CONVERGENCE, -1);
            ok = 0;
            break;
          }
          if (!kTimeoutOnly && ld(&status->code) != 0) {  // an error anywhere ends the wait
            ok = 0;
            break;
          }
        }
      }
      __threadfence();
    }
    s_ok[0] = ok;
  } else if (threadIdx.x == 32) {
    s_ok[1] = kTimeoutOnly || ld(&status->code) == 0;
  }
  __syncthreads();
  return s_ok[0] && s_ok[1];
}

}  // namespace dev
}  // namespace ecl
