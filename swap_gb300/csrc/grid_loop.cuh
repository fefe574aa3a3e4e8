// grid_loop.cuh -- a loop of phases in one launch: the barrier its blocks meet
// at, and the launch of such a kernel.
#pragma once

#include <cuda_runtime.h>

namespace loop {

// At least this many polls of a barrier (about a second): a block may wait for
// the rest of its grid to find room beside another stream's kernels, however
// short the caller wants the waits for its own copies.
constexpr unsigned MIN_POLLS = 1u << 20;

// The barrier between two phases.  Every wait is bounded: when one runs out,
// sync() is false in the whole block, which then returns.
struct Barrier {
  unsigned* bar;  // [0] arrivals, [1] blocks that are through
  unsigned polls;
  unsigned target;
  bool ok;
  // Every block's stores before it are visible to every block after it;
  // false: the wait ran out (the caller returns).
  template <bool CLUSTER>
  __device__ __forceinline__ bool sync() {
    if (CLUSTER) {
      asm volatile(
          "barrier.cluster.arrive.release.aligned;\n"
          "barrier.cluster.wait.acquire.aligned;" ::
              : "memory");
      return true;
    }
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(bar, 1u);
      unsigned v, n = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      } while (v < target && n++ < polls);
      __threadfence();
      ok = v >= target;
    }
    return !__syncthreads_or(threadIdx.x == 0 && !ok);
  }
  // The last block to finish leaves the counters at zero for the next launch.
  __device__ __forceinline__ void done() {
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
        bar[0] = 0u;
        bar[1] = 0u;
        __threadfence();
      }
    }
  }
};

// Launches kernel cooperatively with min(blocks, SMs) blocks on st, one per
// SM.  Loops of several contexts on one GPU run one after the other: two
// grids whose blocks wait for their own kind must not hold half of the SMs
// each.
cudaError_t launch(const void* kernel, long long blocks, int threads, void** args, cudaStream_t st);

}  // namespace loop
