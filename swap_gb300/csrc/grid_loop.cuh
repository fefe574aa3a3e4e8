// grid_loop.cuh -- a loop of phases in one launch: the barrier its blocks meet
// at, and the launch of such a kernel.
#pragma once

#include <cuda_runtime.h>

namespace loop {

// At least this many polls of a barrier (about a second): a block may wait for
// the rest of its grid to find room beside another stream's kernels, however
// short the caller wants the waits for its own copies.
constexpr unsigned MIN_POLLS = 1u << 20;

// The barrier between two phases, 0.9 us at 152 blocks: one releasing add and
// an acquiring poll (1.2 us with a full fence on either side; 20 FP32 steps of
// 64x32x32 cells 5.64 -> 5.42 ms, 10 FP64 steps of 16^3 cells 4.21 -> 3.88).
// Every wait is bounded: when one runs out,
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
      // release: the block's stores (before the block's barrier) are visible
      // to whoever acquires the count
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      unsigned v, n = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      } while (v < target && n++ < polls);
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
