#pragma once
#include <cuda_runtime.h>

namespace nw {

// Final sums of a reduction in the kernel that wrote its partials: the block
// that takes a tile's last ticket sums them (and returns the counter to zero).
// The partials are read past the L1 (__ldcg): other blocks wrote them.
__device__ __forceinline__ bool last_block(int* ticket, int blocks) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // the block's writes, seen through the barrier
    last = atomicAdd(ticket, 1) == blocks - 1;
    if (last) {
      *ticket = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last != 0;
}

}  // namespace nw
