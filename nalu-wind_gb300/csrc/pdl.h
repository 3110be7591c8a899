#pragma once
#include <cuda_runtime.h>

#include "nw_internal.h"

namespace nw {

// Programmatic dependent launch. A kernel launched by pdl_launch may start
// while the kernel before it on the stream (or in the captured graph) still
// runs: its blocks are placed, its index arithmetic done and its pattern
// arrays (fixed since set-up) loaded under the other's end. pdl_wait then waits
// until everything the earlier kernels wrote is visible, and lets the next
// kernel start in the same way; nothing that an earlier kernel may write or
// read is touched before it (values too: the kernel that refreshes them may be
// the one before).
//
// It pays for chains of short kernels bound by latency: the learned cycle (9.09
// -> 8.53 ms for 90 iterations), its network layers' product included, and the
// level-scheduled sweeps (22.4 -> 18.6 ms for 43x64x43 nodes, their levels then
// still in blocks of 256). The multi-dots, multi-axpys and scalings lost by it
// (32^3 GMRES 1.38 -> 1.57 ms, 1.08 M rows 17.4 -> 18.8 ms), the node sweeps too
// (1.55 -> 1.58 ms), and the sparse product with the system's matrix gained
// nothing: they are launched plainly.
//
// pdl_wait takes the pointers to such memory and hands them back through an
// opaque statement behind the wait: a load through a const __restrict__
// parameter is otherwise free to move above it.
template <typename T>
__device__ __forceinline__ void pdl_behind(T& p) {
  size_t g = p ? __cvta_generic_to_global(p) : 0;  // stays known as global memory
  asm volatile("" : "+l"(g)::"memory");
  p = static_cast<T>(g ? __cvta_global_to_generic(g) : nullptr);
}
template <typename... T>
__device__ __forceinline__ void pdl_wait(T&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  (pdl_behind(p), ...);
}

template <typename... P, typename... A>
void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  NW_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

}  // namespace nw
