// Overlapped launches (programmatic dependent launch).
//
// A kernel launched in a stream behind another one normally starts some 2.2 us
// after it has drained (measured on GB300: dependent DAXPYs of 4096, 1M and
// 4M elements take 4.10, 6.15 and 12.3 us each).  launch() asks for the
// grid to be set up while its predecessor still runs, and begin() is the
// device side: it lets the successor be set up in turn, then waits until every
// preceding grid has completed and its writes are visible (1.79, 3.63 and
// 9.93 us each).  In a CUDA graph the edge between two such nodes becomes a
// programmatic one (1.95 -> 1.74 and 3.79 -> 3.58 us a node).
//
// Rules for a kernel that is launched by launch():
//  * every thread calls begin() before its first access to global memory, so
//    no grid can complete before its predecessors have;
//  * a location that an earlier kernel may have written is not read through
//    the non-coherent path (__ldg, or a const __restrict__ kernel parameter
//    that the compiler turns into one): the data must be constant for the
//    lifetime of the grid, which now begins before its predecessor ends.
//    Plain loads do, all of a tile's before its first store, so that they
//    are still in flight together;
//  * indexes or pointers depend on begin()'s result (a zero that the compiler
//    cannot see through), so that no load can be moved ahead of the wait.
#pragma once

#include "b200_internal.cuh"

#include <utility>

namespace b200 {

// Lets the next grid of the stream be set up, waits for the preceding ones;
// returns 0.
__device__ __forceinline__ unsigned int begin() {
  unsigned int zero;
  asm volatile(
      "griddepcontrol.launch_dependents;\n\t"
      "griddepcontrol.wait;\n\t"
      "mov.u32 %0, 0;"
      : "=r"(zero)
      :
      : "memory");
  return zero;
}

// kernel<<<grid, block, smem, st>>>(args...) with the overlap above; launch
// errors are left for after_launch().
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                   A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace b200
