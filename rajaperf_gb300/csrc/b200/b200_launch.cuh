// Overlapped launches (programmatic dependent launch).
//
// A kernel launched in a stream behind another one normally starts some 2.2 us
// after it has drained (measured on GB300: dependent DAXPYs of 4096, 1M and
// 4M elements take 4.23, 6.23 and 12.4 us each).  launch() asks for the
// grid to be set up as its predecessor's CTAs end, and begin() is the
// device side: it waits until every preceding grid has completed and its writes
// are visible (1.47, 3.57 and 9.4 us each).  In a CUDA graph the edge between
// two such nodes becomes a programmatic one (1.80 -> 1.28 and 3.81 -> 3.32 us a node).
//
// The successor's CTAs are placed as slots fall free.  Letting that begin earlier,
// at this grid's own start, gains nothing and loses where neither grid fills the
// chip: the CTAs go to the SMs that this grid left emptier, or that ended first,
// and wait there, two or three on one SM and none on the next.  A call in a graph
// (us; set up after the predecessor, at its start, as its CTAs end): FDTD_2D, 8
// steps of 500^2, 57.3, 85.6, 53.5; HYDRO_2D 200^2 6.9, 9.9, 6.1; REDUCE_SUM of
// 700001 7.2, 9.8, 6.9; VOL3D 50^3 14.9, 17.8, 14.5; the 1-D kernels at 4096 and
// 200000 elements, 14 calls, 40.6, 34.3, 32.4 and 67.9, 72.7, 62.3.  A persistent
// kernel whose CTAs have an SM to themselves has no such loss, and its successor
// gains from the earlier start (INDEXLIST, 3M items, 17.3, 13.3, 14.3 us):
// begin_early().  (So would, by less than 1 %, grids of many waves, but a test of
// the grid's size in every thread costs more: JACOBI_2D at 1002^2 526 -> 539 us.)
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

// Waits for the preceding grids of the stream; returns 0.
__device__ __forceinline__ unsigned int begin() {
  unsigned int zero;
  asm volatile(
      "griddepcontrol.wait;\n\t"
      "mov.u32 %0, 0;"
      : "=r"(zero)
      :
      : "memory");
  return zero;
}

// The same, and lets the next grid be set up at once.
__device__ __forceinline__ unsigned int begin_early() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  return begin();
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
