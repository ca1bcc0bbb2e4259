// Element-wise "map" launcher shared by the LCALS, Apps and Basic kernels.
//
// A functor `f` is applied to i in [0, n) in two steps: f.compute(i) loads
// and computes element i into an F::Out, f.store(i, out) writes it.  CTAs own
// tiles of BS*IT consecutive indices; inside a tile the IT items of a thread
// are BS apart, so every warp access is contiguous, and all of a thread's
// items are computed before the first is stored: the stores, which could
// alias the next item's inputs for all the compiler knows, then keep no load
// from being issued early.  No element reads what another element writes.
// A functor with kOneByOne = true stores each item before the next is
// computed: those with many inputs, whose items in flight together would only
// cost registers (DEL_DOT_VEC_2D 96 instead of 80 and 250 instead of 199 us at
// 4M zones, ENERGY 162 instead of 144 us, INT_PREDICT 34.8 instead of 24 us and
// DIFF_PREDICT 34.6 instead of 26 us at 1M).
#pragma once

#include "b200_launch.cuh"

#include <type_traits>

namespace b200 {

template <typename F, typename = void>
struct one_by_one : std::false_type {};
template <typename F>
struct one_by_one<F, std::enable_if_t<F::kOneByOne>> : std::true_type {};

template <int BS, int IT, typename F>
__global__ void __launch_bounds__(BS) map_kernel(F f, int64_t n) {
  const int64_t first = begin() + threadIdx.x;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (BS * IT); t0 < n;
       t0 += static_cast<int64_t>(gridDim.x) * (BS * IT)) {
    if constexpr (one_by_one<F>::value) {
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int64_t i = t0 + u * BS + first;
        if (i < n) f.store(i, f.compute(i));
      }
    } else {
      typename F::Out r[IT];
      if (t0 + BS * IT <= n) {  // a whole tile: no bounds test between the loads
#pragma unroll
        for (int u = 0; u < IT; ++u) r[u] = f.compute(t0 + u * BS + first);
#pragma unroll
        for (int u = 0; u < IT; ++u) f.store(t0 + u * BS + first, r[u]);
      } else {
#pragma unroll
        for (int u = 0; u < IT; ++u) {
          const int64_t i = t0 + u * BS + first;
          if (i < n) r[u] = f.compute(i);
        }
#pragma unroll
        for (int u = 0; u < IT; ++u) {
          const int64_t i = t0 + u * BS + first;
          if (i < n) f.store(i, r[u]);
        }
      }
    }
  }
}

// Launches map_kernel with the tuning's block size and items per thread; a
// short array takes fewer items per thread (spread).
template <typename F>
int launch_map1d(const char* name, const F& f, int64_t n, const b200_tune* tune,
                 cudaStream_t st, int def_block = 256, int def_items = 4) {
  if (n <= 0) return B200_OK;
  Shape s = resolve_1d(tune, n, def_block, spread(n, def_block, def_items), 1);
  if (!valid_block(s.block)) return invalid("%s: bad block size %d", name, s.block);
  B200_DISPATCH_BLOCK(s.block, BS, B200_DISPATCH_ITEMS(s.items, IT,
    launch(map_kernel<BS, IT, F>, s.grid, BS, 0, st, f, n)));
  return after_launch(name);
}

// A coherent load (b200_launch.cuh: not the non-coherent path).
template <typename T>
__device__ __forceinline__ T ld(const T* p) { return *p; }

}  // namespace b200
