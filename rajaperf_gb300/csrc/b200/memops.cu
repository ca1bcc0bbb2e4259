// MEMCPY (y[i] = x[i]) and MEMSET (x[i] = val) of the Algorithm group.
//
// MEMCPY is Stream COPY's kernel (16-byte vectors, all loads of a tile before
// its stores).  MEMSET stores 16-byte vectors of the value, block x items
// vectors per CTA tile; a pointer that is not 16-byte aligned takes 8-byte
// stores.
#include "b200_launch.cuh"

using namespace b200;

namespace {

constexpr int kBlock = 256;
constexpr int kItems = 4;

// With 16-byte vectors the odd last element is the last CTA's.
template <int BS, int IT, typename V>
__global__ void __launch_bounds__(BS) memset_kernel(double* x, double val, int64_t n) {
  constexpr int kVec = sizeof(V) / sizeof(double);
  const int64_t first = begin() + threadIdx.x;
  V v;
  if constexpr (kVec == 2) v = make_double2(val, val);
  else v = val;
  const int64_t units = n / kVec;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (BS * IT); t0 < units;
       t0 += static_cast<int64_t>(gridDim.x) * (BS * IT)) {
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int64_t j = t0 + u * BS + first;
      if (j < units) reinterpret_cast<V*>(x)[j] = v;
    }
  }
  if (kVec == 2 && (n & 1) && blockIdx.x == gridDim.x - 1 && first == 0) x[n - 1] = val;
}

}  // namespace

extern "C" {

int b200_algorithm_memcpy(const double* x, double* y, int64_t n, const b200_tune* tune,
                          b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!x || !y))) return invalid("b200_algorithm_memcpy: bad args");
  return b200_stream_copy(x, y, n, tune, stream);
}

int b200_algorithm_memset(double* x, double val, int64_t n, const b200_tune* tune,
                          b200_stream_t stream) {
  if (n < 0 || (n > 0 && !x)) return invalid("b200_algorithm_memset: bad args");
  if (n == 0) return B200_OK;
  cudaStream_t st = as_stream(stream);
  const bool vec = aligned16(x) && !(tune && tune->vec == 1) && n >= 2;
  const int64_t units = vec ? n >> 1 : n;
  const Shape s = resolve_1d(tune, units, kBlock, spread(units, kBlock, kItems), vec ? 2 : 1);
  if (!valid_block(s.block)) return invalid("b200_algorithm_memset: bad block size");
  B200_DISPATCH_BLOCK(s.block, BS, B200_DISPATCH_ITEMS(s.items, IT,
    if (vec) launch(memset_kernel<BS, IT, double2>, s.grid, BS, 0, st, x, val, n);
    else launch(memset_kernel<BS, IT, double>, s.grid, BS, 0, st, x, val, n)));
  return after_launch("b200_algorithm_memset");
}

}  // extern "C"
