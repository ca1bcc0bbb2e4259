// Stream group: COPY, MUL, ADD, TRIAD, DOT.
//
// Streaming layout: each CTA owns tiles of block*items 16-byte vectors
// (double2) and every thread issues all of its loads for a tile before any
// store, so a CTA keeps block*items*16 bytes per operand in flight.  The grid
// is one tile per CTA (the hardware scheduler balances the tail); arrays that
// are not 16-byte aligned take the scalar path with the same shape.
#include "b200_internal.cuh"
#include "b200_launch.cuh"
#include "b200_reduce.cuh"

using namespace b200;

namespace {

constexpr int kBlock = 256;
constexpr int kItems = 4;

// Grid-stride tile loop shared by the map kernels.  `VEC` doubles per access.
#define TILE_LOOP(BS, IT, UNITS)                                              \
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (BS * IT);            \
       t0 < (UNITS);                                                          \
       t0 += static_cast<int64_t>(gridDim.x) * (BS * IT))

// One element-wise body per kernel: out[i] = f(in1[i], in2[i]) (COPY and MUL
// read one array).
struct CopyOp {
  static constexpr int kInputs = 1;
  __device__ double operator()(double a, double) const { return a; }
};
struct MulOp {
  static constexpr int kInputs = 1;
  double alpha;
  __device__ double operator()(double c, double) const { return alpha * c; }
};
struct AddOp {
  static constexpr int kInputs = 2;
  __device__ double operator()(double a, double b) const { return a + b; }
};
struct TriadOp {
  static constexpr int kInputs = 2;
  double alpha;
  __device__ double operator()(double b, double c) const { return b + alpha * c; }
};

template <typename Op>
__device__ __forceinline__ double apply(const Op& f, double x, double y) { return f(x, y); }
template <typename Op>
__device__ __forceinline__ double2 apply(const Op& f, double2 x, double2 y) {
  return make_double2(f(x.x, y.x), f(x.y, y.y));
}

// All loads of a tile are issued before its stores.  With 16-byte vectors an
// odd n leaves one element, done by the first thread of the last CTA: a
// second launch for it cost 2 us behind every call (n = 4099: 20 launches a
// rep of the Stream, Basic and LCALS kernels instead of 16).
template <int BS, int IT, typename V, typename Op>
__global__ void __launch_bounds__(BS)
stream_kernel(const double* in1, const double* in2, double* out, Op f, int64_t n) {
  constexpr int kVec = sizeof(V) / sizeof(double);
  const int64_t first = begin() + threadIdx.x;
  const V* a = reinterpret_cast<const V*>(in1);
  const V* b = reinterpret_cast<const V*>(in2);
  V* c = reinterpret_cast<V*>(out);
  const int64_t units = n / kVec;
  TILE_LOOP(BS, IT, units) {
    V ra[IT], rb[IT];
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int64_t j = t0 + u * BS + first;
      if (j < units) {
        ra[u] = a[j];
        if (Op::kInputs == 2) rb[u] = b[j];
      }
    }
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int64_t j = t0 + u * BS + first;
      if (j < units) c[j] = apply(f, ra[u], Op::kInputs == 2 ? rb[u] : ra[u]);
    }
  }
  if (kVec == 2 && (n & 1) && blockIdx.x == gridDim.x - 1 && first == 0) {
    const double x = in1[n - 1];
    out[n - 1] = f(x, Op::kInputs == 2 ? in2[n - 1] : x);
  }
}

// ---- DOT -------------------------------------------------------------------
// Thread partial sums run over the thread's elements in increasing index
// order; the last CTA combines the per-CTA partials in CTA order.
template <int BS, int IT>
__global__ void __launch_bounds__(BS)
dot_kernel(const double* a, const double* b, int64_t n, bool vec2, double dot_init,
           double* accum, double* partials, unsigned int* counter) {
  __shared__ double smem[BS / 32];
  __shared__ bool last_flag;
  const int64_t first = begin() + threadIdx.x;
  double s = 0.0;
  if (vec2) {
    const double2* a2 = reinterpret_cast<const double2*>(a);
    const double2* b2 = reinterpret_cast<const double2*>(b);
    const int64_t units = n >> 1;
    TILE_LOOP(BS, IT, units) {
      double2 ra[IT], rb[IT];
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        int64_t j = t0 + u * BS + first;
        if (j < units) { ra[u] = a2[j]; rb[u] = b2[j]; }
      }
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        int64_t j = t0 + u * BS + first;
        if (j < units) { s += ra[u].x * rb[u].x; s += ra[u].y * rb[u].y; }
      }
    }
    if ((n & 1) && blockIdx.x == 0 && first == 0) s += a[n - 1] * b[n - 1];
  } else {
    TILE_LOOP(BS, IT, n) {
      double ra[IT], rb[IT];
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        int64_t j = t0 + u * BS + first;
        if (j < n) { ra[u] = a[j]; rb[u] = b[j]; }
      }
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        int64_t j = t0 + u * BS + first;
        if (j < n) s += ra[u] * rb[u];
      }
    }
  }
  s = block_sum<BS>(s, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
  if (arrive_last(counter, &last_flag)) {
    double t = 0.0;
    for (int i = threadIdx.x; i < static_cast<int>(gridDim.x); i += BS)
      t += __ldcg(partials + i);
    t = block_sum<BS>(t, smem);
    if (threadIdx.x == 0) {
      *accum += dot_init + t;
      *counter = 0u;
    }
  }
}

// Shared launcher: the vector path when every pointer is 16-byte aligned, the
// scalar one otherwise.  A short array takes fewer items per thread (spread).
template <typename Op>
int launch_stream(const char* name, const double* in1, const double* in2, double* out, Op f,
                  int64_t n, const b200_tune* tune, cudaStream_t st) {
  if (n == 0) return B200_OK;
  const bool vec = aligned16(in1) && aligned16(in2) && aligned16(out) && n >= 2 &&
                   !(tune && tune->vec && tune->vec != 2);
  const int64_t units = vec ? n >> 1 : n;
  const Shape s = resolve_1d(tune, units, kBlock, spread(units, kBlock, kItems), vec ? 2 : 1);
  if (!valid_block(s.block)) return invalid("%s: bad block size %d", name, s.block);
  B200_DISPATCH_BLOCK(s.block, BS, B200_DISPATCH_ITEMS(s.items, IT,
    if (vec) launch(stream_kernel<BS, IT, double2, Op>, s.grid, BS, 0, st, in1, in2, out, f, n);
    else launch(stream_kernel<BS, IT, double, Op>, s.grid, BS, 0, st, in1, in2, out, f, n)));
  return after_launch(name);
}

}  // namespace

extern "C" {

int b200_stream_copy(const double* a, double* c, int64_t n,
                     const b200_tune* tune, b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!a || !c))) return invalid("b200_stream_copy: bad args");
  return launch_stream("b200_stream_copy", a, a, c, CopyOp{}, n, tune, as_stream(stream));
}

int b200_stream_mul(double* b, const double* c, double alpha, int64_t n,
                    const b200_tune* tune, b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!b || !c))) return invalid("b200_stream_mul: bad args");
  return launch_stream("b200_stream_mul", c, c, b, MulOp{alpha}, n, tune, as_stream(stream));
}

int b200_stream_add(const double* a, const double* b, double* c, int64_t n,
                    const b200_tune* tune, b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!a || !b || !c)))
    return invalid("b200_stream_add: bad args");
  return launch_stream("b200_stream_add", a, b, c, AddOp{}, n, tune, as_stream(stream));
}

int b200_stream_triad(double* a, const double* b, const double* c,
                      double alpha, int64_t n, const b200_tune* tune,
                      b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!a || !b || !c)))
    return invalid("b200_stream_triad: bad args");
  return launch_stream("b200_stream_triad", b, c, a, TriadOp{alpha}, n, tune,
                       as_stream(stream));
}

size_t b200_reduce_workspace_bytes(int64_t n, const b200_tune* tune) {
  int block = (tune && tune->block_size) ? tune->block_size : kBlock;
  // The smallest tile (1 item per thread) gives the largest grid, so the
  // workspace covers every reduction entry point and item count.
  return reduce_ws_bytes_for_grid(reduce_grid(n, tune, block, 1));
}

int b200_stream_dot(const double* a, const double* b, int64_t n,
                    double dot_init, double* dot_accum, void* workspace,
                    size_t workspace_bytes, const b200_tune* tune,
                    b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!a || !b)) || !dot_accum)
    return invalid("b200_stream_dot: bad args");
  int block = (tune && tune->block_size) ? tune->block_size : kBlock;
  int items = (tune && tune->items) ? tune->items : kItems;
  if (!valid_block(block)) return invalid("b200_stream_dot: bad block size %d", block);
  bool vec = aligned16(a) && aligned16(b) && !(tune && tune->vec == 1);
  int grid = reduce_grid(n, tune, block, items * (vec ? 2 : 1));
  size_t need = reduce_ws_bytes_for_grid(grid);
  if (!workspace || workspace_bytes < need) {
    set_error("b200_stream_dot: workspace %zu bytes, need %zu", workspace_bytes,
              need);
    return B200_ERR_WORKSPACE;
  }
  unsigned int* counter = static_cast<unsigned int*>(workspace);
  double* partials = reinterpret_cast<double*>(static_cast<char*>(workspace) + 256);
  cudaStream_t st = as_stream(stream);
  B200_DISPATCH_BLOCK(block, BS, B200_DISPATCH_ITEMS(items, IT,
    launch(dot_kernel<BS, IT>, grid, BS, 0, st, a, b, n, vec, dot_init, dot_accum, partials,
           counter)));
  return after_launch("b200_stream_dot");
}

}  // extern "C"
