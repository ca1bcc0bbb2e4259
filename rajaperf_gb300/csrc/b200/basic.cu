// Basic group kernels used by the batched small-size suite: DAXPY, INIT3,
// MULADDSUB (suite src/basic/*.hpp bodies).
#include "b200_internal.cuh"
#include "b200_map.cuh"

using namespace b200;

namespace {

// basic/DAXPY.hpp: y[i] += a * x[i]
struct Daxpy {
  double* y;
  const double* x;
  double a;
  using Out = double;
  __device__ Out compute(int64_t i) const { return y[i] + a * ld(x + i); }
  __device__ void store(int64_t i, Out v) const { y[i] = v; }
};

// basic/INIT3.hpp: out1 = out2 = out3 = -in1 - in2
struct Init3 {
  double* out1;
  double* out2;
  double* out3;
  const double* in1;
  const double* in2;
  using Out = double;
  __device__ Out compute(int64_t i) const { return -ld(in1 + i) - ld(in2 + i); }
  __device__ void store(int64_t i, Out v) const {
    out3[i] = v;
    out2[i] = v;
    out1[i] = v;
  }
};

// basic/MULADDSUB.hpp
struct MulAddSub {
  double* out1;
  double* out2;
  double* out3;
  const double* in1;
  const double* in2;
  struct Out { double product, sum, difference; };
  __device__ Out compute(int64_t i) const {
    const double a = ld(in1 + i), b = ld(in2 + i);
    return {a * b, a + b, a - b};
  }
  __device__ void store(int64_t i, const Out& o) const {
    out1[i] = o.product;
    out2[i] = o.sum;
    out3[i] = o.difference;
  }
};

}  // namespace

extern "C" {

int b200_basic_daxpy(double* y, const double* x, double a, int64_t n,
                     const b200_tune* tune, b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!x || !y))) return invalid("b200_basic_daxpy: bad args");
  return launch_map1d("b200_basic_daxpy", Daxpy{y, x, a}, n, tune, as_stream(stream));
}

int b200_basic_init3(double* out1, double* out2, double* out3, const double* in1,
                     const double* in2, int64_t n, const b200_tune* tune,
                     b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!out1 || !out2 || !out3 || !in1 || !in2)))
    return invalid("b200_basic_init3: bad args");
  return launch_map1d("b200_basic_init3", Init3{out1, out2, out3, in1, in2}, n, tune,
                      as_stream(stream));
}

int b200_basic_muladdsub(double* out1, double* out2, double* out3, const double* in1,
                         const double* in2, int64_t n, const b200_tune* tune,
                         b200_stream_t stream) {
  if (n < 0 || (n > 0 && (!out1 || !out2 || !out3 || !in1 || !in2)))
    return invalid("b200_basic_muladdsub: bad args");
  return launch_map1d("b200_basic_muladdsub", MulAddSub{out1, out2, out3, in1, in2}, n,
                      tune, as_stream(stream));
}

}  // extern "C"
