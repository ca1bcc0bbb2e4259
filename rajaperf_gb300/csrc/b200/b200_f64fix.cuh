// Chains of exactly rounded FP64 adds on the integer pipes, in fixed point.
//
// b200_f64emu.cuh's adds unpack both operands and pack the result, some 36 to
// 65 integer instructions each.  A stencil adds the same few values, all of
// similar size, again and again: here a value is unpacked once, into a 64-bit
// integer in a unit of the thread's own (`Unit`, from one of its values'
// exponents), and an add of two such integers is exact; rounding the sum to its
// 53 leading bits (round53) gives what the FP64 pipe's add would, in about 11
// instructions, and only the last sum is packed into a double again.
//
// Range: values of one sign whose exponents lie in a window of 7 (8) binades fit
// exactly as magnitudes (f < 2^59 or 2^60), so sums of up to 15 (7) of them stay
// below 2^63 - 2^10.  A value outside the window or of the other sign (zeros, subnormals,
// infinities and NaNs among them) sets `slow`, and the caller redoes the point
// on the FP64 pipe.  The unit is kept far from both ends of the exponent
// range, so no intermediate result is subnormal or overflows, and a zero sum
// can only come from a cancellation: +0, as round to nearest has it.
#pragma once

#include "b200_f64emu.cuh"

namespace b200 {
namespace f64fix {

// Sign (bit 11) and biased exponent of the window's lowest binade: an integer
// f stands for +-f * 2^(exponent - 1075).
struct Unit {
  uint32_t low;
};

// The window that starts `below` binades under x's.
__device__ __forceinline__ Unit unit_at(double x, int below, bool& slow) {
  const uint32_t e = static_cast<uint32_t>(__double2hiint(x)) >> 20;
  const uint32_t low = e - static_cast<uint32_t>(below);
  slow |= (low & 0x7ffu) - 200u > 1600u;  // also x zero, subnormal, infinite or NaN
  return Unit{low};
}

// x in the unit; BINADES: the window's.  Eight serve HEAT_3D, which sums six
// values; the test for seven is the cheaper one (JACOBI_2D 529 us a pass at
// 1002^2 and 40 steps, with eight 538).
template <uint32_t BINADES = 7>
__device__ __forceinline__ int64_t fix(double x, Unit u, bool& slow) {
  static_assert(BINADES == 7 || BINADES == 8, "sums of what its callers add fit in 63 bits");
  const uint64_t b = f64emu::bits_opaque(x);
  const uint32_t s = (static_cast<uint32_t>(b >> 32) >> 20) - u.low;
  slow |= s > BINADES - 1u;
  int64_t m;
  asm("shl.b64 %0, %1, %2;" : "=l"(m) : "l"((b & f64emu::kFrac) | f64emu::kHidden), "r"(s));
  return m;
}

// f + v as one multiply-add, on the FMA pipe instead of the ALU
__device__ __forceinline__ int64_t add_small(int64_t f, uint32_t v) {
  int64_t r;
  asm("mad.wide.u32 %0, %1, 1, %2;" : "=l"(r) : "r"(v), "l"(f));
  return r;
}

// f rounded to its 53 leading bits, ties to even (|f| < 2^63 - 2^10).  With p
// the bits to drop, adding 2^(p-1) - 1 plus the last kept bit carries into the
// kept part exactly when rounding up is due; the two's complement of a
// negative value rounds alike (ties go to the even neighbour on either side).
__device__ __forceinline__ int64_t round53(int64_t f) {
  const uint32_t lo = static_cast<uint32_t>(f);
  int32_t top;  // index of the upper word's first bit that differs from its sign, or -1
  asm("bfind.s32 %0, %1;" : "=r"(top) : "r"(static_cast<int32_t>(f >> 32)));
  const uint32_t p = static_cast<uint32_t>(max(top - 20, 0));
  uint32_t drop;  // 2^p - 1
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(drop) : "r"(p));
  const uint32_t bias = (drop >> 1) + ((lo >> p) & 1u & drop);
  return add_small(f, bias) & ~static_cast<int64_t>(drop);
}

// f * 2^k in the unit as a double, rounded to nearest even.
__device__ __forceinline__ double pack(int64_t f, Unit u, int k) {
  const int64_t s = f >> 63;
  const uint64_t a = static_cast<uint64_t>((f ^ s) - s);
  const uint32_t lz = static_cast<uint32_t>(__clzll(static_cast<long long>(a)));
  const uint64_t w = a << (lz & 63u), m = w >> 11;
  const uint32_t up =
      ((static_cast<uint32_t>(w) & 0x7ffu) + 0x3ffu + (static_cast<uint32_t>(m) & 1u)) >> 11;
  const uint64_t e = u.low + static_cast<uint32_t>(10 + k) - lz;  // one less: m has the hidden bit
  const uint64_t sign = static_cast<uint64_t>(f) & f64emu::kSign;
  return a == 0u ? 0.0 : f64emu::from_bits(sign ^ ((e << 52) + m + up));
}

// c * (f in the unit), rounded to nearest even, for f > 0 of at most 53
// significant bits and a positive normal c given by its significand (53 bits)
// and biased exponent.  The product of the two significands, both shifted up
// to bit 63, is exact in 128 bits; what lies below its upper word only breaks
// ties.
__device__ __forceinline__ double pack_times(int64_t f, Unit u, uint64_t mant, int exponent) {
  const uint32_t lz = static_cast<uint32_t>(__clzll(f));
  const uint64_t w = static_cast<uint64_t>(f) << (lz & 63u), c = mant << 11;
  uint64_t hi = __umul64hi(w, c);
  const uint64_t lo = w * c;
  const uint32_t top = static_cast<uint32_t>(hi >> 63);
  hi = top ? hi : (hi << 1) | (lo >> 63);
  const uint32_t below = (lo << (1u - top)) != 0u ? 1u : 0u;
  const uint64_t m = hi >> 11;
  const uint32_t up =
      (((static_cast<uint32_t>(hi) & 0x7ffu) | below) + 0x3ffu + (static_cast<uint32_t>(m) & 1u)) >>
      11;
  const uint64_t e = u.low + static_cast<uint32_t>(exponent - 1023 + 10) + top - lz;
  return f64emu::from_bits((e << 52) + m + up);
}

}  // namespace f64fix
}  // namespace b200
