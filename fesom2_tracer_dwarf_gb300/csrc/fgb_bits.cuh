// Comparisons and sign tests of FP64 values on the integer pipe.
//
// An FP64 comparison occupies the FP64 pipe for 16 cycles per warp and SM like
// any FP64 instruction, sixty times an integer one; the order of two doubles
// that are not NaN is the order of their bits read as sign-magnitude integers.
// Each helper gives the value the floating-point expression gives (the sign
// of a zero result may differ) and leaves NaNs and infinities to the hardware
// comparison.
#pragma once
#include <cstdint>

#include "fgb_intdiv.cuh"

namespace fgb {
namespace bits64 {

using intdiv::from_bits;
using intdiv::to_bits;

// Order-preserving integer key (its own inverse): a < b as keys exactly when
// a < b as numbers, -0 below +0, and every NaN outside [-kKeyInf - 1, kKeyInf].
__device__ __forceinline__ long long key(double x) {
  const long long b = (long long)to_bits(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double unkey(long long k) {
  return from_bits((uint64_t)(k ^ ((k >> 63) & 0x7fffffffffffffffLL)));
}
constexpr long long kKeyInf = 0x7ff0000000000000LL;  // key(+inf); key(-inf) is -kKeyInf - 1

__device__ __forceinline__ unsigned mag_hi(double x) { return (unsigned)(to_bits(x) >> 32) & 0x7fffffffu; }
// Neither infinite nor NaN.
__device__ __forceinline__ bool finite(double x) { return mag_hi(x) < 0x7ff00000u; }
__device__ __forceinline__ bool finite(double x, double y) { return max(mag_hi(x), mag_hi(y)) < 0x7ff00000u; }

// a < b ? a : b
__device__ __forceinline__ double lesser(double a, double b) {
  if (!finite(a, b)) return a < b ? a : b;
  return key(a) < key(b) ? a : b;
}
// a > b ? a : b
__device__ __forceinline__ double greater(double a, double b) {
  if (!finite(a, b)) return a > b ? a : b;
  return key(a) > key(b) ? a : b;
}
// x >= 0 by the sign bit: -0 and NaN may go either way.
__device__ __forceinline__ bool sign_clear(double x) { return (long long)to_bits(x) >= 0; }
__device__ __forceinline__ double negate_if(double x, bool neg) {
  return from_bits(to_bits(x) ^ ((uint64_t)neg << 63));
}
// |x|, exactly as fabs (a sign-bit operation), kept off the FP64 pipe.
__device__ __forceinline__ double magnitude(double x) { return from_bits(to_bits(x) & 0x7fffffffffffffffull); }

// 2 x and x / 2, exact; zeros, subnormal and extreme exponents by multiplication.
__device__ __forceinline__ double twice(double x) {
  const uint64_t b = to_bits(x);
  const unsigned e = (unsigned)(b >> 32) & 0x7ff00000u;
  if (e - 0x00100000u >= 0x7fd00000u) return x + x;
  return from_bits(b + (1ull << 52));
}
__device__ __forceinline__ double half(double x) {
  const uint64_t b = to_bits(x);
  const unsigned e = (unsigned)(b >> 32) & 0x7ff00000u;
  if (e - 0x00200000u >= 0x7fd00000u) return x * 0.5;
  return from_bits(b - (1ull << 52));
}

}  // namespace bits64
}  // namespace fgb
