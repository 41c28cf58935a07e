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
// Below 2^511 in magnitude (so not a NaN): twice the product of two such numbers is finite.
__device__ __forceinline__ bool moderate(double x) { return mag_hi(x) < 0x5fe00000u; }
__device__ __forceinline__ bool moderate(double x, double y) { return max(mag_hi(x), mag_hi(y)) < 0x5fe00000u; }

// The floating-point expressions behind the integer ones (see one_turn).
using intdiv::behind_branch;
static __device__ __noinline__ double hw_lesser(double a, double b) {
  return behind_branch<double>([&] { return a < b ? a : b; });
}
static __device__ __noinline__ double hw_greater(double a, double b) {
  return behind_branch<double>([&] { return a > b ? a : b; });
}
static __device__ __noinline__ bool hw_exceeds(double a, double b) {
  return behind_branch<bool>([&] { return a > b; });
}
static __device__ __noinline__ double hw_upwind(double v, double t1, double t2) {
  return behind_branch<double>([&] { return 0.5 * (t1 * (v + fabs(v)) + t2 * (v - fabs(v))); });
}
static __device__ __noinline__ bool hw_product_positive(double a, double b) {
  return behind_branch<bool>([&] { return a * b > 0.0; });
}

// a < b ? a : b
__device__ __forceinline__ double lesser(double a, double b) {
  if (!finite(a, b)) return hw_lesser(a, b);
  return key(a) < key(b) ? a : b;
}
// a > b ? a : b
__device__ __forceinline__ double greater(double a, double b) {
  if (!finite(a, b)) return hw_greater(a, b);
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
  if ((b << 1) == 0) return x;
  if (e - 0x00100000u >= 0x7fd00000u) return intdiv::hw_mul(x, 2.0);
  return from_bits(b + (1ull << 52));
}
__device__ __forceinline__ double half(double x) {
  const uint64_t b = to_bits(x);
  const unsigned e = (unsigned)(b >> 32) & 0x7ff00000u;
  if ((b << 1) == 0) return x;
  if (e - 0x00200000u >= 0x7fd00000u) return intdiv::hw_mul(x, 0.5);
  return from_bits(b - (1ull << 52));
}

// (t1 (v + |v|) + t2 (v - |v|)) / 2, the upwind product of a first-order flux:
// one factor in brackets is zero and the other 2 v, so it is v times the
// upwind value, one FP64 instruction. Where that is not the expression's value
// bit for bit (a subnormal product, whose double rounds first; a double that
// overflows; infinities and NaNs) the expression as written, or with `plain`
// v * t1 (the surface flux, t1 = t2).
__device__ __forceinline__ double upwind(double v, double t1, double t2, bool plain = false) {
  const bool first = sign_clear(v);
  const double p = (first ? t1 : t2) * v;
  const unsigned rest = max(mag_hi(v), mag_hi(first ? t2 : t1));
  if (rest >= 0x7fe00000u || mag_hi(p) - 0x00100000u >= 0x7fd00000u) {
    if ((to_bits(p) << 1) == 0 && rest < 0x7fe00000u) return p;  // zero times a number
    return plain ? intdiv::hw_mul(v, t1) : hw_upwind(v, t1, t2);
  }
  return p;
}
// a * b > 0, from the signs; factors small enough for the product to vanish by multiplication.
__device__ __forceinline__ bool product_positive(double a, double b) {
  const uint64_t ua = to_bits(a), ub = to_bits(b);
  if ((ua << 1) == 0 || (ub << 1) == 0) return false;
  const unsigned ea = mag_hi(a) >> 20, eb = mag_hi(b) >> 20;  // biased exponents
  if (min(ea, eb) < 550u || max(ea, eb) == 0x7ffu) return hw_product_positive(a, b);
  return (long long)(ua ^ ub) >= 0;
}
// a > b (of finite zeros: +0 > -0).
__device__ __forceinline__ bool exceeds(double a, double b) { return finite(a, b) ? key(a) > key(b) : hw_exceeds(a, b); }

}  // namespace bits64
}  // namespace fgb
