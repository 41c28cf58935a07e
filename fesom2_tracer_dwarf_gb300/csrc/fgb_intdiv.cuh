// Correctly rounded FP64 division and multiplication on the integer pipe.
//
// This GPU issues one FP64 warp instruction per 16 cycles and SM (about two
// lanes a cycle), against four integer warp instructions per cycle: a hardware
// division, some nine dependent FP64 instructions, costs as much issue time as
// several hundred integer ones. The quotient of two significands is an integer
// problem, so it is solved there: a 64-bit reciprocal of the divisor by
// Newton's iteration from a single-precision estimate, a 64-bit product, and
// where that leaves the rounding open an exact remainder (the standard
// argument of correctly rounded division: the quotient of two p-bit
// significands is never halfway between two p-bit numbers, and the sign of the
// remainder at the midpoint decides). Every result is the IEEE
// round-to-nearest-even quotient, bit for bit; zeros, subnormals, infinities,
// NaNs and results near the ends of the exponent range go to the hardware
// division. A divisor used several times is prepared once (Divisor): about 30
// integer instructions, and 30 more per quotient. With it, and comparisons on
// the integer pipe (fgb_bits.cuh), the exact form's FCT ratio stage fell from
// 8.10 to 2.09 ms and its update from 7.28 to 2.67 ms (512^2 x 48, 2 tracers).
//
// Compiles for the host too, where the CPU tests compare it with the hardware.
#pragma once
#include <cstdint>
#include <cstring>

#ifndef FGB_HOST_RCP32
#define FGB_HOST_RCP32(f) (1.0f / (f))
#endif
#ifdef __CUDACC__
#define FGB_HD __host__ __device__ __forceinline__
#define FGB_COLD static __host__ __device__ __noinline__
#else
#define FGB_HD inline
#define FGB_COLD static
#endif

namespace fgb {
namespace intdiv {

// The bits of a double, by a move that the compiler does not see through: it
// turns integer tests of a double's bits (is it zero, is it finite) back into
// floating-point ones, which occupy the FP64 pipe (the element-gradient kernel
// issued 8.67 FP64 instructions per item with them, 6.0 without).
FGB_HD uint64_t to_bits(double x) {
#ifdef __CUDA_ARCH__
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
  return u;
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
FGB_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
FGB_HD int max_of(int a, int b) { return a > b ? a : b; }
FGB_HD uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
FGB_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
// 1 / f for f in [1, 2), within one unit of the last place.
FGB_HD float rcp32(float f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
#else
  return FGB_HOST_RCP32(f);
#endif
}

// The floating-point expressions behind the integer paths are rarely taken and
// must stay behind a branch: predicated into the common path, as the compiler
// does with a few instructions even of a function that is not inlined, they
// occupy the FP64 pipe there all the same. A loop is not predicated; this one
// runs once (a lane index is below 32), which the compiler does not know
// (512^2 x 48, 2 tracers: step 7.73 ms, without the loop 7.82).
FGB_HD uint32_t one_turn() {
#ifdef __CUDA_ARCH__
  uint32_t lane;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  return (lane >> 5) + 1;
#else
  return 1;
#endif
}
template <typename T, typename F>
FGB_HD T behind_branch(F f) {
  T r;
  uint32_t n = one_turn();
  do {
    r = f();
  } while (--n);
  return r;
}

FGB_COLD double hw_div(double a, double b) { return a / b; }

// The significand 1.f of a normal number as a 64-bit integer, leading bit set.
FGB_HD uint64_t significand(uint64_t bits) { return (1ull << 63) | (bits << 11); }

struct Divisor {
  uint64_t x;  // 2^64 / (B / 2^63), B the significand: low by less than 6 units
  double b;
  int e;       // biased exponent; far out of range for divisors the integer path leaves to the hardware
};

// The divisor b with its x from an earlier prepare(b).
FGB_HD Divisor prepared(double b, uint64_t x) {
  const int e = (int)(to_bits(b) >> 52) & 0x7ff;
  return Divisor{x, b, (unsigned)(e - 1) >= 2046u ? -100000 : e};
}

FGB_HD Divisor prepare(double b) {
  Divisor d = prepared(b, 0);
  const uint64_t B = significand(to_bits(b));
  const uint32_t Bhi = (uint32_t)(B >> 32), Blo = (uint32_t)B;
  // x0 / 2^32 below 2^63 / B by a factor of 1 - 2^-20 .. 1 - 2^-23: the estimate of the
  // truncated significand's reciprocal (relative error 2^-23, truncation 2^-23) times 1 - 2^-21
  const uint32_t fb = 0x3f800000u | ((Bhi >> 8) & 0x7fffffu);
#ifdef __CUDA_ARCH__
  const uint32_t x0 = __float2uint_rz(rcp32(__uint_as_float(fb)) * 4294965248.0f);
#else
  float f;
  std::memcpy(&f, &fb, 4);
  const uint32_t x0 = (uint32_t)(rcp32(f) * 4294965248.0f);
#endif
  // error term in units of 2^-63, below 2^43; x1 low by a factor of 1 - 2^-40 .. 1 - 2^-46
  const uint64_t E0 = (1ull << 63) - ((uint64_t)Bhi * x0 + mulhi32(Blo, x0));
  const uint64_t x1 = ((uint64_t)x0 << 32) + (((uint64_t)x0 * (uint32_t)(E0 >> 11)) >> 20);
  // below 2^24; its floor, the truncated factor and the truncated product each lose at most two units of x
  const uint32_t E1 = (uint32_t)(((1ull << 63) - 1) - mulhi64(B, x1));
  d.x = x1 + (((x1 >> 32) * (uint64_t)E1) >> 31);
  return d;
}

// The divisors 3 and 6: x = floor(2^64 / 1.5).
FGB_HD Divisor three() { return Divisor{0xaaaaaaaaaaaaaaaaull, 3.0, 1024}; }
FGB_HD Divisor six() { return Divisor{0xaaaaaaaaaaaaaaaaull, 6.0, 1025}; }

// a / d.b, rounded to nearest even.
FGB_HD double divide(double a, const Divisor& d) {
  const uint64_t bits = to_bits(a), A = significand(bits);
  const int ea = (int)(bits >> 52) & 0x7ff;
  // quotient of the significands times 2^63, in (2^62, 2^64), low by less than 10 units
  // (6 of the reciprocal's and one for each dropped part of the product)
  const uint32_t Ahi = (uint32_t)(A >> 32), Alo = (uint32_t)A, xhi = (uint32_t)(d.x >> 32), xlo = (uint32_t)d.x;
  const uint64_t Q = (uint64_t)Ahi * xhi + mulhi32(Ahi, xlo) + mulhi32(Alo, xhi);
  const uint32_t big = (uint32_t)(Q >> 63);  // quotient in [1, 2): one more bit below the last kept one
  const uint64_t t = Q + (512u << big);
  const uint32_t sh = 10 + big;
  uint64_t R = t >> sh;
  const int e = ea - d.e + 1021 + (int)big;  // the exponent field less one: R's leading bit adds it
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)e >= 2045u) {
    if ((bits << 1) == 0 && d.e > 0) return from_bits((bits ^ to_bits(d.b)) & (1ull << 63));  // zero by a normal number
    return hw_div(a, d.b);
  }
  if (((uint32_t)t << (32 - sh)) >= 0u - (10u << (32 - sh))) {
    // within 10 units below a midpoint: the remainder there decides, and its magnitude is far below 2^63
    const int64_t rem = (int64_t)(((A >> 11) << (54 - big)) - (2 * R + 1) * (significand(to_bits(d.b)) >> 11));
    R += rem >= 0;
  }
  return from_bits((((uint64_t)(uint32_t)e << 52) + R) | ((bits ^ to_bits(d.b)) & (1ull << 63)));
}

FGB_HD double divide(double a, double b) { return divide(a, prepare(b)); }

// a * b, rounded to nearest even, for kernels whose FP64 pipe is the bound
// while the integer pipe has room (some 35 integer instructions): gradients,
// volume fluxes and MUSCL increments with some of their products here 3.7 ms
// against 4.5 for 512^2 x 48, 2 tracers.
FGB_COLD double hw_mul(double a, double b) {
  return behind_branch<double>([&] { return a * b; });
}
// What the truncated product leaves open: the exact product's high half, rounded with its low
// half as the tie breaker.
FGB_COLD uint64_t round_product(uint64_t A, uint64_t B, uint32_t sh) {
  const uint64_t hi = mulhi64(A, B), R = (hi + (1ull << (sh - 1))) >> sh;
  const bool tie = (hi << (64 - sh)) == (1ull << 63) && A * B == 0;
  return tie ? R & ~1ull : R;
}
FGB_HD double multiply(double a, double b) {
  const uint64_t ua = to_bits(a), ub = to_bits(b), A = significand(ua), B = significand(ub);
  const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
  // the product of the significands / 2^64, in [2^62, 2^64), low by less than 3 units (dropped parts)
  const uint32_t Ahi = (uint32_t)(A >> 32), Alo = (uint32_t)A, Bhi = (uint32_t)(B >> 32), Blo = (uint32_t)B;
  const uint64_t Q = (uint64_t)Ahi * Bhi + mulhi32(Ahi, Blo) + mulhi32(Alo, Bhi);
  const uint32_t big = (uint32_t)(Q >> 63), sh = 10 + big;
  const int e = ea + eb - 1024 + (int)big;  // the exponent field less one
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)e >= 2045u) {
    if (((ua << 1) == 0 || (ub << 1) == 0) && max_of(ea, eb) < 2047) return from_bits((ua ^ ub) & (1ull << 63));
    return hw_mul(a, b);
  }
  const uint64_t t = Q + (512u << big);
  uint64_t R = t >> sh;
  // up to 3 units below a rounding boundary, or on it (a tie)
  if (((uint32_t)t << (32 - sh)) + (3u << (32 - sh)) < (4u << (32 - sh))) R = round_product(A, B, sh);
  return from_bits((((uint64_t)(uint32_t)e << 52) + R) | ((ua ^ ub) & (1ull << 63)));
}

}  // namespace intdiv
}  // namespace fgb
