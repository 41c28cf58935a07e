// Compares intdiv::divide and multiply (and, on the device, the helpers of bits64) with the
// floating-point hardware: random operands, quotients next to midpoints, extreme
// significands and exponents, special values. Compiled as C++ it checks the host
// build and prints the number of differing results; compiled by nvcc into a
// library, check_device does the same on the GPU.
#include <cstdio>
#include <cstdlib>

#ifdef ULPS  // the single-precision estimate pushed off by that many units in its last place
#include <cmath>
static float nudged(float f) {
  float r = 1.0f / f;
  for (int i = 0; i < (ULPS < 0 ? -ULPS : ULPS); ++i) r = std::nextafterf(r, ULPS < 0 ? 0.0f : 2.0f);
  return r;
}
#define FGB_HOST_RCP32(f) nudged(f)
#endif
#include "fgb_intdiv.cuh"
#ifdef __CUDACC__
#include "fgb_bits.cuh"
#endif

using namespace fgb::intdiv;

FGB_HD uint64_t next(uint64_t& s) {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
FGB_HD bool is_nan(uint64_t u) { return (u & ~(1ull << 63)) > 0x7ff0000000000000ull; }
FGB_HD bool same(double x, double y, bool zero_sign) {
  const uint64_t u = to_bits(x), v = to_bits(y);
  if (is_nan(u) || is_nan(v)) return is_nan(u) && is_nan(v);
  return u == v || (!zero_sign && (u << 1) == 0 && (v << 1) == 0);
}

// One pair of operands of the given kind.
FGB_HD void operands(int kind, uint64_t& s, double& a, double& b) {
  const uint64_t M = (1ull << 52) - 1, ma = next(s) & M, mb = next(s) & M, sg = next(s) & (1ull << 63);
  const uint64_t ea = 900 + next(s) % 246, eb = 900 + next(s) % 246, r = next(s);
  switch (kind) {
    case 0:
      a = from_bits(sg | ea << 52 | ma), b = from_bits(eb << 52 | mb);
      break;
    case 1:  // short significands: exact and repeating quotients
      a = (double)(int64_t)(r >> (ea % 63 + 1)), b = (double)(int64_t)((ma << 11 >> (eb % 63 + 1)) | 1);
      break;
    case 2: {  // next to a midpoint: a within a unit of (m + 1/2) b, from the product's high bits
      const uint64_t p = 2 * ((1ull << 52) | ma) + 1, q = (1ull << 52) | mb;
      const uint64_t hi = mulhi64(p << 10, q << 11);  // p q / 2^43
      const uint64_t top = hi >> 10;                  // p q / 2^53
      const uint64_t bits = top >> 53 ? (1024ull << 52 | ((top >> 1) & M)) : (1023ull << 52 | (top & M));
      a = from_bits(bits + r % 3 - 1), b = from_bits(1023ull << 52 | mb);
      break;
    }
    case 3:  // next to powers of two
      a = from_bits(ea << 52 | (r & 1 ? M - (r >> 8) % 4 : (r >> 8) % 4));
      b = from_bits(eb << 52 | (r & 2 ? M - (r >> 16) % 4 : (r >> 16) % 4));
      break;
    case 4:  // any bits
      a = from_bits(r), b = from_bits(ma | mb << 30);
      break;
    case 5:  // quotients into the subnormal range
      a = from_bits(sg | (r % 60) << 52 | ma), b = from_bits((1000 + (r >> 8) % 60) << 52 | mb);
      break;
    case 6:  // and past the largest number
      a = from_bits((2046 - r % 60) << 52 | ma), b = from_bits((1022 - (r >> 8) % 60) << 52 | mb);
      break;
    default: {
      const uint64_t sp[8] = {0, 1, 0x0010000000000000ull, 0x3ff0000000000000ull, 0x3ffffffffffffffful,
                              0x7fefffffffffffffull, 0x7ff0000000000000ull, 0x7ff8000000000000ull};
      a = from_bits(sp[r & 7] | sg), b = from_bits(sp[(r >> 3) & 7] | (r << 57 & 1ull << 63));
    }
  }
}

#ifdef __CUDACC__
static __global__ void k_check(int n, unsigned long long seed, unsigned long long* bad) {
  namespace B = fgb::bits64;
  uint64_t s = seed ^ (0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1));
  for (int i = 0; i < n; ++i) {
    double a, b;
    operands(i & 7, s, a, b);
    int d = !same(divide(a, b), a / b, true) + !same(multiply(a, b), a * b, true);
    d += !same(multiply(a, from_bits(to_bits(b) & ~((1ull << 27) - 1))), a * from_bits(to_bits(b) & ~((1ull << 27) - 1)), true);
    d += !same(B::lesser(a, b), a < b ? a : b, false) + !same(B::greater(a, b), a > b ? a : b, false);
    d += !same(B::twice(a), a + a, true) + !same(B::half(a), a * 0.5, true) + !same(B::magnitude(a), fabs(a), true);
    if (d) atomicAdd(bad, (unsigned long long)d);
  }
}
extern "C" long long check_device(int blocks, int n, unsigned long long seed) {
  unsigned long long *bad, out = 0;
  if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return -1;
  k_check<<<blocks, 256>>>(n, seed, bad);
  const cudaError_t e = cudaMemcpy(&out, bad, 8, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return e == cudaSuccess ? (long long)out : -1;
}
#else
int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 8000000;
  uint64_t s = 88172645463325252ull;
  long long bad = 0;
  for (long long i = 0; i < n; ++i) {
    double a, b;
    operands((int)(i & 7), s, a, b);
    bad += !same(divide(a, b), a / b, true) + !same(multiply(a, b), a * b, true);
    // short significands: exact products and ties
    for (int cut = 20; cut < 32; cut += 3) {
      const double x = from_bits(to_bits(a) >> cut << cut), y = from_bits(to_bits(b) >> (53 - cut) << (53 - cut));
      bad += !same(multiply(x, y), x * y, true);
    }
  }
  std::printf("%lld\n", bad);
  return bad != 0;
}
#endif
