// Compares what tests/intdiv_check.cu leaves out with the floating-point hardware: the constant divisors and divisors
// prepared elsewhere (host and device) and, on the device, the comparisons, the upwind product and the limiter's sums.
// The operands are that file's, and pairs whose product is near the smallest numbers.
#define main intdiv_check_main
#include "intdiv_check.cu"
#undef main
#ifdef __CUDACC__
#include "fgb_kernels.cuh"
#endif

static FGB_HD int check_divisors(double a, double b) {
  const Divisor p = prepare(b);
  return !same(divide(a, three()), a / 3.0, true) + !same(divide(a, six()), a / 6.0, true) +
         !same(divide(a, prepared(b, p.x)), a / b, true);
}
// Products around the subnormal range: exponents that add up to the smallest ones.
static FGB_HD void small_products(uint64_t& s, double& a, double& b) {
  const uint64_t M = (1ull << 52) - 1, ma = next(s) & M, mb = next(s) & M, sa = next(s) << 63, sb = next(s) << 63;
  const uint64_t ea = 1 + next(s) % 1000, sum = 950 + next(s) % 100;
  a = from_bits(sa | ea << 52 | ma);
  b = from_bits(sb | (sum > ea ? sum - ea : 1) << 52 | mb);
}

#ifdef __CUDACC__
static __global__ void k_check_bits(int n, unsigned long long seed, unsigned long long* bad) {
  namespace B = fgb::bits64;
  uint64_t s = seed ^ (0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1));
  for (int i = 0; i < n; ++i) {
    double a, b, c, d;
    const int kind = i % 9;
    if (kind == 8) small_products(s, a, b), small_products(s, c, d);
    else operands(kind, s, a, b), operands((int)(next(s) & 7), s, c, d);
    if (next(s) & 1) a = -a;
    if (next(s) & 1) c = -c;
    int w = check_divisors(a, b);
    w += B::product_positive(a, b) != (a * b > 0.0);
    // of zeros +0 exceeds -0; every other pair as the hardware compares
    const bool zeros = (to_bits(a) << 1) == 0 && (to_bits(b) << 1) == 0;
    w += B::exceeds(a, b) != (zeros ? (long long)to_bits(a) > (long long)to_bits(b) : a > b);
    w += B::unkey(B::key(a)) != a && !is_nan(to_bits(a));
    // v a, c upwind: the written expression; at the surface v a alone
    w += !same(B::upwind(b, a, c), 0.5 * (a * (b + fabs(b)) + c * (b - fabs(b))), false);
    w += !same(B::upwind(b, a, a, true), b * a, false);
    w += B::moderate(a, b) && isinf(2.0 * b * a);
    // the limiter's sums of two vertical and some horizontal terms
    double pos, neg, rp = fmax(0.0, a) + fmax(0.0, -c), rm = fmin(0.0, a) + fmin(0.0, -c);
    if (isnan(a) || isnan(c)) rp = rm = a + c;  // a NaN joins both sums
    fgb::first_parts(a, c, pos, neg);
    double t[3] = {b, d, -a};
    for (int k = 0; k < 3; ++k) {
      rp += isnan(t[k]) ? t[k] : fmax(0.0, t[k]);
      rm += isnan(t[k]) ? t[k] : fmin(0.0, t[k]);
      fgb::add_part(t[k], pos, neg);
    }
    fgb::spread_nan(pos, neg);
    w += !same(pos, rp, false) + !same(neg, rm, false);
    if (w) atomicAdd(bad, (unsigned long long)w);
  }
}
extern "C" long long check_bits_device(int blocks, int n, unsigned long long seed) {
  unsigned long long *bad, out = 0;
  if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return -1;
  k_check_bits<<<blocks, 256>>>(n, seed, bad);
  const cudaError_t e = cudaMemcpy(&out, bad, 8, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return e == cudaSuccess ? (long long)out : -1;
}
#else
int main() {
  uint64_t s = 88172645463325252ull;
  long long bad = 0;
  for (long long i = 0; i < 9000000; ++i) {
    double a, b;
    if (i % 9 == 8) small_products(s, a, b);
    else operands((int)(i % 9), s, a, b);
    bad += check_divisors(a, b);
  }
  std::printf("%lld\n", bad);
  return bad != 0;
}
#endif
