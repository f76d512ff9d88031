// exp(x) in FP64 by P. T. P. Tang's table-driven method ("Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM Trans. Math. Softw. 15(2), 1989), for the sweep's
// Maxwellian values (x <= 0), from the mathematics:
//   x = (256 m + j) ln2/256 + r,  j = 0..255,  |r| <= ln2/512,
//   exp(x) = 2^m * 2^(j/256) * exp(r),
// with k = 256 m + j the integer nearest x*256/ln2 (rounded by adding and
// subtracting 1.5*2^52), r = x - k*ln2/256 by two fused multiply-adds with
// ln2/256 split into a 32-bit head and its remainder, and exp(r) - 1 by the
// Taylor polynomial of degree 4 (truncation error |r|^5/120 < 4e-17
// relative).  The table tab[j] = 2^(j/256) is the caller's (in shared memory,
// 2 KB; with 64 entries the polynomial took a degree more); 2^m is applied by
// an integer add to the exponent field.  From x = -707 down (results under
// 1e-307) the value is flushed to +0, by an integer comparison of the high
// word, which keeps the FP64 pipe free and lets a NaN, whatever its sign,
// through.  Measured against long-double exp on the host
// (tests/test_exp_tang.py).
#pragma once
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define DGBGK_HD __host__ __device__ __forceinline__
#else
#define DGBGK_HD inline
#endif

namespace dgbgk {

constexpr int EXP_BITS = 8, EXP_TAB = 1 << EXP_BITS;

DGBGK_HD double dbl_from_bits(int64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double d;
  std::memcpy(&d, &b, sizeof d);
  return d;
#endif
}
DGBGK_HD int64_t dbl_bits(double d) {
#if defined(__CUDA_ARCH__)
  return (int64_t)__double_as_longlong(d);
#else
  int64_t b;
  std::memcpy(&b, &d, sizeof b);
  return b;
#endif
}

DGBGK_HD double exp_tang(double x, const double* __restrict__ tab) {
  const double inv_step = 369.3299304675746;        // 256 / ln2
  const double step_hi = 0.00270760617331689;      // ln2/256, leading 32 bits
  const double step_lo = 7.453964567463233e-13;     // ln2/256 - step_hi
  const double shift = 6755399441055744.0;          // 1.5 * 2^52
  const double ks = fma(x, inv_step, shift);        // k in the low word
  const double kd = ks - shift;
  const int k = (int)(uint32_t)dbl_bits(ks);
  double r = fma(-kd, step_hi, x);
  r = fma(-kd, step_lo, r);
  double p = fma(r, 1.0 / 24.0, 1.0 / 6.0);
  p = fma(r, p, 0.5);
  p = fma(r, p, 1.0);
  p = r * p;  // exp(r) - 1
  const double t = tab[k & (EXP_TAB - 1)];
  const double y = fma(t, p, t);
  const int64_t m = (int64_t)(k >> EXP_BITS);  // floor(k / 256)
  // 2^m: m added to the exponent field (two's complement, shifted unsigned)
  const double v = dbl_from_bits((int64_t)((uint64_t)dbl_bits(y) + ((uint64_t)m << 52)));
  // high words from -707 to -infinity, NaNs not among them
  const uint32_t h = (uint32_t)((uint64_t)dbl_bits(x) >> 32);
  return h - 0xC0861800u <= 0xFFF00000u - 0xC0861800u ? 0.0 : v;
}

}  // namespace dgbgk
