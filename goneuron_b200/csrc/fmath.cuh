// fmath.cuh -- exponential and hyperbolic tangent rounded to float32 as the reference does (float64 libm, then rounded), without
// float64 arithmetic.
//
// The reference evaluates its activations as float32(math.Exp(float64(x))) (activations.go:25-58, :135-143).  Done literally on
// the GPU, one such value is a chain of some twenty float64 operations: it set the pace of the recurrences (two in a row per
// time-step) and of the element-wise GELU passes (20 us for 5.5 M elements, 7 us of memory traffic).  Here the result is formed
// as an unevaluated sum of two floats (Dekker 1971: error-free sums and, with fma, products) good to about 2^-29, and rounded
// once: at most 0.53 ulp from the exact value, where one float64 rounding gives 0.5.
// Argument reduction after Cody and Waite (1980): x = n ln 2 + r, |r| <= ln(2)/2, ln 2 in three pieces of which the first has few
// enough bits for n times it to be exact; e^r by its Taylor series.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace gn {

struct FPair { float h, l; };
__host__ __device__ __forceinline__ FPair two_sum(float a, float b) { const float s = a + b, bb = s - a; return FPair{s, (a - (s - bb)) + (b - bb)}; }
__host__ __device__ __forceinline__ FPair fast_two_sum(float a, float b) { const float s = a + b; return FPair{s, b - (s - a)}; }      // |a| >= |b|
// 2^n for -126 <= n <= 127
__host__ __device__ __forceinline__ float pow2i(int n) {
#ifdef __CUDA_ARCH__
  return __int_as_float((n + 127) << 23);
#else
  return ldexpf(1.f, n);
#endif
}
// r and n with x = n ln 2 + r, |r| <= 0.3466; |x| below about 120
__host__ __device__ __forceinline__ FPair ln2_reduce(float x, float& n) {
  n = rintf(x * 1.44269504088896341f);
  const float r0 = fmaf(-n, 0.693359375f, x);                        // 355 / 512: exact
  const float c = 2.1219444170128554e-4f;
#ifdef __CUDA_ARCH__
  const float p = __fmul_rn(n, c);                                   // (not to be contracted into the sums below)
#else
  const float p = n * c;
#endif
  const float pe = fmaf(n, c, -p);
  const FPair r = two_sum(r0, p);
  return FPair{r.h, r.l + fmaf(n, -1.6465949582897082e-12f, pe)};
}
// e^r - 1 - r as a pair: r^2 / 2 without error, the rest of the Taylor series (remainder 2e-10) in float
__host__ __device__ __forceinline__ FPair exp_tail(FPair r) {
  const float t = r.h * r.h, tl = fmaf(r.h, r.h, -t);
  float q = fmaf(1.f / 40320.f, r.h, 1.f / 5040.f);
  q = fmaf(q, r.h, 1.f / 720.f); q = fmaf(q, r.h, 1.f / 120.f); q = fmaf(q, r.h, 1.f / 24.f); q = fmaf(q, r.h, 1.f / 6.f);
  return FPair{0.5f * t, fmaf(q, t * r.h, fmaf(r.h, r.l, 0.5f * tl))};
}
// e^r as a normalised pair
__host__ __device__ __forceinline__ FPair exp_small(FPair r) {
  const FPair e = exp_tail(r), a = fast_two_sum(1.f, r.h), b = fast_two_sum(a.h, e.h);
  return fast_two_sum(b.h, b.l + (a.l + (r.l + e.l)));
}
// float32(exp(x))
__host__ __device__ __forceinline__ float exp_rn(float x) {
  float y = x > 90.f ? 90.f : x; y = y < -110.f ? -110.f : y;        // (a NaN passes)
  float nf; const FPair e = exp_small(ln2_reduce(y, nf));
  const int n = (int)nf, n1 = n >> 1;                                // two factors: 2^n itself may be out of range
  return e.h * pow2i(n1) * pow2i(n - n1);                            // (e.h is the pair rounded to float)
}
// float32(tanh(x)) = sign(x) m / (m + 2) with m = e^(2|x|) - 1
__host__ __device__ __forceinline__ float tanh_rn(float x) {
  float a = fabsf(x); a = a > 10.f ? 10.f : a;                       // (tanh(10) rounds to 1; a NaN passes)
  const float y = a + a;
  FPair m;
  if (y < 0.34f) {
    const FPair e = exp_tail(FPair{y, 0.f});
    m = fast_two_sum(y, e.h); m = fast_two_sum(m.h, m.l + e.l);
  } else {
    float nf; const FPair e = exp_small(ln2_reduce(y, nf)); const float s = pow2i((int)nf);
    m = two_sum(e.h * s, -1.f); m = fast_two_sum(m.h, fmaf(e.l, s, m.l));
  }
  const FPair d0 = two_sum(2.f, m.h), d = fast_two_sum(d0.h, d0.l + m.l);
  const float i = 1.f / d.h, q = m.h * i, rem = fmaf(-q, d.l, fmaf(-q, d.h, m.h) + m.l);
  return copysignf(fmaf(rem, i, q), x);
}

// GELU, tanh form (activations.go:241-275): x / (1 + e^-y) with y = 2 sqrt(2 / pi) (x + 0.044715 x^3).  One function for the element-wise pass
// and for the epilogues that write their result as operand planes, where its arithmetic is what an element costs.
// m = e^y - 1 in plain float (reduction and series as above, one rounding for the product with 2^n); then
//   y > 1: x - x / (m + 2),   |y| <= 1: x / 2 + x (m / 2) / (m + 2),   y < -1: x (m + 1) / (m + 2)
// so that what the quotient's two ulp apply to is at most a quarter of x.  Against float64 over all x the error is below 9.5e-8 |x|,
// root mean square 2.4e-8 |x|; the reference's own order, float32 around a rounded tanh, has 1.20e-7 and 3.3e-8 (it adds 1 to the tanh).
// With the hardware's exponential and quotient it was 1.8e-7 and 4.7e-8 for some twenty instructions less (a training step of 24
// sequences of 150 tokens, width 384: 1297 us, now 1312; 1387 with the tanh above).
__device__ __forceinline__ float gelu_f(float x) {
  const float y = fminf(fmaxf(x * fmaf(0.07135481627f * x, x, 1.5957691216057308f), -80.f), 80.f);      // (a NaN becomes -80)
  const float t = fmaf(y, 1.44269504088896341f, 12582912.f), n = t - 12582912.f;       // 1.5 2^23: rounds to a whole number, low bits of t
  const float r = fmaf(n, 2.1219444170128554e-4f, fmaf(n, -0.693359375f, y)), s = __int_as_float((__float_as_int(t) << 23) + 0x3f800000);
  float q = fmaf(1.f / 5040.f, r, 1.f / 720.f);
  q = fmaf(q, r, 1.f / 120.f); q = fmaf(q, r, 1.f / 24.f); q = fmaf(q, r, 1.f / 6.f); q = fmaf(q, r, 0.5f);
  const float p = fmaf(r * r, q, r), m = fmaf(p, s, s - 1.f);
  const bool hi = y > 1.f, lo = y < -1.f;
  const float v = fmaf(x, __fdividef(hi ? -1.f : lo ? fmaf(p, s, s) : 0.5f * m, m + 2.f), hi ? x : lo ? 0.f : 0.5f * x);
  return fabsf(y) < 80.f ? v : x * (y > 0.f ? 1.f : 0.f);                              // (infinities as the reference's product gives them)
}

}  // namespace gn
