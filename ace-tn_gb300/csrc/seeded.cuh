// Reciprocal and square root in FP64 from FP32 seeds.
//
// CUDA's own are sequences of some ten dependent FP64 instructions, each of which occupies
// an SM quarter for 64 cycles here, in the serial chain of every Householder column, pivot
// and rotation.  The forms below take four to seven.
//
//  * 1 / x: with e = 1 - x r, 1 / x = r / (1 - e) = r (1 + e + e^2 + ...); three terms are
//    kept (the hyperpower iteration of order three, M. Altman, Pacific J. Math. 10 (1960)
//    1107).  The seed is an FP32 quotient (2 ulp, 2^-22) of a mantissa cut to 24 bits
//    (2^-23): |e| < 2^-21, and what is left out is e^3 < 2^-63.  The correction r (e + e^2)
//    is below 2^-21 of r, so its rounding errors do not count beside the last addition's:
//    the result is within one ulp.
//  * sqrt(x): with r = 1 - x y^2, x^(-1/2) = y (1 - r)^(-1/2) = y (1 + r / 2 + 3 r^2 / 8 +
//    ...), the binomial series; the seed's |r| < 2^-20 leaves 5 r^3 / 16 < 2^-61.  From z, so
//    refined, s = x z is within two roundings of the root, and one step of Heron's iteration
//    in the form s + z (x - s^2) / 2, whose residual an FMA has exactly up to its last
//    rounding, brings it within one ulp.
#pragma once

namespace ctm {

// |x| = m 2^e, m in [1, 2) as FP32 (truncated to 24 bits); false for zeros, subnormal and
// non-finite values.
__device__ __forceinline__ bool split_f64(double x, float& m, int& e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = int(b >> 52) & 0x7ff;
  m = __uint_as_float(0x3f800000u | (unsigned(b >> 29) & 0x7fffffu));
  e = ex - 1023;
  return ex != 0 && ex != 2047;
}

// FP32 value (normal) times 2^e as FP64, by bit patterns (a conversion takes an FP64 issue
// slot); 0 below the range.
__device__ __forceinline__ double join_f64(float v, int e) {
  const unsigned u = __float_as_uint(v);
  const int ex = int((u >> 23) & 0xffu) - 127 + 1023 + e;
  if (((u >> 23) & 0xffu) == 0u || ex < 1) return 0.0;
  const unsigned long long b = ((unsigned long long)(u & 0x80000000u) << 32) |
                               ((unsigned long long)ex << 52) |
                               ((unsigned long long)(u & 0x7fffffu) << 29);
  return __longlong_as_double((long long)b);
}

__device__ __forceinline__ double times_pow2(double x, int e) {  // results stay normal
  return __longlong_as_double(__double_as_longlong(x) + ((long long)e << 52));
}

// 1 / x, 1 <= x < 2, from its mantissa m.
__device__ __forceinline__ double mantissa_reciprocal(double x, float m) {
  const double r = join_f64(__fdividef(1.f, m), 0);
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// 1 / d for d > 0 within one ulp (subnormal results and arguments by a division).
__device__ __forceinline__ double positive_reciprocal(double d) {
  float m;
  int e;
  if (!split_f64(d, m, e) || e < -1000 || e > 1000) return 1.0 / d;
  return times_pow2(mantissa_reciprocal(times_pow2(d, -e), m), -e);
}

// alpha = -sign(a) sqrt(d) and beta = 2 / |v|^2 = 1 / (d - alpha a), d >= a^2: the root
// within one ulp, beta within 2^-51.4 (one rounding of d - alpha a besides); both 0 for a
// zero column, NaN for a non-finite one.
__device__ __forceinline__ void reflector(double d, double a, double& alpha, double& beta) {
  float m;
  int e;
  if (!split_f64(d, m, e)) {
    const bool finite = ((unsigned long long)__double_as_longlong(d) << 1) < 0xffe0000000000000ull;
    alpha = beta = finite ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const int odd = e & 1, half = (e - odd) / 2;
  const double x = times_pow2(d, -(e - odd));  // in [1, 4)
  const double y = double(rsqrtf(odd ? 2.f * m : m));
  const double r = fma(-(x * y), y, 1.0);
  const double z = fma(y * r, fma(r, 0.375, 0.5), y);
  double s = x * z;
  s = fma(0.5 * z, fma(-s, s, x), s);
  s = times_pow2(s, half);
  alpha = a >= 0.0 ? -s : s;
  beta = positive_reciprocal(fma(-alpha, a, d));
}

}  // namespace ctm
