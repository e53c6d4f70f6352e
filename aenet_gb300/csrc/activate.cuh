// Activation functions of the per-species networks and their derivatives
// (ff_activate, src/ext/feedforward.f90:932-969): 0 linear, 1 tanh,
// 2 sigmoid, 3 scaled tanh 1.7159 tanh(2x/3), 4 twisted tanh
// (scaled tanh + 0.1 x).
#pragma once

static __device__ __forceinline__ float tanh_t(float x) { return tanhf(x); }
static __device__ __forceinline__ double tanh_t(double x) { return tanh(x); }
static __device__ __forceinline__ float exp_t(float x) { return expf(x); }
static __device__ __forceinline__ double exp_t(double x) { return exp(x); }

// tanh in FP64 without branches, for kernels that the FP64 pipe bounds: tanh x
// = m / (m + 2), m = e^(2x) - 1 = 2^k (e^r - 1) + (2^k - 1) with 2x = k ln 2 +
// r, |r| <= ln 2 / 2; (e^r - 1 - r) / r^2 by its Chebyshev interpolant of
// degree 9 (4e-17 of e^r - 1 with these coefficients), the quotient by a
// third-order reciprocal step from an FP32 seed and one correction.  What the
// roundings of e^r - 1, m and m + 2 leave off is kept and enters that
// correction.  About 35 FP64 instructions at every x, accurate relative to the
// value down to zero: at most 1.36 ulp (the library's tanh 1.45; without the
// low parts 2.5).
__device__ __forceinline__ double tanh_even(double x) {
  const long long bits = __double_as_longlong(x), mag = bits & 0x7fffffffffffffffLL;
  // beyond 22 tanh rounds to 1
  const double ax = __longlong_as_double(mag < 0x4036000000000000LL ? mag : 0x4036000000000000LL);
  const double magic = 6755399441055744.0;          // 1.5 * 2^52: rounds to an integer
  const double kd = fma(ax, 2.0 * 1.4426950408889634074, magic);
  const int k = (int)__double_as_longlong(kd);
  const double kf = kd - magic;
  double r = fma(-kf, 0.693147180559663, ax + ax);  // ln 2 to 41 bits: exact product
  r = fma(-kf, 2.8235290563031577e-13, r);
  double p = 2.5100385495510319078e-8;
  p = fma(p, r, 2.7620088445409748161e-7);
  p = fma(p, r, 2.7557268459997064772e-6);
  p = fma(p, r, 0.000024801521295954375131);
  p = fma(p, r, 0.00019841269863053616878);
  p = fma(p, r, 0.0013888888917213716901);
  p = fma(p, r, 0.0083333333333300618325);
  p = fma(p, r, 0.041666666666624127873);
  p = fma(p, r, 0.16666666666666667453);
  p = fma(p, r, 0.50000000000000010221);
  const double c = p * r, ph = fma(c, r, r), pl = fma(c, r, r - ph);   // e^r - 1
  const double s = __longlong_as_double((long long)(k + 1023) << 52), s1 = s - 1.0;
  const double m = fma(s, ph, s1), ml = fma(s, pl, fma(s, ph, s1 - m));
  // m + 2 and its low part, from the larger of the two (m >= 1.83 from k = 2 on)
  const double hi = k < 2 ? 2.0 : m, lo = k < 2 ? m : 2.0;
  const double d = m + 2.0, dl = lo - (d - hi);
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
  const double y = (double)f, e = fma(-d, y, 1.0);
  const double inv = fma(y, fma(e, e, e), y);
  double q = m * inv;
  q = fma(fma(-q, d, m) + fma(-q, dl + ml, ml), inv, q);
  // sign, and NaN as it came
  const long long res = __double_as_longlong(q) | (bits & (long long)0x8000000000000000ULL);
  return __longlong_as_double(mag > 0x7ff0000000000000LL ? bits : res);
}

template <typename T>
__device__ __forceinline__ void activate(int t, T x, T& y, T& dy) {
  const T a = T(1.7159), b = T(0.666666666666667), c = T(0.1);
  switch (t) {
    case 0: y = x; dy = T(1); break;
    case 1: y = tanh_t(x); dy = T(1) - y * y; break;
    case 2: y = T(1) / (T(1) + exp_t(-x)); dy = y * (T(1) - y); break;
    case 3: { T tb = tanh_t(b * x); y = a * tb; dy = a * (T(1) - tb * tb) * b; } break;
    case 4: { T tb = tanh_t(b * x); y = a * tb + c * x; dy = a * (T(1) - tb * tb) * b + c; } break;
    default: y = T(0); dy = T(0);
  }
}
