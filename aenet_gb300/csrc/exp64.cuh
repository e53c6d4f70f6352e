// Exponentials in FP64 for kernels that the FP64 pipe (two lanes per clock and
// SM) bounds: powers of 2^(1/32) from a table (load pipe), the power of two by
// the exponent's bits, a short series for the rest.
#pragma once

// 2^(j / 32) and what its rounding left off
static __device__ const double2 EXP2_32[32] = {
    {1.0, 0.0},
    {1.0218971486541166, 5.109225028973444e-17},
    {1.0442737824274138, 8.551889705537965e-17},
    {1.0671404006768237, -7.899853966841582e-17},
    {1.0905077326652577, -3.046782079812471e-17},
    {1.1143867425958924, 1.0410278456845571e-16},
    {1.1387886347566916, 8.912812676025408e-17},
    {1.1637248587775775, 3.8292048369240935e-17},
    {1.189207115002721, 3.982015231465646e-17},
    {1.215247359980469, -7.712630692681488e-17},
    {1.241857812073484, 4.658027591836937e-17},
    {1.2690509571917332, 2.667932131342186e-18},
    {1.2968395546510096, 2.5382502794888315e-17},
    {1.3252366431597413, -2.8587312100388614e-17},
    {1.3542555469368927, 7.70094837980299e-17},
    {1.383909881963832, -6.770511658794786e-17},
    {1.4142135623730951, -9.667293313452913e-17},
    {1.4451808069770467, -3.0237581349939873e-17},
    {1.4768261459394993, -3.483994556892796e-17},
    {1.5091644275934228, -1.016455327754295e-16},
    {1.5422108254079407, 7.949834809697621e-17},
    {1.5759808451078865, -1.0136916471278304e-17},
    {1.6104903319492543, 2.4707192569797888e-17},
    {1.645755478153965, -1.0125679913674773e-16},
    {1.681792830507429, 8.199010020581497e-17},
    {1.718619298122478, -1.851380418263111e-17},
    {1.7562521603732995, 2.960140695448873e-17},
    {1.7947090750031072, 1.8227458427912087e-17},
    {1.8340080864093424, 3.283107224245627e-17},
    {1.8741676341103, -6.122763413004143e-17},
    {1.9152065613971474, -1.0619946056195963e-16},
    {1.9571441241754002, 8.960767791036668e-17},
};

// x = k ln 2 / 32 + r, |r| < ln 2 / 64, exp x = 2^(k / 32) (1 + r + r^2 (1/2 +
// ... + r^4 / 720)).  Twelve FP64 instructions; error at most 0.56 ulp over 15
// million arguments (exp: 0.89; without the low parts 1.02); |x| beyond 700,
// infinities and NaN go to the library.  750 rutile atoms: forward 481 -> 457
// us, adjoint 846 -> 822 us against exp.
__device__ __forceinline__ double exp_table(double x) {
  if ((__double2hiint(x) & 0x7fffffff) >= 0x4085e000) return exp(x);
  const double magic = 6755399441055744.0;   // 1.5 * 2^52: rounds to an integer
  const double kd = fma(x, 46.16624130844683, magic);
  const int k = __double2loint(kd);
  const double kf = kd - magic;
  double r = fma(-kf, 0.02166084937925916, x);   // ln 2 / 32 to 31 bits: exact product
  r = fma(-kf, 1.3239129268154012e-11, r);
  double p = fma(r, 1.0 / 720.0, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r * r, r);
  const double2 t = __ldg(EXP2_32 + (k & 31));
  const double v = t.x + fma(t.x, p, t.y);   // in (0.98, 2)
  return __hiloint2double(__double2hiint(v) + ((k >> 5) << 20), __double2loint(v));
}

// tanh x = h / (h + 1), h = (e^2x - 1) / 2 = 2^(k/32) (e^2u - 1) / 2 + (2^(k/32)
// - 1) / 2 with x = k ln 2 / 64 + u, |u| < ln 2 / 128, without branches; the
// quotient by one Newton step from an FP32 seed and one correction, which
// takes what the roundings of e^2u - 1, h and h + 1 left off.  Thirty FP64
// instructions at every x, accurate relative to the value down to zero: at
// most 1.23 ulp over 15 million arguments, rms 0.29 (the library's tanh 1.45 and
// 0.32; without the low parts 2.5 and 0.46).
__device__ __forceinline__ double tanh_even(double x) {
  const long long bits = __double_as_longlong(x), mag = bits & 0x7fffffffffffffffLL;
  // beyond 22 tanh rounds to 1
  const double ax = __longlong_as_double(mag < 0x4036000000000000LL ? mag : 0x4036000000000000LL);
  const double magic = 6755399441055744.0;          // 1.5 * 2^52: rounds to an integer
  const double kd = fma(ax, 2.0 * 46.16624130844683, magic);
  const int k = __double2loint(kd);
  const double kf = kd - magic;
  double u = fma(-kf, 0.5 * 0.02166084937925916, ax);   // ln 2 / 64 to 31 bits: exact product
  u = fma(-kf, 0.5 * 1.3239129268154012e-11, u);
  double p = fma(u, 4.0 / 315.0, 2.0 / 45.0);
  p = fma(p, u, 2.0 / 15.0);
  p = fma(p, u, 1.0 / 3.0);
  p = fma(p, u, 2.0 / 3.0);
  p = fma(p, u, 1.0);
  const double c = p * u, ph = fma(c, u, u), pl = fma(c, u, u - ph);   // (e^2u - 1) / 2
  const double2 w = __ldg(EXP2_32 + (k & 31));
  const int up = (k >> 5) << 20, half = up - (1 << 20);
  const double t = __hiloint2double(__double2hiint(w.x) + up, __double2loint(w.x));
  const double th = __hiloint2double(__double2hiint(w.x) + half, __double2loint(w.x));
  const int tl_hi = __double2hiint(w.y);
  const double tl = __hiloint2double(tl_hi ? tl_hi + half : 0, __double2loint(w.y));   // (zero stays)
  const double a = th - 0.5, h = fma(t, ph, a);
  const double hl = fma(t, pl, fma(t, ph, a - h)) + tl;
  // h + 1 and its low part, from the larger of the two (h < 1 below k = 32 but
  // for a rounding)
  const double big = k < 32 ? 1.0 : h, small = k < 32 ? h : 1.0;
  const double d = h + 1.0, dl = small - (d - big);
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
  const double y = (double)f, inv = fma(y, fma(-d, y, 1.0), y);
  double q = h * inv;
  q = fma(fma(-q, d, h) + fma(-q, dl + hl, hl), inv, q);
  // sign, and NaN as it came
  const long long res = __double_as_longlong(q) | (bits & (long long)0x8000000000000000ULL);
  return __longlong_as_double(mag > 0x7ff0000000000000LL ? bits : res);
}
