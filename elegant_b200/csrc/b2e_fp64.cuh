/*
 * Correctly rounded FP64 reciprocal, quotient and square root for operands in
 * a known range, built so that what one result iterates on serves the next.
 *
 * The element maps divide several numerators by one divisor (both slopes by
 * the longitudinal momentum, four quotients by cos or by f in a bend substep)
 * and take a square root whose reciprocal is the next divisor.  The IEEE
 * operators cost each of those a seed, an iteration, a range test and a branch
 * of its own; here a square root and its reciprocal share one seed and one
 * iteration, and every further quotient by the same divisor is three
 * operations.  No range test is inside: the callers keep divisors within
 * [2^-200, 2^200] and numerators zero or at least 2^-900 in magnitude.
 *
 * Method.  Seeds are the PTX approximations rcp.approx.ftz.f64 and
 * rsqrt.approx.ftz.f64 (21 significant bits; documented in the PTX ISA).
 * Reciprocal: y = y0 (1 + e + e^2 + e^3) with e = 1 - b y0, which is exact (53 x
 * 21 bits).  Square root: the third-order iteration of the binomial series of
 * (1 - e)^(-1/2), applied to D y0 for the root and to y0 for its reciprocal,
 * then Markstein's correction g + (D - g^2)/(2g) with an exact remainder
 * (P. Markstein, IBM J. Res. Dev. 34, 1990).  Quotient: q = RN(a y), remainder
 * a - q b exact under fma, RN(q + r y), with y = RN(1/b) (the same paper).
 *
 * Why the roundings are right.  Quotient: with y = RN(1/b) the last step
 * returns RN(a/b) for every a (the same paper); a result can round wrongly only
 * where a/b lies within |r| |y - 1/b| of a midpoint, q is then one of the two
 * neighbours, and half an ulp times the relative error of y is below the
 * smallest distance a quotient can have from a midpoint.  The iterations give
 * RN(1/b) but for the significand just below 2 (1/b a hair above a midpoint),
 * which fp_fix sets.  Square root: with g next to the midpoint the remainder is
 * an integer multiple of ulp(g)^2, and a relative error of the factor 1/(2g)
 * below 1.5 2^-53 (here at most 1.32) cannot move it across the rounding
 * boundary.  b2e_selftest_rounding compares all of them with the IEEE
 * operators on the device.
 */
#ifndef B2E_FP64_CUH
#define B2E_FP64_CUH

__device__ __forceinline__ unsigned fp_hi(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ unsigned fp_abs_hi(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }

/* v / 2 and 2 v of a normal number, on the integer pipe */
__device__ __forceinline__ double fp_halve(double v) {
  return __hiloint2double(__double2hiint(v) - 0x00100000, __double2loint(v));
}
__device__ __forceinline__ double fp_twice(double v) {
  return __hiloint2double(__double2hiint(v) + 0x00100000, __double2loint(v));
}

/* RN(1/b) from y, which is that or, for a significand of all ones, may be the
 * power of two below it: 1/(2^e (1 - 2^-53)) rounds to 2^-e (1 + 2^-52) */
__device__ __forceinline__ double fp_fix(double b, double y) {
  const unsigned ones = (fp_hi(b) | 0xfff00000u) & (unsigned)__double2loint(b);
  return __hiloint2double(__double2hiint(y), ones == 0xffffffffu ? 1 : __double2loint(y));
}

__device__ __forceinline__ double fp_rcp_seed(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
__device__ __forceinline__ double fp_rsqrt_seed(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  return y;
}

/* RN(1/b) from y within two ulp of it */
__device__ __forceinline__ double fp_polish(double b, double y) { return fp_fix(b, fma(fma(-b, y, 1.0), y, y)); }

/* RN(1/b): four operations behind the seed */
__device__ __forceinline__ double fp_recip(double b) {
  const double y0 = fp_rcp_seed(b), e = fma(-b, y0, 1.0), p = fma(e, e, e);
  return fp_fix(b, fma(y0, fma(p, e, e), y0));
}

/* RN(a/b) from y = 1/b, b > 0.  The remainder is formed with its sign turned
 * over, so that an exact quotient adds a zero of the opposite sign to q and
 * keeps q, signed zeros included. */
__device__ __forceinline__ double fp_quot(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(q, b, -a), -y, q);
}

/* RN(sqrt(d)); h is half its reciprocal to 1.32 2^-53 */
__device__ __forceinline__ double fp_sqrt_half(double d, double &h) {
  const double y0 = fp_rsqrt_seed(d), t = d * y0, e = fma(-t, y0, 1.0), q = fma(e, 0.375, 0.5) * e;
  const double g = fma(t, q, t), y0h = fp_halve(y0);
  h = fma(y0h, q, y0h);
  return fma(fma(-g, g, d), h, g);
}

__device__ __forceinline__ double fp_sqrt(double d) {
  double h;
  return fp_sqrt_half(d, h);
}

/* RN(sqrt(d)) and the reciprocal of that root */
__device__ __forceinline__ double fp_sqrt_recip(double d, double &y) {
  double h;
  const double s = fp_sqrt_half(d, h);
  y = fp_polish(s, fp_twice(h));
  return s;
}

#endif
