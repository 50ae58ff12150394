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
 * a - q b exact under fma, RN(q + r y) (the same paper).
 *
 * Why the roundings are right, with b in [1, 2) for the significand of a divisor:
 *
 * Reciprocal, fp_polish.  y (2 - b y) is (1/b)(1 - e^2) before the last rounding,
 * e the relative error of y; it rounds to RN(1/b) unless a midpoint lies within
 * e^2/b below 1/b.  For b = B 2^-52 and a midpoint M 2^-54 (M odd) the distance is
 * k 2^-106/b with k = 2^106 - M B odd, so with e below sqrt(3) 2^-53 only k = 1
 * remains, and the only divisor of 2^106 - 1 = 3 107 6361 69431 20394401
 * 28059810762433 in [2^52, 2^53) is 2^53 - 1, the significand of all ones, which
 * fp_fix sets.
 *
 * Reciprocal, fp_recip.  The series is short of e^4 and its sum rounds at
 * 2^-53 e, e at most 2^-19 of the seed, so y is within 0.5 + 2^-20 ulp of 1/b: not
 * always RN(1/b): six divisors in 1e8 have its neighbour.
 *
 * Quotient.  With y = (1/b)(1 + e) the last fma rounds a/b - (q - a/b) e.  Let a/b
 * (a in [1, 2) too) lie next to a midpoint: its distance is |k| 2^-105/b for a >= b,
 * |k| 2^-106/b for a < b, k an integer other than 0, and half an ulp is 2^-53 or
 * 2^-54.  |e| is at most 2^-54 b (1 + 2^-19).  For b below 2 - 2^-18 q is one of the
 * midpoint's neighbours, half an ulp away, and a wrong rounding would take |e| >=
 * |k| 2^-52/b, which is more.  Above, q can be the next one to it, three halves
 * away, so |k| up to 3 comes into question: at most ten numerators per divisor,
 * and b2e_selftest_quotient divides them all.
 *
 * Square root: with g next to the midpoint the remainder is an integer multiple
 * of ulp(g)^2, and a relative error of the factor 1/(2g) below 1.5 2^-53 (here at
 * most 1.32) cannot move it across the rounding boundary.
 *
 * b2e_selftest_rounding and b2e_selftest_quotient compare fp_polish, the quotients
 * and the square roots with the IEEE operators on the device.
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

/* RN(1/b) from y within sqrt(3) 2^-53 of it, relative */
__device__ __forceinline__ double fp_polish(double b, double y) { return fp_fix(b, fma(fma(-b, y, 1.0), y, y)); }

/* 1/b within 0.5 + 2^-20 ulp, enough for fp_quot: four operations behind the seed */
__device__ __forceinline__ double fp_recip(double b) {
  const double y0 = fp_rcp_seed(b), e = fma(-b, y0, 1.0), p = fma(e, e, e);
  return fp_fix(b, fma(y0, fma(p, e, e), y0));
}

/* RN(a/b), b > 0, from y = RN(1/b) or fp_recip(b).  The remainder is formed with its sign turned
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
