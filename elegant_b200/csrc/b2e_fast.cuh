/*
 * Straight-line forms of the KQUAD/KSEXT and CSBEND maps for the particles
 * that stay well inside every limit, which is nearly all of them on nearly
 * every element.  Same expressions in the same order as kmult and csbend
 * (b2e_elements.cuh), bit for bit, with the divisions and square roots of
 * b2e_fp64.cuh, which share seeds and reciprocals and hold no branches.
 *
 * A form returns false, and leaves the particle untouched, when anything
 * leaves the range it was written for: an aperture (or a place too near its
 * edge to tell cheaply), a coordinate, slope or angle limit, a loss, a
 * non-finite or extremely small value.  The caller then runs the general map
 * from the element's entrance, which finds the loss or the value; a particle
 * pays for that once or twice in its life.  Range tests compare the high words of the doubles on
 * the integer pipe.
 *
 * Why: the general maps spend about 180 FP64-pipe operations per bend drift
 * substep and kick, half of them in five separate divisions and a square root,
 * each with its own range branch; these take about 85.
 */
#ifndef B2E_FAST_CUH
#define B2E_FAST_CUH
#include "b2e_elements.cuh"
#include "b2e_fp64.cuh"

/* high words of the limits */
#define FP_HI_2M250 0x30500000u
#define FP_HI_2M10 0x3f500000u
#define FP_HI_2M4 0x3fb00000u
#define FP_HI_2M3 0x3fc00000u
#define FP_HI_2 0x40000000u
#define FP_HI_2P4 0x40300000u
#define FP_HI_2P10 0x40900000u
#define FP_HI_2P100 0x46300000u
#define FP_HI_2P700 0x6bb00000u

/* v zero, or 2^-250 <= |v| below the value whose high word is `end`: products
 * and remainders of such values stay clear of the subnormal range */
__device__ __forceinline__ bool fp_plain(double v, unsigned end) {
  const unsigned h = fp_abs_hi(v);
  return h - FP_HI_2M250 < end - FP_HI_2M250 || (h | (unsigned)__double2loint(v)) == 0;
}

/* v in [value of lo, value of hi) by high words; negative and non-finite v are out */
__device__ __forceinline__ bool fp_within(double v, unsigned lo, unsigned hi) { return fp_hi(v) - lo < hi - lo; }

/* surely inside the aperture: (x/x_max)^2 + (y/y_max)^2 below 0.998 or so, a
 * half-axis that is not checked counting as infinite.  Rectangles contain that
 * ellipse, and so do the super-ellipses of exponents above 2.  False for
 * non-finite x or y. */
__device__ __forceinline__ bool ap_surely_inside(double x, double y, const DevAperture *ap) {
  const double u = x * ap->inv_x, v = y * ap->inv_y;
  return fp_abs_hi(fma(u, u, v * v)) < 0x3feff000u;
}

__device__ __forceinline__ bool ap_surely_inside(double x, double y, const DevAperture *ap, const DevElem &e) {
  if (e.flags & EF_REVERSE_TILT) {
    const double x0 = x, y0 = y;
    x = x0 * e.rev_cos + y0 * e.rev_sin;
    y = -x0 * e.rev_sin + y0 * e.rev_cos;
  }
  return ap_surely_inside(x, y, ap);
}

/* the exact test, out of line: only particles near or beyond the edge take it */
static __device__ __noinline__ bool ap_inside_exact(double x, double y, const DevAperture *ap, const DevElem *e) {
  return mult_aperture_ok(x, y, ap, *e);
}

__device__ __forceinline__ bool ap_inside(double x, double y, const DevAperture *ap, const DevElem &e) {
  return ap_surely_inside(x, y, ap, e) || ap_inside_exact(x, y, ap, &e);
}

/* offset_misalign with the square root only where dz uses it: zero times a
 * positive finite root is a zero of dz's sign */
__device__ __forceinline__ void offset_misalign_fast(Part &p, double dx, double dy, double dz) {
  const double r = dz == 0 ? 1.0 : fp_sqrt((1 + p.xp * p.xp) + p.yp * p.yp);
  p.s = p.s + dz * r;
  p.x = (p.x - dx) + dz * p.xp;
  p.y = (p.y - dy) + dz * p.yp;
}

/* entrance and exit limits of kmult (coordinates, slopes), and slopes below 2 */
__device__ __forceinline__ bool inside_limits(const Part &p, const DevGlobals &g) {
  const unsigned cl = min(fp_hi(g.coord_limit), FP_HI_2P100), sl = min(fp_hi(g.slope_limit), FP_HI_2);
  return fp_abs_hi(p.x) < cl && fp_abs_hi(p.y) < cl && fp_abs_hi(p.xp) < sl && fp_abs_hi(p.yp) < sl;
}

__device__ __forceinline__ bool plain_transverse(const Part &p) {
  return fp_plain(p.x, FP_HI_2P100) && fp_plain(p.y, FP_HI_2P100) && fp_plain(p.xp, FP_HI_2) && fp_plain(p.yp, FP_HI_2);
}

/* p/sqrt(p^2 + 1) */
__device__ __forceinline__ bool beta_fast(double p, double &beta) {
  double ir;
  const double r = fp_sqrt_recip(p * p + 1, ir);
  beta = fp_quot(p, r, ir);
  return fp_within(p, FP_HI_2M10, FP_HI_2P100);
}

/* ---- KQUAD / KSEXT without K1/J1, steering, fringes or quantum excitation
 * (EF_FAST).  The radiation block's round trip always runs (EF_RADBLOCK).  Per
 * kick: the round trip of the momenta through 1 + delta, one square root whose
 * reciprocal divides both momenta; per drift one square root.  SR adds the
 * classical radiation of each kick (kmult_radiation), with delta changing
 * inside the trip; rc: the element's DevRad constants. */
template <bool SR>
__device__ __forceinline__ bool kmult_fast(Part &pio, const DevElem &e, const DevAperture *ap, const DevGlobals &g,
                                           const double *rc) {
  const double *c = e.c;
  const int order = (int)c[KM_ORDER], nSlices = (int)c[KM_NSLICES], nSub = (int)c[KM_NSUB];
  const double dx = c[KM_DX], dy = c[KM_DY];
  Part p = pio;
  if (e.flags & EF_ENTRANCE_OFFSET)
    offset_misalign_fast(p, dx, dy, c[KM_DZ]);
  if (e.flags & EF_ENTRANCE_ROTATE)
    rotate_misalign(p, c[KM_COS_TILT], c[KM_SIN_TILT]);
  double dp = p.dp, A = 1 + dp, A2 = A * A, inv_A = fp_recip(A);
  bool ok = inside_limits(p, g) && plain_transverse(p) && fp_within(A, FP_HI_2M4, FP_HI_2P4);
  double x = p.x, xp = p.xp, y = p.y, yp = p.yp, s = 0, r, ir, d, qx, qy;
  r = fp_sqrt_recip((1 + xp * xp) + yp * yp, ir);
  qx = fp_quot(A * xp, r, ir);
  qy = fp_quot(A * yp, r, ir);
  d = (A2 - qx * qx) - qy * qy;
  r = fp_sqrt_recip(d, ir);
  ok = ok && fp_within(d, FP_HI_2M10, FP_HI_2P10);
  xp = fp_quot(qx, r, ir);
  yp = fp_quot(qy, r, ir);
  for (int i = 0; i < nSlices && ok; i++) {
    if (ap)
      ok = ap_inside(x + dx, y + dy, ap, e);
#pragma unroll 1
    for (int step = 0;; step++) {
      const double dsh = c[KM_DSH0 + step];
      x = x + xp * dsh;
      y = y + yp * dsh;
      s = s + dsh * fp_sqrt((1 + xp * xp) + yp * yp);
      if (step == nSub - 1)
        break;
      const double kick = c[KM_KICK0 + step];
      double fx, fy;
      if (order == 1) {
        fx = y;
        fy = x;
      } else {
        fx = x * y;
        fy = 0.5 * (x * x);
        fy = fy + -0.5 * (y * y);
      }
      const double kx = kick * fy, ky = kick * fx;
      qx = qx - kx;
      qy = qy + ky;
      if (SR) {
        /* slopes before the loss, the field squared from the kick over its
         * share of the slice, the loss, and the momenta scaled to the new
         * delta (zero kicks only enter squared, whatever their sign) */
        d = (A2 - qx * qx) - qy * qy;
        r = fp_sqrt_recip(d, ir);
        ok = ok && fp_within(d, FP_HI_2M10, FP_HI_2P10);
        xp = fp_quot(qx, r, ir);
        yp = fp_quot(qy, r, ir);
        const double share = rc[RK_KFRAC0 + step], drift = rc[RK_DRIFT];
        const double inv_share = fp_recip(share), inv_drift = fp_recip(drift);
        const double a = fp_quot(fp_quot(kx, share, inv_share), drift, inv_drift);
        const double b = fp_quot(fp_quot(ky, share, inv_share), drift, inv_drift);
        const double ds = fp_sqrt((1 + xp * xp) + yp * yp) * (drift * share);
        qx = fp_quot(qx, A, inv_A);
        qy = fp_quot(qy, A, inv_A);
        dp = dp - ((rc[RK_RAD] * A2) * (a * a + b * b)) * ds;
        A = 1 + dp;
        A2 = A * A;
        inv_A = fp_recip(A);
        ok = ok && fp_within(A, FP_HI_2M4, FP_HI_2P4);
        qx = qx * A;
        qy = qy * A;
      } else {
        qx = fp_quot(qx, A, inv_A) * A;
        qy = fp_quot(qy, A, inv_A) * A;
      }
      /* without radiation the test of the momenta before the round trip
       * differs from this one by rounding only, so it cannot fail where d is
       * 2^-10 or more */
      d = (A2 - qx * qx) - qy * qy;
      r = fp_sqrt_recip(d, ir);
      ok = ok && fp_within(d, FP_HI_2M10, FP_HI_2P10);
      xp = fp_quot(qx, r, ir);
      yp = fp_quot(qy, r, ir);
    }
  }
  if (!ok || (ap && !ap_inside(x + dx, y + dy, ap, e)))
    return false;
  /* the slopes are those of the last kick: the momenta have not changed since */
  p.x = x;
  p.xp = xp;
  p.y = y;
  p.yp = yp;
  if (SR) {
    /* path length at the changed velocity (multipole.c:1391-1394) */
    double beta0, beta1;
    if (!fp_plain(p.s, FP_HI_2P100) || !beta_fast(g.p_central * (1 + p.dp), beta0) ||
        !beta_fast(g.p_central * A, beta1))
      return false;
    const double both = beta0 + beta1;
    p.s = beta1 * (fp_quot(p.s, beta0, fp_recip(beta0)) + fp_quot(2 * s, both, fp_recip(both)));
    p.dp = dp;
  } else
    p.s = p.s + s;
  if (!inside_limits(p, g))
    return false;
  if (e.flags & EF_EXIT_MISALIGN) {
    if (e.flags & EF_ENTRANCE_ROTATE)
      rotate_misalign(p, c[KM_COS_TILT], -c[KM_SIN_TILT]);
    if (e.flags & EF_ENTRANCE_OFFSET)
      offset_misalign_fast(p, -dx, -dy, -c[KM_DZ]);
  }
  pio = p;
  return true;
}

/* sqrt((1 + delta)^2 - QY^2) of the bend drift and its reciprocal */
__device__ __forceinline__ bool bend_root(double A, double QY, double &f, double &inv_f) {
  const double d = A * A - QY * QY;
  f = fp_sqrt_recip(d, inv_f);
  return fp_within(d, FP_HI_2M10, FP_HI_2P10);
}

/* The series of b2e_asin (to n = 4 for |x| <= 2^-6, else to n = 10), b2e_sin and
 * b2e_cos (short for |x| <= 2^-4, else long), where the long ones enter the
 * short ones' Horner chains: the same operations, with the branch around the
 * high-order terms only.  The coefficients are operands from constant memory;
 * as literals each costs two moves in front of its fma. */
static __constant__ double kAsinSeries[10] = {
  (2.0 / 3.0) * 0x1p-2,       (6.0 / 5.0) * 0x1p-4,      (20.0 / 7.0) * 0x1p-6,    (70.0 / 9.0) * 0x1p-8,
  (252.0 / 11.0) * 0x1p-10,   (924.0 / 13.0) * 0x1p-12,  (3432.0 / 15.0) * 0x1p-14, (12870.0 / 17.0) * 0x1p-16,
  (48620.0 / 19.0) * 0x1p-18, (184756.0 / 21.0) * 0x1p-20};
static __constant__ double kSinSeries[9] = { /* -1/3!, 1/5!, ..., -1/19! */
  -1.0 / 6.0, 1.0 / 120.0, -1.0 / 5040.0, 1.0 / 362880.0, -1.0 / 39916800.0, 1.0 / 6227020800.0,
  -1.0 / 1307674368000.0, 1.0 / 355687428096000.0, -1.0 / 121645100408832000.0};
static __constant__ double kCosSeries[9] = { /* 1/4!, -1/6!, ..., 1/20! */
  1.0 / 24.0, -1.0 / 720.0, 1.0 / 40320.0, -1.0 / 3628800.0, 1.0 / 479001600.0, -1.0 / 87178291200.0,
  1.0 / 20922789888000.0, -1.0 / 6402373705728000.0, 1.0 / 2432902008176640000.0};

__device__ __forceinline__ double asin_series(double x, bool tiny) {
  const double w = x * x;
  double p = kAsinSeries[3];
  if (!tiny) {
    double q = kAsinSeries[9];
#pragma unroll
    for (int k = 8; k >= 4; k--)
      q = fma(q, w, kAsinSeries[k]);
    p = fma(q, w, kAsinSeries[3]);
  }
#pragma unroll
  for (int k = 2; k >= 0; k--)
    p = fma(p, w, kAsinSeries[k]);
  return fma(x * w, p, x);
}

/* the high-order terms of both, which enter the Horner chains below in the
 * place of their leading coefficients */
__device__ __forceinline__ double sin_prefix(double w) {
  double q = kSinSeries[8];
#pragma unroll
  for (int k = 7; k >= 3; k--)
    q = fma(q, w, kSinSeries[k]);
  return q;
}
__device__ __forceinline__ double cos_prefix(double w) {
  double q = kCosSeries[8];
#pragma unroll
  for (int k = 7; k >= 2; k--)
    q = fma(q, w, kCosSeries[k]);
  return q;
}

__device__ __forceinline__ double sin_tail(double r, double w, double p) {
#pragma unroll
  for (int k = 2; k >= 0; k--)
    p = fma(p, w, kSinSeries[k]);
  return fma(r * w, p, r);
}

/* 0.5 w is exact, so the two differences with it are one fma each */
__device__ __forceinline__ double cos_tail(double w, double p) {
  p = fma(p, w, kCosSeries[1]);
  p = fma(p, w, kCosSeries[0]);
  const double t = fma(-0.5, w, 1.0);
  return t + (fma(-0.5, w, 1.0 - t) + (w * w) * p);
}

/* |v| <= limit, on the integer pipe (NaN is above every limit) */
__device__ __forceinline__ bool abs_at_most(double v, double limit) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) <= __double_as_longlong(limit);
}

/* drift substep (bend_drift): f and inv_f as bend_root leaves them.  sin_max
 * collects the high word of the largest |sin phi|, for one test per element:
 * below 1/8 the series hold, and with the slice angles EF_FAST admits |arg| is
 * below pi/4. */
__device__ __forceinline__ void bend_drift_fast(double &X, double &QX, double &Y, double QY, double &dist, double A,
                                                double f, double inv_f, double rho0, double dsh_rho0,
                                                unsigned &sin_max) {
  const double sin_phi = fp_quot(QX, f, inv_f);
  sin_max = max(sin_max, fp_abs_hi(sin_phi));
  const double phi = asin_series(sin_phi, abs_at_most(sin_phi, 0x1p-6)), arg = dsh_rho0 + phi;
  const double wa = arg * arg, wp = phi * phi;
  double ps = kSinSeries[3], pc = kCosSeries[2], pp = kCosSeries[2];
  const bool small = abs_at_most(arg, 0x1p-4), small_phi = abs_at_most(phi, 0x1p-4);
  if (!(small && small_phi)) { /* one branch for the three series */
    ps = small ? ps : sin_prefix(wa);
    pc = small ? pc : cos_prefix(wa);
    pp = small_phi ? pp : cos_prefix(wp);
  }
  const double sine = sin_tail(arg, wa, ps), cosi = cos_tail(wa, pc), cos_phi = cos_tail(wp, pp);
  const double ic = fp_recip(cosi), ip = fp_recip(cos_phi);
  const double tang = fp_quot(sine, cosi, ic), ratio = fp_quot(cos_phi, cosi, ic);
  const double factor = fp_quot((rho0 + X) * cos_phi, f, inv_f) * (tang - fp_quot(sin_phi, cos_phi, ip));
  QX = f * sine;
  Y = Y + QY * factor;
  dist = dist + factor * A;
  X = rho0 * (ratio - 1) + ratio * X;
}

/* nSlices slices of the bend (csbend_integrate without field terms).  QY changes
 * only by rounding, in the round trip through 1 + delta after a kick (TRIP), and
 * stays put from the first trip that leaves it alone: the trip depends on
 * nothing else.  So its trips stop there, and f and 1/f are formed again only
 * while it moves.  With radiation (TRIP_SR; rad_coef in rad, 1/rho0 as the
 * radiation's formulas take it in inv_rho) delta changes inside every trip, and
 * A, 1/A and f with it. */
enum BendTrip { TRIP_NONE, TRIP, TRIP_SR };
template <BendTrip MODE>
__device__ __forceinline__ bool bend_slices_fast(double &X, double &QX, double &Y, double &QY, double &dist, double &A,
                                                 double inv_A, const double *c, int nSlices, int nSub,
                                                 const DevAperture *ap, const DevElem &e, double *delta = nullptr,
                                                 double rad = 0, double inv_rho = 0) {
  const double rho0 = c[CB_RHO0];
  double f, inv_f, DP = MODE == TRIP_SR ? *delta : 0;
  unsigned sin_max = 0;
  bool ok = bend_root(A, QY, f, inv_f), moves = MODE == TRIP;
  dist = 0;
  for (int i = 0; i < nSlices && ok; i++) {
    if (ap)
      ok = ap_inside(X, Y, ap, e);
#pragma unroll 1
    for (int j = 0;; j++) {
      bend_drift_fast(X, QX, Y, QY, dist, A, f, inv_f, rho0, c[CB_DSH0 + j], sin_max);
      if (j == nSub - 1)
        break;
      const double ds = c[CB_DS0 + j], t = (-ds) * (1 + fp_quot(X, rho0, c[CB_INV_RHO0]));
      QX = QX + fp_quot(t, c[CB_RHO_ACTUAL], c[CB_INV_RHO_ACTUAL]);
      if (MODE == TRIP) {
        QX = fp_quot(QX, A, inv_A) * A;
        if (moves) {
          const double q = fp_quot(QY, A, inv_A) * A;
          moves = q != QY;
          if (moves) {
            QY = q;
            ok = bend_root(A, QY, f, inv_f) && ok;
          }
        }
      } else if (MODE == TRIP_SR) {
        /* radiation after the kick (csbend.c:1603-1622) in the dipole field, F2 = 1 */
        const double a = 1 + X * inv_rho, A2 = A * A, d = (A2 - QX * QX) - QY * QY;
        double ir;
        const double r = fp_sqrt_recip(d, ir), g = fp_quot(a, r, ir);
        const double xp = QX * g, yp = QY * g, m = (a * a + xp * xp) + yp * yp;
        ok = ok && fp_within(d, FP_HI_2M10, FP_HI_2P10) && fp_within(m, FP_HI_2M10, FP_HI_2P10);
        QX = fp_quot(QX, A, inv_A);
        QY = fp_quot(QY, A, inv_A);
        DP = DP - ((rad * A2) * ds) * fp_sqrt(m);
        A = 1 + DP;
        inv_A = fp_recip(A);
        QX = QX * A;
        QY = QY * A;
        ok = bend_root(A, QY, f, inv_f) && ok && fp_within(A, FP_HI_2M4, FP_HI_2P4);
      }
    }
  }
  if (MODE == TRIP_SR)
    *delta = DP;
  return ok && sin_max < FP_HI_2M3 && (!ap || ap_inside(X, Y, ap, e));
}

/* first-order edge with nonzero angles or fringe (csbend), out of line */
struct EdgeSlopes {
  double xp, yp;
};
static __device__ __noinline__ EdgeSlopes bend_edge_o1(double xp, double yp, double x, double y, double dp, double rho_actual,
                                                       const double *tan_e) {
  /* tan_e: CB_TAN_E, CB_E, CB_PSI of one face, in that order */
  const double rho = (1 + dp) * rho_actual, delta_xp = (tan_e[0] / rho) * x;
  EdgeSlopes r;
  r.xp = xp + delta_xp;
  r.yp = yp - (b2e_tan(tan_e[1] - tan_e[2] / (1 + dp)) / rho) * y;
  return r;
}

/* ---- CSBEND without field terms, ETILT, second-order or simple edges and
 * quantum excitation (EF_FAST); with SR, classical radiation in the body and
 * none at the edges, whose angles are zero; rc: the element's DevRad constants */
template <bool SR>
__device__ __forceinline__ bool csbend_fast(Part &pio, const DevElem &e, const DevAperture *ap, const DevGlobals &g,
                                            const double *rc) {
  const double *c = e.c;
  const double ct = c[CB_COS_TT], st = c[CB_SIN_TT];
  Part p = pio;
  double x, y, xp, yp, s, Q4, r, ir, f, A = 1 + p.dp;
  const double inv_A = fp_recip(A);
  bool ok = plain_transverse(p) && fp_plain(p.s, FP_HI_2P100) && fp_within(A, FP_HI_2M4, FP_HI_2P4);
  s = p.s + c[CB_DZI] * (c[CB_DZI] == 0 ? 1.0 : fp_sqrt((1 + p.xp * p.xp) + p.yp * p.yp));
  p.x = (p.x + c[CB_DXI]) + c[CB_DZI] * p.xp;
  p.y = (p.y + c[CB_DYI]) + c[CB_DZI] * p.yp;
  x = p.x * ct + p.y * st;
  y = -p.x * st + p.y * ct;
  xp = p.xp * ct + p.yp * st;
  yp = -p.xp * st + p.yp * ct;
  if (e.flags & EF_EDGE1) {
    if (e.flags & EF_EDGE1_FLAT) {
      /* no edge angle, no fringe: the zeros that the divisions by rho give */
      const double rho = A * c[CB_RHO_ACTUAL], z = c[CB_TAN_E1] * rho;
      xp = xp + z * x;
      yp = yp - z * y;
    } else {
      const EdgeSlopes es = bend_edge_o1(xp, yp, x, y, p.dp, c[CB_RHO_ACTUAL], c + CB_TAN_E1);
      xp = es.xp;
      yp = es.yp;
    }
  }
  r = fp_sqrt_recip((1 + xp * xp) + yp * yp, ir);
  ok = ok && fp_plain(xp, FP_HI_2) && fp_plain(yp, FP_HI_2);
  f = fp_quot(A, r, ir);
  xp = xp * f;
  yp = yp * f;
  /* a kick adds a zero to QY, which a negative zero would not survive */
  ok = ok && fp_hi(yp) != 0x80000000u;
  if (!ok)
    return false;
  double dp = p.dp;
  if (!(SR ? bend_slices_fast<TRIP_SR>(x, xp, y, yp, Q4, A, inv_A, c, (int)c[CB_NSLICES], (int)c[CB_NSUB], ap, e, &dp,
                                       rc[RB_RAD], rc[RB_INV_RHO0])
           : bend_slices_fast<TRIP>(x, xp, y, yp, Q4, A, inv_A, c, (int)c[CB_NSLICES], (int)c[CB_NSUB], ap, e)))
    return false;
  {
    const double d = (A * A - xp * xp) - yp * yp;
    r = fp_sqrt_recip(d, ir);
    ok = fp_within(d, FP_HI_2M10, FP_HI_2P10);
  }
  f = fp_quot(1.0, r, ir);
  xp = xp * f;
  yp = yp * f;
  {
    /* time-of-flight velocity fix (csbend.c:1278-1288); without radiation the
     * exit velocity is the entrance's, and beta s / beta rounds twice */
    double beta0, beta1;
    ok = beta_fast(g.p_central * (1 + p.dp), beta0) && ok;
    beta1 = beta0;
    if (SR)
      ok = beta_fast(g.p_central * A, beta1) && ok;
    s = fp_quot(beta1 * s, beta0, fp_recip(beta0)) + Q4;
  }
  if (e.flags & EF_EDGE2) {
    if (e.flags & EF_EDGE2_FLAT) {
      const double rho = A * c[CB_RHO_ACTUAL], z = c[CB_TAN_E2] * rho;
      xp = xp + z * x;
      yp = yp - z * y;
    } else {
      const EdgeSlopes es = bend_edge_o1(xp, yp, x, y, dp, c[CB_RHO_ACTUAL], c + CB_TAN_E2);
      xp = es.xp;
      yp = es.yp;
    }
  }
  p.x = (x * ct - y * st) + 0.0;
  p.y = (x * st + y * ct) + 0.0;
  p.xp = (xp * ct - yp * st) + 0.0;
  p.yp = (xp * st + yp * ct) + 0.0;
  p.s = s + 0.0;
  p.dp = dp;
  ok = ok && fp_abs_hi(p.xp) < FP_HI_2 && fp_abs_hi(p.yp) < FP_HI_2;
  p.x = p.x + (c[CB_DXF] + c[CB_DZF] * p.xp);
  p.y = p.y + (c[CB_DYF] + c[CB_DZF] * p.yp);
  p.s = p.s + c[CB_DZF] * (c[CB_DZF] == 0 ? 1.0 : fp_sqrt((1 + p.xp * p.xp) + p.yp * p.yp));
  if (!ok)
    return false;
  pio = p;
  return true;
}

/* The general maps out of line, for elements or particles the forms above do
 * not take.  The particle travels in a local copy, so that the caller's stays
 * in registers on the other path. */
template <bool RAD>
static __device__ __noinline__ int kmult_call(Part *p, const DevElem *e, const DevAperture *ap, DevGlobals g,
                                              const RadSite *rs) {
  return kmult<RAD>(*p, *e, ap, g, *rs);
}
template <bool RAD>
__device__ __forceinline__ int kmult_general(Part &p, const DevElem &e, const DevAperture *ap, const DevGlobals &g,
                                             const RadSite &rs) {
  Part t = p;
  const RadSite site = rs;
  const int lost = kmult_call<RAD>(&t, &e, ap, g, &site);
  p = t;
  return lost;
}
template <bool RAD>
static __device__ __noinline__ int csbend_call(Part *p, const DevElem *e, const DevAperture *ap, DevGlobals g,
                                               const RadSite *rs) {
  return csbend<RAD>(*p, *e, ap, g, *rs);
}
template <bool RAD>
__device__ __forceinline__ int csbend_general(Part &p, const DevElem &e, const DevAperture *ap, const DevGlobals &g,
                                              const RadSite &rs) {
  Part t = p;
  const RadSite site = rs;
  const int lost = csbend_call<RAD>(&t, &e, ap, g, &site);
  p = t;
  return lost;
}

#endif
