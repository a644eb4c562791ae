/*
 * pgdg_math.cuh -- scalar arithmetic of the device path.
 *
 * Exact-order helpers (root_d, eos, Hugoniot, MGFM) use explicit round-to-nearest
 * intrinsics on the device so the compiler cannot contract them into FMAs; the
 * split/merge translation unit relies on this to reproduce the oracle's FP64
 * results bit for bit.  Templated helpers (kernel functions, EOS in R) are for
 * the stage kernels, where FMA contraction is allowed.
 */
#ifndef PGDG_MATH_CUH
#define PGDG_MATH_CUH

#include <cstdint>
#include <cmath>

#ifdef __CUDACC__
#define PGDG_HD __host__ __device__ __forceinline__
#else
#define PGDG_HD inline
#endif

namespace pgdg {

constexpr double PI_REF = 3.1415926;  /* glbparam.h:36 */
constexpr double CELL_RATIO = 3.2;    /* glbparam.h:31 */
constexpr double CUT_OFF = 2.;        /* glbparam.h:32 */

/* ---------------- exact-order FP64 operations ---------------- */
#if defined(__CUDA_ARCH__)
PGDG_HD double dadd(double a, double b) { return __dadd_rn(a, b); }
PGDG_HD double dsub(double a, double b) { return __dsub_rn(a, b); }
PGDG_HD double dmul(double a, double b) { return __dmul_rn(a, b); }
PGDG_HD double ddiv(double a, double b) { return __ddiv_rn(a, b); }
PGDG_HD double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }
PGDG_HD double dsqrt(double a) { return __dsqrt_rn(a); }
#else
PGDG_HD double dadd(double a, double b) { volatile double r = a + b; return r; }
PGDG_HD double dsub(double a, double b) { volatile double r = a - b; return r; }
PGDG_HD double dmul(double a, double b) { volatile double r = a * b; return r; }
PGDG_HD double ddiv(double a, double b) { volatile double r = a / b; return r; }
PGDG_HD double dfma(double a, double b, double c) { return std::fma(a, b, c); }
PGDG_HD double dsqrt(double a) { return std::sqrt(a); }
#endif

PGDG_HD double powern_d(double a, int n) {
  double r = 1;
  for (int i = 0; i < n; i++) r = dmul(r, a);
  return r;
}

/* deterministic ln(x) (atanh series), accurate to ~1e-17 relative */
PGDG_HD double det_log(double x) {
  int e;
  double m = frexp(x, &e);
  if (m < 0.70710678118654752) { m = dmul(m, 2.0); e -= 1; }
  double t = ddiv(dsub(m, 1.0), dadd(m, 1.0));
  double t2 = dmul(t, t);
  double s = 0.0;
  for (int k = 23; k >= 3; k -= 2) s = dmul(dadd(s, ddiv(1.0, (double)k)), t2);
  s = dmul(dadd(s, 1.0), t);
  return dadd(dmul(2.0, s), dmul((double)e, 0.69314718055994531));
}

/* x^(1/d) as the reference's pow(x, 1./DIM): sqrt for d == 2; for d == 3 the
 * exponent is the double 1/3 - 1/(3*2^54), so the value is
 * cbrt(x) * x^(-1/(3*2^54)), refined in double-double before one final rounding.
 * Independent restatement of the oracle's root_d; tests hold the two equal. */
PGDG_HD double root_d(double x, int d) {
  if (d == 2) return dsqrt(x);
  if (!(x > 0.0) || isinf(x)) return pow(x, 1.0 / 3.0);
  double y0 = cbrt(x);
  double p = dmul(y0, y0);
  double pl = dfma(y0, y0, -p);
  double q = dmul(p, y0);
  double ql = dfma(p, y0, -q);
  ql = dadd(ql, dmul(pl, y0));
  double r = dadd(dsub(q, x), ql);
  double delta = ddiv(r, dmul(3.0, p));
  double eps_l = dmul(det_log(x), 1.8503717077085943e-17);
  double corr = dmul(y0, eps_l);
  double small = dsub(-delta, corr);
  return dadd(y0, small);
}

PGDG_HD double amax1(double a, double b) { return a >= b ? a : b; }
PGDG_HD double amin1(double a, double b) { return a <= b ? a : b; }
PGDG_HD float amax1(float a, float b) { return a >= b ? a : b; }
PGDG_HD float amin1(float a, float b) { return a <= b ? a : b; }

/* EOS (mpm.cpp:859-876), exact order */
PGDG_HD double eos_p_x(double ee, double g, double pinf) { return dsub(dmul(ee, dsub(g, 1)), dmul(g, pinf)); }

/* ---------------- templated stage arithmetic ---------------- */
template <typename R>
PGDG_HD R eos_p(R ee, R g, R pinf) { return ee * (g - R(1)) - g * pinf; }
template <typename R>
PGDG_HD R eos_rhoe(R p, R g, R pinf) { return (p + g * pinf) / (g - R(1)); }

/* quotient of the stage arithmetic: the FP32 path uses the fast division
 * (within 2 ulp for divisors of normal magnitude), every other build the IEEE
 * division, so the exact path is unchanged */
template <typename R, bool EX>
__device__ __forceinline__ R qdiv(R a, R b) {
  if constexpr (!EX && sizeof(R) == 4) return __fdividef(a, b);
  else return a / b;
}

template <typename R>
PGDG_HD R sqrt_r(R x);
template <>
PGDG_HD double sqrt_r<double>(double x) { return sqrt(x); }
template <>
PGDG_HD float sqrt_r<float>(float x) { return sqrtf(x); }

/* Wendland C4 normalisation C(h) (particle.cpp:139-141) */
template <typename R>
PGDG_HD R wendland_C(R h, int d) {
  R hh = (d == 2) ? h * h : h * h * h;
  return (d == 2) ? R(1.0 / PI_REF) / hh * R(7. / 4.) : R(1.0 / PI_REF) / hh * R(21. / 16.);
}

/* ---------------- MGFM (FP64, exact order) ---------------- */
PGDG_HD double rhols_cal(double rhol, double pl, double ps, double g, double pinf) {
  double vn = dadd(dadd(dmul(dadd(g, 1), ps), dmul(dsub(g, 1), pl)), dmul(dmul(2, g), pinf));
  double vd = dadd(dadd(dmul(dsub(g, 1), ps), dmul(dadd(g, 1), pl)), dmul(dmul(2, g), pinf));
  return ddiv(dmul(rhol, vn), vd);
}
PGDG_HD double wl_cal(double rhol, double pl, double ps, double g, double pinf) {
  double in = dadd(dadd(dmul(dadd(g, 1.0), ps), dmul(dsub(g, 1.0), pl)), dmul(dmul(2.0, g), pinf));
  return dsqrt(dmul(dmul(0.5, rhol), in));
}
/* 1 / b correctly rounded */
PGDG_HD double drcp(double b) {
#if defined(__CUDA_ARCH__)
  return __drcp_rn(b);
#else
  return ddiv(1.0, b);
#endif
}
/* a / b correctly rounded, given y = 1 / b correctly rounded: a quotient from y,
 * corrected twice by its exact remainder (Markstein, IBM J. Res. Dev. 34, 1990:
 * with y correctly rounded and a quotient within one unit in the last place, the
 * corrected quotient is the correctly rounded one).  5 FP64 instructions where
 * a division is about 10 and the FP64 pipe sets the pace.  Outside exponents
 * that keep every step normal, for b <= 0, and for a = -0 (whose remainder +0 would
 * turn it into +0), the division itself. */
PGDG_HD double ddiv_by(double a, double b, double y) {
#if defined(__CUDA_ARCH__)
  const int ha = __double2hiint(a);
  const unsigned ea = ((unsigned)ha & 0x7fffffffu) >> 20, eb = (unsigned)__double2hiint(b) >> 20;
  if ((ea - 400u < 1200u || (ha | __double2loint(a)) == 0) && eb - 600u < 800u) { /* a sign bit in b fails the range too */
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
  }
#endif
  return ddiv(a, b);
}

/* d/dp of (p - p0) / W(p), with d = p - p0 and y = 1 / W; d / W^2 rho (g + 1) / 4 / W
 * keeps the reference's order (the quarter is exact) */
PGDG_HD double jaco_cal(double W, double y, double d, double rhol, double g) {
  double t = ddiv(d, dmul(W, W));
  t = dmul(t, rhol);
  t = dmul(t, dadd(g, 1));
  t = dmul(t, 0.25);
  t = ddiv_by(t, W, y);
  return dsub(y, t);
}

/* Two-shock Newton solve; variant 0 = mpm.cpp:882-926, 1 = Triple_point_2phase/
 * mpm.cpp:1373-1416.  seed_p > 0 replaces the initial p*.  Returns iterations.
 *
 * A problem without a positive root: f(p) = u_l - u_r - (p - p_l) / W_l -
 * (p - p_r) / W_r falls and is convex, so f(1e-8) >= f(p) + |f'(p)| (p - 1e-8).  With
 * f(1e-8) < 0 Newton's step |f / f'| is longer than p - 1e-8, so the cap 0.6 p decides
 * it for every p > 2.5e-8; and |f(p)| >= |f(1e-8)|, so with f(1e-8) below the
 * tolerance no iterate on the way converges.  The iterates down to 4e-8 are then
 * p - 0.6 p, two operations in place of about 130, and the rest runs as usual: the
 * same bits and counts.  descent = 1 looks for this at once (the caller knows
 * that f(1e-8) < 0), 0 after two capped steps downwards. */
PGDG_HD int mgfm(double ul, double ur, double pl, double pr, double rhol, double rhor, double gl,
                 double pinfl, double gr, double pinfr, int variant, double seed_p, double out[3], int descent = 0) {
  double pstar;
  if (variant == 0) {
    pl = amax1(pl, 1e-10);
    pr = amax1(pr, 1e-10);
    rhol = amax1(rhol, 1e-10);
    rhor = amax1(rhor, 1e-10);
    pstar = amax1(pl, pr);
  } else {
    if (pl < 0) pl = 0;
    if (pr < 0) pr = 0;
    pstar = dmul(dadd(pl, pr), 0.5);
  }
  if (seed_p > 0) pstar = seed_p;
  const double du = dsub(ul, ur);
  const double tol = amax1(1e-8, dmul(1e-3, fabs(du)));
  double f1 = 1., Wl = 0, ql = 0, pold = pstar, usl;
  int nn = 0, down = descent ? 2 : 0;
  do {
    if (down == 2) {
      down = 3; /* looked at once */
      /* the convexity above holds for these; the margins cover the rounding of f */
      if (pstar > 4e-8 && pstar < 1e100 && rhol > 0 && rhor > 0 && gl > 1 && gr > 1 && pinfl >= 0 && pinfr >= 0) {
        const double f0 = dsub(dsub(du, ddiv(dsub(1e-8, pl), wl_cal(rhol, pl, 1e-8, gl, pinfl))),
                               ddiv(dsub(1e-8, pr), wl_cal(rhor, pr, 1e-8, gr, pinfr)));
        if (f0 < dmul(-1.001, tol) && f0 > -1e100)
          while (pstar > 4e-8 && nn < 48) {
            pstar = dsub(pstar, dmul(0.6, pstar));
            nn++;
          }
      }
    }
    Wl = wl_cal(rhol, pl, pstar, gl, pinfl);
    const double Wr = wl_cal(rhor, pr, pstar, gr, pinfr);
    const double yl = drcp(Wl), yr = drcp(Wr), dl = dsub(pstar, pl), dr = dsub(pstar, pr);
    ql = ddiv_by(dl, Wl, yl);
    f1 = dsub(dsub(du, ql), ddiv_by(dr, Wr, yr));
    const double jac = dsub(-jaco_cal(Wl, yl, dl, rhol, gl), jaco_cal(Wr, yr, dr, rhor, gr));
    double dp = ddiv(-f1, jac);
    const double cap = dmul(0.6, pstar);
    if (fabs(dp) > cap) {
      dp = copysign(cap, dp);
      if (dp < 0 && down < 2) down++;
    }
    pold = pstar;
    pstar = dadd(pstar, dp);
    pstar = amax1(pstar, 1e-8);
    nn++;
    /* every quantity of an iteration is a function of pstar alone: once an
     * unconverged iterate repeats (the 1e-8 floor of a problem without a
     * positive root) the remaining iterations up to the cap reproduce it bit
     * for bit, so leave with the cap count the full loop would report */
    if (pstar == pold && fabs(f1) > tol) {
      nn = 50;
      break;
    }
  } while (fabs(f1) > tol && nn < 50);
  /* the density and (variant 0) the velocity of the last iterate evaluated */
  if (variant == 0) usl = dsub(ul, ql);
  else usl = dsub(ul, ddiv(dsub(pstar, pl), Wl));
  out[0] = rhols_cal(rhol, pl, pold, gl, pinfl);
  out[1] = pstar;
  out[2] = usl;
  return nn;
}

/* The same solve without the shared reciprocals and the replay, for the FP32
 * residual's inline calls (two or three iterations each, where neither pays
 * much): inlined there, any other form of it changes how the compiler contracts
 * the FP32 arithmetic around the call, and with it the residual's rounding. */
PGDG_HD double jaco_serial(double W, double pl, double rhol, double ps, double g) {
  double t = ddiv(dsub(ps, pl), dmul(W, W));
  t = dmul(t, rhol);
  t = dmul(t, dadd(g, 1));
  t = ddiv(t, 4.);
  t = ddiv(t, W);
  return dsub(ddiv(1., W), t);
}

PGDG_HD int mgfm_serial(double ul, double ur, double pl, double pr, double rhol, double rhor, double gl,
                 double pinfl, double gr, double pinfr, int variant, double seed_p, double out[3]) {
  double pstar;
  if (variant == 0) {
    pl = amax1(pl, 1e-10);
    pr = amax1(pr, 1e-10);
    rhol = amax1(rhol, 1e-10);
    rhor = amax1(rhor, 1e-10);
    pstar = amax1(pl, pr);
  } else {
    if (pl < 0) pl = 0;
    if (pr < 0) pr = 0;
    pstar = dmul(dadd(pl, pr), 0.5);
  }
  if (seed_p > 0) pstar = seed_p;
  double tol = amax1(1e-8, dmul(1e-3, fabs(dsub(ul, ur))));
  double f1 = 1.;
  double rhols = 0, usl = 0, Wl = 0, Wr = 0;
  int nn = 0;
  do {
    Wl = wl_cal(rhol, pl, pstar, gl, pinfl);
    Wr = wl_cal(rhor, pr, pstar, gr, pinfr);
    if (variant == 0) usl = dsub(ul, ddiv(dsub(pstar, pl), Wl));
    rhols = rhols_cal(rhol, pl, pstar, gl, pinfl);
    f1 = dsub(dsub(dsub(ul, ur), ddiv(dsub(pstar, pl), Wl)), ddiv(dsub(pstar, pr), Wr));
    double jac = dsub(-jaco_serial(Wl, pl, rhol, pstar, gl), jaco_serial(Wr, pr, rhor, pstar, gr));
    double dp = ddiv(-f1, jac);
    double cap = dmul(0.6, pstar);
    if (fabs(dp) > cap) dp = copysign(cap, dp);
    const double pold = pstar;
    pstar = dadd(pstar, dp);
    pstar = amax1(pstar, 1e-8);
    nn++;
    /* every quantity of an iteration is a function of pstar alone: once an
     * unconverged iterate repeats (the 1e-8 floor of a problem without a
     * positive root) the remaining iterations up to the cap reproduce it bit
     * for bit, so leave with the cap count the full loop would report */
    if (pstar == pold && fabs(f1) > tol) {
      nn = 50;
      break;
    }
  } while (fabs(f1) > tol && nn < 50);
  if (variant != 0) usl = dsub(ul, ddiv(dsub(pstar, pl), Wl));
  out[0] = rhols;
  out[1] = pstar;
  out[2] = usl;
  return nn;
}

}  // namespace pgdg
#endif
