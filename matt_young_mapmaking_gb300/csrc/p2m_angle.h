/*
 * p2m_angle.h -- a candidate pixel's angular distance from a disc centre in float-float
 * arithmetic, for the painting kernels; the same operations on the host, where the accuracy
 * is tested (tests/test_angle_cpu.py).
 *
 * Pairs (hi, lo) stand for hi + lo.  Each step is an error-free transformation (Dekker's and
 * Knuth's two-sum, the two-product by a fused multiply-add) or a correction whose rounding is
 * small against the result.
 */
#ifndef P2M_ANGLE_H
#define P2M_ANGLE_H

#include "p2m_fmath.h"

#if defined(__CUDA_ARCH__)
#define FFMA(a, b, c) __fmaf_rn((a), (b), (c))
#else
#include <math.h>
#define FFMA(a, b, c) fmaf((a), (b), (c))
#endif

/* sin(y) - y by its Taylor series through y^15, for the half longitude offset y of a
   candidate from the disc centre: |y| < pi/2 + pi/npr <= 2.37, where the truncation stays
   below 1e-8; the result is a correction to y, so its relative rounding (a few ulp)
   costs ~y^2/6 ulp of sin(y).  y2 = y^2. */
P2M_HD float p2m_sin_minus_arg(float y, float y2) {
  float p = 1.0f / 1307674368000.0f;      /* 1/15! */
  p = FFMA(p, y2, -1.0f / 6227020800.0f); /* -1/13! */
  p = FFMA(p, y2, 1.0f / 39916800.0f);    /* 1/11! */
  p = FFMA(p, y2, -1.0f / 362880.0f);     /* -1/9! */
  p = FFMA(p, y2, 1.0f / 5040.0f);        /* 1/7! */
  p = FFMA(p, y2, -1.0f / 120.0f);        /* -1/5! */
  p = FFMA(p, y2, 1.0f / 6.0f);           /* 1/3! */
  return FMUL(FMUL(-y, y2), p);           /* -y^3 (1/3! - y^2/5! + ...) */
}

/* asin(u) - u by its series through u^15 for 0 <= u <= 1/4 (truncation < 1e-12 of u); u2 = u^2 */
P2M_HD float p2m_asin_minus_arg(float u, float u2) {
  float p = 143.0f / 10240.0f;
  p = FFMA(p, u2, 231.0f / 13312.0f);
  p = FFMA(p, u2, 63.0f / 2816.0f);
  p = FFMA(p, u2, 35.0f / 1152.0f);
  p = FFMA(p, u2, 5.0f / 112.0f);
  p = FFMA(p, u2, 3.0f / 40.0f);
  p = FFMA(p, u2, 1.0f / 6.0f);
  return FMUL(FMUL(u, u2), p);
}

/* chord^2 = c2 + c2l of a candidate n pixels from its item's origin, c2 the nearest float but
   for the last bit: A + B sin^2(y), y = n d + y0, with A, B (ah, al, bh, bl), y0 and d (y0h,
   y0l, dh, dl) as pairs.  *ysq: y^2. */
P2M_HD float p2m_chord_sq(float ah, float al, float bh, float bl, float y0h, float y0l, float dh,
                          float dl, int n, float *c2l, float *ysq) {
  /* y: the product as an exact pair plus n d_lo, then Knuth's two-sum */
  const float fn = (float)n;
  const float pd = FMUL(fn, dh);
  const float pe = FFMA(fn, dl, FFMA(fn, dh, -pd));
  const float y = FADD(pd, y0h), yb = FSUB(y, pd);
  float yl = FADD(FADD(FSUB(pd, FSUB(y, yb)), FSUB(y0h, yb)), FADD(pe, y0l));
  /* sin(y + yl) = y + (sin(y) - y) + yl cos(y), cos(y) as 1 - y^2/2; |sin(y) - y| < |y| */
  const float y2 = FMUL(y, y);
  const float sc = p2m_sin_minus_arg(y, y2);
  yl = FMUL(yl, FFMA(y2, -0.5f, 1.0f));
  const float su = FADD(y, sc);
  const float sv = FADD(FSUB(sc, FSUB(su, y)), yl);
  /* normalised: the square of the low word is left out below */
  const float sh = FADD(su, sv), sl = FSUB(sv, FSUB(sh, su));
  /* sin^2, B sin^2, A + B sin^2 */
  const float q = FMUL(sh, sh);
  const float qe = FFMA(FADD(sh, sh), sl, FFMA(sh, sh, -q));
  const float b = FMUL(bh, q);
  const float be = FFMA(bl, q, FFMA(bh, qe, FFMA(bh, q, -b)));
  const float c2 = FADD(ah, b), cb = FSUB(c2, ah);
  *c2l = FADD(FADD(FSUB(ah, FSUB(c2, cb)), FSUB(b, cb)), FADD(al, be));
  *ysq = y2;
  return c2;
}

/* The angle 2 asin(chord / 2) as *hi + *lo from chord^2 = c2 + c2l (normal, well above the
   smallest) and rs, 1 / sqrt(c2) to 2^-22; returns u = chord / 2.  Beyond u = 1/4 only u counts.
   Newton's iteration for the root and then for its reciprocal brings both to about their last
   bit; the second step of the root then leaves an error of second order in them, 2^-47. */
P2M_HD float p2m_chord_angle(float c2, float c2l, float rs, float *hi, float *lo) {
  float hr = FMUL(0.5f, rs);
  const float c0 = FMUL(c2, rs), ch = FFMA(FFMA(-c0, c0, c2), hr, c0);
  hr = FFMA(hr, FFMA(-ch, rs, 1.0f), hr);
  const float dy = FMUL(FADD(FFMA(-ch, ch, c2), c2l), hr);
  const float chord = FADD(ch, dy), cl = FSUB(dy, FSUB(chord, ch));
  /* angle = chord + 2 (asin(u) - u) + the low word times the arc sine's slope, 1 + u^2/2 */
  const float u = FMUL(0.5f, chord), u2 = FMUL(u, u);
  const float ac = FMUL(2.0f, p2m_asin_minus_arg(u, u2));
  *hi = FADD(chord, ac);
  *lo = FFMA(cl, FFMA(u2, 0.5f, 1.0f), FSUB(ac, FSUB(*hi, chord)));
  return u;
}

#endif /* P2M_ANGLE_H */
