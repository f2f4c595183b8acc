// Householder reflector of (alpha, x) with ||x||^2 = xn2 (zlarfg semantics):
// beta = -sign(Re alpha) ||(alpha, x)||, tau, and sc = 1 / (alpha - beta), the factor
// of x in v = (1, x sc).
#pragma once
#include <float.h>

#include "common.cuh"

// a / b from r = 1 / b: the product's residual, exact by FMA, corrects it (Markstein)
AGB_DEV float quotient(float a, float b, float r) {
  const float q = a * r;
  return fmaf(fmaf(-b, q, a), r, q);
}

// float: the square root and the divisions come from one reciprocal square root, a
// reciprocal and their Newton steps (an IEEE square root and four IEEE divisions in a
// row are a third of a column's latency), each result rounded once: ||QR - A|| of a
// 128 x 64 matrix 3.78 u, 4.18 u without the last corrections, 3.93 u with IEEE
// operations; they cost 0.4% of a 512 x 256 QR.  A subnormal squared norm (the column's
// below 1.1e-19) leaves the column as it is.
AGB_DEV void reflector(float2 alpha, float xn2, float& beta, float2& t, float2& sc) {
  const float ss = fmaf(alpha.x, alpha.x, fmaf(alpha.y, alpha.y, xn2));
  if ((xn2 == 0.f && alpha.y == 0.f) || ss < FLT_MIN) {
    beta = alpha.x;
    t = sc = make_float2(0.f, 0.f);
    return;
  }
  float y = rsqrtf(ss);
  y = fmaf(0.5f * y, fmaf(-ss * y, y, 1.f), y);
  float m = ss * y;
  m = fmaf(0.5f * y, fmaf(-m, m, ss), m);  // the square root, rounded once
  y = fmaf(y, fmaf(-m, y, 1.f), y);        // its reciprocal
  beta = -copysignf(m, alpha.x);
  const float ib = -copysignf(y, alpha.x);
  const float dx = alpha.x - beta;  // no cancellation: beta has the other sign
  t = make_float2(quotient(-dx, beta, ib), quotient(-alpha.y, beta, ib));
  const float den = fmaf(dx, dx, alpha.y * alpha.y), id = __frcp_rn(den);
  sc = make_float2(quotient(dx, den, id), quotient(-alpha.y, den, id));
}
AGB_DEV void reflector(double2 alpha, double xn2, double& beta, double2& t, double2& sc) {
  if (xn2 == 0.0 && alpha.y == 0.0) {
    beta = alpha.x;
    t = sc = make_double2(0.0, 0.0);
    return;
  }
  beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x);
  t = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
  sc = cinv(csub(alpha, make_double2(beta, 0.0)));
}

// The same where nothing scales the matrix, so that a squared norm may be subnormal:
// such a column is scaled by 2^50 first.
AGB_DEV void reflector_unscaled(float2 alpha, float xn2, float& beta, float2& t, float2& sc) {
  const bool small = fmaf(alpha.x, alpha.x, fmaf(alpha.y, alpha.y, xn2)) < FLT_MIN;
  const float f = small ? 0x1p50f : 1.f;
  reflector(make_float2(alpha.x * f, alpha.y * f), xn2 * f * f, beta, t, sc);
  beta *= small ? 0x1p-50f : 1.f;
  sc = make_float2(sc.x * f, sc.y * f);
}
AGB_DEV void reflector_unscaled(double2 alpha, double xn2, double& beta, double2& t, double2& sc) {
  reflector(alpha, xn2, beta, t, sc);
}
