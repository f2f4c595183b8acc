// Householder reflector of (alpha, x) with ||x||^2 = xn2 (zlarfg semantics):
// beta = -sign(Re alpha) ||(alpha, x)||, tau, and sc = 1 / (alpha - beta), the factor
// of x in v = (1, x sc).
#pragma once
#include <float.h>

#include "common.cuh"

// float: the square root and the division by beta come from one reciprocal
// square root with a Newton step (an IEEE square root and four IEEE divisions in a
// row are a third of a column's latency).  A subnormal squared norm (the column's
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
  const float m = ss * y;
  beta = -copysignf(m, alpha.x);
  const float ib = -copysignf(y, alpha.x);
  t = make_float2((beta - alpha.x) * ib, -alpha.y * ib);
  const float dx = alpha.x - beta;  // no cancellation: beta has the other sign
  const float id = __frcp_rn(fmaf(dx, dx, alpha.y * alpha.y));
  sc = make_float2(dx * id, -alpha.y * id);
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
