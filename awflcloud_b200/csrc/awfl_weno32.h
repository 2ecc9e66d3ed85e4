// The FP32 form's WENO reconstruction of one stencil, on float or on pairs of lanes. The
// includer declares fmaT and rcpT for its scalar types first.
#pragma once

#include "awfl_internal.h"

namespace awfl {

// The ord-5 WENO reconstruction to the three GLL points in differences of the stencil: with
// d_i = u[i+1]-u[i] and s_i = d[i+1]-d[i], the three parabolas are u[2] - s_i/24 + a_i x +
// (s_i/2) x^2 and the bridge polynomial has the few coefficients of w5, where the matrix
// form multiplies 49 entries. Equal in exact arithmetic; about 100 FP32 instructions instead of
// 150, and u[2] enters the values unrounded. The sweep is issue-bound: with the time series on
// point pairs (Pts, awfl_fp32.cuh), 1,500 -> 1,130 instructions per cell and split, 256x256x128 step 1.433 -> 1.200 ms.
template <class T> __device__ __forceinline__ void weno_gll5(const T (&u)[5], T (&out)[3]) {
  using namespace w5;
  const T d0 = u[1] - u[0], d1 = u[2] - u[1], d2 = u[3] - u[2], d3 = u[4] - u[3];
  const T s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
  const T a0 = fmaT(.5f, s0, d1), c = fmaT(.5f, s1, d1), a2 = fmaT(-.5f, s2, d2);
  const T S = s0 + s2, g = s2 - s0;
  const T e0 = fmaT((float)kE0S, S, (float)kE01 * s1);
  const T h1 = fmaT((float)kH1, g, c);
  const T h2 = fmaT((float)kH2S, S, (float)kH21 * s1);
  const T h3 = (float)kH3 * g;
  const T h4 = fmaT((float)kH4, S, (float)(-2 * kH4) * s1);
  // smoothness indicators (coefs_to_tv of the parabolas and of the bridge polynomial)
  const float k13 = (float)(13. / 12);
  const T t0 = fmaT(a0, a0, (k13 * s0) * s0), t1 = fmaT(c, c, (k13 * s1) * s1), t2 = fmaT(a2, a2, (k13 * s2) * s2);
  T t3 = fmaT(h1, fmaT(.5f, h3, h1), (39.1125f * h3) * h3);
  t3 = fmaT(h2, fmaT(4.2f, h4, (float)(13. / 3) * h2), t3);
  t3 = fmaT(625.8f * h4, h4, t3);
  const T avg = (t0 + t1 + t2) * (float)(1. / 3);
  t3 = fmaT(t3 - avg, (float)kSigma, avg);
  // weights idl/(tv^2 + eps) over idl[0] (two products fewer), and so is the eps of their
  // normalisation: w/(sum + eps) is the scheme's whatever the size of the values (from
  // differences of about 1e3 on, sum is no longer large against eps)
  const T eps = T(1.0e-20f);
  T w[4] = {rcpT(fmaT(t0, t0, eps)), (float)(kD1 / kD0) * rcpT(fmaT(t1, t1, eps)), rcpT(fmaT(t2, t2, eps)),
            (float)(kD3 / kD0) * rcpT(fmaT(t3, t3, eps))};
  T inv = rcpT(((w[0] + w[1]) + (w[2] + w[3])) + T((float)(1.0e-20 / kD0)));
#pragma unroll
  for (int i = 0; i < 4; i++) {  // map_weights (WenoLimiter.h:12-17)
    const double d = i == 1 ? kD1 : (i == 3 ? kD3 : kD0);
    const T x = w[i] * inv;
    w[i] = (x * fmaT(x, x + (float)(-3 * d), T((float)(d + d * d)))) * rcpT(fmaT(x, (float)(1 - 2 * d), T((float)(d * d))));
  }
  inv = rcpT(((w[0] + w[1]) + (w[2] + w[3])) + eps);
  const T Q = fmaT(w[0], s0, fmaT(w[1], s1, w[2] * s2));
  const T P = fmaT(w[0], a0, fmaT(w[1], c, fmaT(w[2], a2, w[3] * fmaT(.25f, h3, h1))));
  // the normalised weights sum to 1 - eps*inv, which shows from differences of about 3e7 on:
  // that is u[2]'s share (256x256x128 step 1136 -> 1140 us)
  const T E = fmaT(-1.0e-20f, u[2], w[3] * e0);
  const T mid = fmaT(inv, fmaT((float)(-1. / 24), Q, E), u[2]);
  const T ev = fmaT(inv, fmaT((float)(1. / 12), Q, fmaT(w[3], fmaT(.0625f, h4, .25f * h2), E)), u[2]);
  const T od = (.5f * inv) * P;
  out[0] = ev - od;
  out[1] = mid;
  out[2] = ev + od;
}

// The ord-9 WENO reconstruction to the five GLL points in differences of the stencil. The
// centred candidate P_2 is formed from central differences; candidates that are neighbours
// agree on their four shared cells, so they differ by a fifth difference D_j of six cells
// times a fixed polynomial (w9: P_3 - P_2 = D_2 N, P_4 - P_3 = D_3 M, the mirror images on the
// other side), and so does the bridge polynomial (four D_j, by parity in sums and differences
// of mirror pairs). The outer candidates' indicators take their coefficients from their own
// differences: two steps of D_j from P_2's lose a smooth outer candidate in a rough stencil
// (10 instructions, 128x128x64 step 422 -> 428 us). Equal to the matrix form in exact
// arithmetic; about 280 instead of 390 FP32 instructions, and u[4]
// enters the values unrounded. Error against FP64 over the stencil's largest value, matrix
// form -> this one, root mean square and 99.9% quantile: random 6.0e-8 -> 3.4e-8 and 2.9e-7 ->
// 2.4e-7, smooth 7.2e-8 -> 2.5e-8 and 2.8e-7 -> 8.6e-8, jump 7.6e-8 -> 2.9e-8 and 3.3e-7 ->
// 1.2e-7; the largest of 4 million random stencils 8.5e-7 -> 9.2e-7. The sweep is issue-bound:
// 128x128x64 step 0.608 -> 0.483 ms when the matrices went.
template <class T> __device__ __forceinline__ void weno_gll9(const T (&u)[9], T (&out)[5]) {
  using namespace w9;
  T d1[8], d2[7], d3[6], d4[5], D[4];
#pragma unroll
  for (int i = 0; i < 8; i++) d1[i] = u[i + 1] - u[i];
#pragma unroll
  for (int i = 0; i < 7; i++) d2[i] = d1[i + 1] - d1[i];
#pragma unroll
  for (int i = 0; i < 6; i++) d3[i] = d2[i + 1] - d2[i];
#pragma unroll
  for (int i = 0; i < 5; i++) d4[i] = d3[i + 1] - d3[i];
#pragma unroll
  for (int i = 0; i < 4; i++) D[i] = d4[i + 1] - d4[i];
  // the candidates' coefficients of x .. x^4 (their indicators and weights need no more), and
  // P_2's constant, less u[4]
  T a[5][5];
  const T m3 = d3[2] + d3[3];
  const T p0 = fmaT((float)(3. / 640), d4[2], (float)(-1. / 24) * d2[3]);
  a[2][1] = fmaT((float)(-5. / 48), m3, .5f * (d1[3] + d1[4]));
  a[2][2] = fmaT(-.0625f, d4[2], .5f * d2[3]);
  a[2][3] = (float)(1. / 12) * m3;
#pragma unroll
  for (int i = 0; i < 5; i++) a[i][4] = (float)(1. / 24) * d4[i];
  constexpr Poly n = kN, m = kM, ha = kHa, hb = kHb;
#pragma unroll
  for (int i = 1; i < 4; i++) {
    const float sg = i % 2 ? 1.f : -1.f;
    a[3][i] = fmaT((float)n.c[i], D[2], a[2][i]);
    a[1][i] = fmaT(sg * (float)n.c[i], D[1], a[2][i]);
  }
  a[4][1] = fmaT((float)(-3. / 16), d4[4], fmaT((float)(7. / 24), d3[4], fmaT(-.5f, d2[4], d1[4])));
  a[4][2] = fmaT((float)(7. / 16), d4[4], .5f * (d2[4] - d3[4]));
  a[4][3] = fmaT(-.25f, d4[4], (float)(1. / 6) * d3[4]);
  a[0][1] = fmaT((float)(3. / 16), d4[0], fmaT((float)(7. / 24), d3[1], fmaT(.5f, d2[2], d1[3])));
  a[0][2] = fmaT((float)(7. / 16), d4[0], .5f * (d2[2] + d3[1]));
  a[0][3] = fmaT(.25f, d4[0], (float)(1. / 6) * d3[1]);
  // the bridge polynomial's
  const T se = D[2] - D[1], so = D[2] + D[1], te = D[3] - D[0], to = D[3] + D[0];
  T h[9];
#pragma unroll
  for (int i = 1; i < 9; i++) {
    const T b = i < 5 ? a[2][i < 5 ? i : 0] : T(0.f);
    h[i] = i < 5 ? fmaT((float)hb.c[i], i % 2 ? to : te, fmaT((float)ha.c[i], i % 2 ? so : se, b))
                 : fmaT((float)hb.c[i], i % 2 ? to : te, (float)ha.c[i] * (i % 2 ? so : se));
  }
  // smoothness indicators (coefs_to_tv), row by row
  auto tv9 = [&](const T *p) {
    T r = p[1] * fmaT(.03125f, p[7], fmaT(.125f, p[5], fmaT(.5f, p[3], p[1])));
    r = fmaT(p[3], fmaT(32.643229166666664f, p[7], fmaT(63.066964285714285f, p[5], 39.1125f * p[3])), r);
    r = fmaT(p[5], fmaT(52976.979166666664f, p[7], 15645.903707837302f * p[5]), r);
    r = fmaT(27599374.140625f * p[7], p[7], r);
    r = fmaT(p[2], fmaT(.5138888888888888f, p[8], fmaT(1.5535714285714286f, p[6], fmaT(4.2f, p[4], (float)(13. / 3) * p[2]))), r);
    r = fmaT(p[4], fmaT(1044.5833333333333f, p[8], fmaT(1513.6279761904761f, p[6], 625.8357142857143f * p[4])), r);
    r = fmaT(p[6], fmaT(2542895.f, p[8], 563252.5334821428f * p[6]), r);
    return fmaT(1766359945.f * p[8], p[8], r);
  };
  T tv[6];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const T *p = a[i];
    T r = p[1] * fmaT(.5f, p[3], p[1]);
    r = fmaT(p[2], fmaT(4.2f, p[4], (float)(13. / 3) * p[2]), r);
    r = fmaT(39.1125f * p[3], p[3], r);
    tv[i] = fmaT(625.8f * p[4], p[4], r);
  }
  tv[5] = tv9(h);
  const T avg = (((tv[0] + tv[1]) + (tv[3] + tv[4])) + tv[2]) * .2f;
  tv[5] = fmaT(tv[5] - avg, (float)kSigma, avg);
  const T eps = T(1.0e-20f);
  T w[6];
#pragma unroll
  for (int i = 0; i < 6; i++) w[i] = (float)ideal(i) * rcpT(fmaT(tv[i], tv[i], eps));
  T inv = rcpT((((w[0] + w[1]) + (w[3] + w[4])) + (w[2] + w[5])) + eps);
#pragma unroll
  for (int i = 0; i < 6; i++) {  // map_weights (WenoLimiter.h:12-17)
    const double d = ideal(i);
    const T x = w[i] * inv;
    w[i] = (x * fmaT(x, x + (float)(-3 * d), T((float)(d + d * d)))) * rcpT(fmaT(x, (float)(1 - 2 * d), T((float)(d * d))));
  }
  inv = rcpT((((w[0] + w[1]) + (w[3] + w[4])) + (w[2] + w[5])) + eps);
  // sum of the weights times (P_i - P_2) and (bridge - P_2), even and odd parts
  const T x2 = ((w[3] + w[4]) * inv) * D[2], x1 = ((w[0] + w[1]) * inv) * D[1];
  const T x3 = (w[4] * inv) * D[3], x0 = (w[0] * inv) * D[0], wh = w[5] * inv;
  // the normalised weights sum to 1 - eps*inv, as at ord 5: P_2's share (428 -> 431 us)
  const T lack = -1.0e-20f * inv, uc = fmaT(lack, u[4], u[4]), pc = fmaT(lack, p0, p0);
  T ac[5];
#pragma unroll
  for (int i = 1; i < 5; i++) ac[i] = fmaT(lack, a[2][i], a[2][i]);
  const T ne = x2 - x1, no = x2 + x1, me = x3 - x0, mo = x3 + x0;
  const T ae = wh * se, ao = wh * so, be = wh * te, bo = wh * to;
  auto even = [&](double x) {
    T r = fmaT((float)n.even(x), ne, pc);
    r = fmaT((float)m.even(x), me, r);
    r = fmaT((float)ha.even(x), ae, r);
    return fmaT((float)hb.even(x), be, r);
  };
  out[2] = uc + even(0.);
  constexpr double xs[2] = {.5, kX1};
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const double x = xs[j];
    T ev = even(x);
    ev = uc + fmaT((float)(x * x), fmaT((float)(x * x), ac[4], ac[2]), ev);
    T od = (float)x * fmaT((float)(x * x), ac[3], ac[1]);
    od = fmaT((float)n.odd(x), no, od);
    od = fmaT((float)m.odd(x), mo, od);
    od = fmaT((float)ha.odd(x), ao, od);
    od = fmaT((float)hb.odd(x), bo, od);
    out[j] = ev - od;
    out[4 - j] = ev + od;
  }
}

}  // namespace awfl
