// Host side of the FP64 path's divisions by known divisors (awfl_div.cuh) and of the
// constants that its reconstruction derives from the transform tables.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "awfl_internal.h"

namespace awfl {
namespace host {

// 1/b = h + l with |h| rounded towards zero and l of its sign, so that a/b =
// fma(a, h, a*l) (div_known) is the IEEE quotient, the sign of a zero included (N.
// Brisebarre, J.-M. Muller, "Correctly rounded multiplication by arbitrary precision
// constants", IEEE Trans. Computers 57(2), 2008). The value rounded last lies within 2^-104
// of the quotient, so only a dividend whose quotient is that close to a rounding midpoint
// can go wrong: with integer significands X and B of 53 bits and an odd 54-bit midpoint M,
// |X*2^s - M*B| <= 8. There is none for a B of less than 50 significant bits (3, 5, every
// spacing like 20000/256), and otherwise at most 32 of the 2^52 significands X.
inline void split_recip(double b, double *h, double *l) {
  int e;
  const uint64_t B = (uint64_t)std::ldexp(std::frexp(std::fabs(b), &e), 53);  // |b| = B * 2^(e-53)
  const unsigned __int128 N = (unsigned __int128)1 << 105;
  const double q = (double)(uint64_t)(N / B), r = (double)(uint64_t)(N % B) / (double)B;  // N/B = q + r, q exact
  *h = std::copysign(std::ldexp(q, 53 - e - 105), b);
  *l = std::copysign(std::ldexp(r, 53 - e - 105), b);
}

// The derived members of Tables; false if the tables lack the structure that the FP64
// reconstruction relies on (zeros and powers of two, the ord-5 entries it has as literals).
template <int ORD> bool complete_tables(Tables<ORD> &t) {
  constexpr int HS = Tables<ORD>::HS, NG = Tables<ORD>::NG;
  t.ridl = 1.0 / t.idl[HS + 1];
  split_recip(t.idl[HS + 1], &t.ridl_h, &t.ridl_l);
  bool ok = true;
  for (int i = 0; i < HS + 2; i++) {
    const double d = t.idl[i];
    const double dd = d * d;
    t.map_a[i] = d + dd;
    t.map_b[i] = 3. * d;
    t.map_c[i] = dd;
    t.map_d[i] = 1. - 2. * d;
  }
  auto rec = [&](int i, int s, int ii) { return t.recon[(i * ORD + s) * ORD + ii]; };
  auto pow2 = [](double x) { int e; return std::fabs(std::frexp(x, &e)) == 0.5; };
  for (int i = 0; i < HS + 1; i++)
    for (int s = 0; s < ORD; s++)
      for (int ii = 0; ii < ORD; ii++)
        if (s > HS || ii > HS) ok = ok && rec(i, s, ii) == 0.0;
  for (int ii = 1; ii < ORD; ii += 2) {
    ok = ok && rec(HS + 1, HS, ii) == 0.0;
    if (ii <= HS) ok = ok && rec(HS / 2, HS / 2, ii) == 0.0;
  }
  for (int s = 0; s < ORD; s++) {
    ok = ok && t.c2g[s * NG + NG / 2] == (s == 0 ? 1.0 : 0.0);
    ok = ok && pow2(t.c2g[s * NG]) && pow2(t.c2g[s * NG + NG - 1]);
  }
  for (int ii = 0; ii < NG; ii++) ok = ok && t.c2g[ii] == 1.0;
  if (ORD == 5) {
    const double d[4] = {w5::kD0, w5::kD1, w5::kD0, w5::kD3};
    for (int i = 0; i < 4; i++) ok = ok && std::fabs(t.idl[i] - d[i]) <= 1e-15;
    ok = ok && t.sigma == w5::kSigma;
    static const double low[3][3][3] = {{{-kW24, .5, .5}, {2 * kW24, -2., -1.}, {kW2324, 1.5, .5}},
                                        {{-kW24, -.5, .5}, {kW1312, 0., -1.}, {-kW24, .5, .5}},
                                        {{kW2324, -1.5, .5}, {2 * kW24, 2., -1.}, {-kW24, -.5, .5}}};
    static const double high[5][5] = {{kH00, kH01, -.0625, -2 * kW24, kW24}, {-kH10, -kH11, .75, 4 * kW24, -4 * kW24},
                                      {kH20, 0., -1.375, 0., .25}, {-kH10, kH11, .75, -4 * kW24, -4 * kW24},
                                      {kH00, -kH01, -.0625, 2 * kW24, kW24}};
    static const double der[9] = {-3., -1., 1., 4., 0., -4., -1., 1., 3.};
    for (int i = 0; i < 3; i++)
      for (int s = 0; s < 3; s++)
        for (int ii = 0; ii < 3; ii++) ok = ok && rec(i, s, ii) == low[i][s][ii];
    for (int s = 0; s < 5; s++)
      for (int ii = 0; ii < 5; ii++) ok = ok && rec(3, s, ii) == high[s][ii];
    static const double c2g[5] = {1., .5, .25, .125, .0625};
    for (int s = 0; s < 5; s++) ok = ok && t.c2g[s * NG + NG - 1] == c2g[s] && t.c2g[s * NG] == (s % 2 ? -c2g[s] : c2g[s]);
    for (int x = 0; x < 9; x++) ok = ok && t.deriv[x] == der[x];
  }
  return ok;
}

// What the FP32 forms (weno_gll5, weno_gll9, deriv32) hold as compile-time constants, against
// the tables that they come from.
inline bool fp32_forms_match(int ord, const double *recon, const double *c2g, const double *deriv, const double *idl,
                             double sigma) {
  auto near = [](double a, double b) { return std::fabs(a - b) <= 1e-12 * std::fmax(1.0, std::fabs(b)); };
  if (ord == 5) {
    static const double der[9] = {-3., -1., 1., 4., 0., -4., -1., 1., 3.};
    bool ok = near(sigma, w5::kSigma);
    for (int i = 0; i < 4; i++) ok = ok && near(idl[i], i == 1 ? w5::kD1 : (i == 3 ? w5::kD3 : w5::kD0));
    for (int x = 0; x < 9; x++) ok = ok && near(deriv[x], der[x]);
    return ok;
  }
  bool ok = near(sigma, w9::kSigma) && near(c2g[1 * 5 + 3], w9::kX1) && near(c2g[1 * 5 + 4], 0.5);
  for (int i = 0; i < 6; i++) ok = ok && near(idl[i], w9::ideal(i));
  for (int i = 0; i < 9; i++) {
    // u = 1 in cell 7 (D_2 = 1, D_3 = -5), then in cell 8 (D_3 = 1); P_2 = 0 for both
    if (i < 5) ok = ok && near(recon[(3 * 9 + 4) * 9 + i], w9::kN.c[i]) && near(recon[(4 * 9 + 4) * 9 + i], w9::kM.c[i]);
    ok = ok && near(recon[(5 * 9 + 7) * 9 + i], w9::kFa.c[i] - 5 * w9::kFb.c[i]) &&
         near(recon[(5 * 9 + 8) * 9 + i], w9::kFb.c[i]);
  }
  for (int s = 0; s < 5; s++)
    for (int ii = 0; ii < 5; ii++) ok = ok && near(deriv[s * 5 + ii], ii < 3 ? w9::kD.d[ii][s] : -w9::kD.d[4 - ii][4 - s]);
  return ok;
}

}  // namespace host
}  // namespace awfl
