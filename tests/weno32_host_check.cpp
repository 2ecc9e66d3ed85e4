// Host evaluation of the FP32 form's WENO reconstruction (awfl_weno32.h) against the general
// routine in FP64 over the values a tracer can have (test_weno32_host.py): stencils scaled by
// 1e-10 to 1e7, where the smoothness indicators' squares pass the scheme's eps of 1e-20 and,
// at the other end, their reciprocals do.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <random>
#include <vector>

#include "awfl_device.cuh"
#include "awfl_recip.h"

namespace awfl {
static float fmaT(float a, float b, float c) { return fmaf(a, b, c); }
static float rcpT(float x) { return 1.f / x; }
}  // namespace awfl
#include "awfl_weno32.h"

using namespace awfl;

template <int ORD> static void weno32(const float (&u)[ORD], float (&out)[OrdTraits<ORD>::NGLL]) {
  if constexpr (ORD == 5) weno_gll5<float>(u, out);
  else weno_gll9<float>(u, out);
}

// A stencil of one of five kinds: random, a wave, a jump, an offset with noise, a slope with
// noise.
template <int ORD> static void draw(std::mt19937_64 &g, int kind, double scale, float (&f)[ORD]) {
  std::normal_distribution<double> nd;
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const double base = u(g), wave = .1 + .8 * fabs(u(g)), phase = 3 * u(g);
  const int jump = (int)(g() % ORD);
  for (int k = 0; k < ORD; k++) {
    double x = nd(g);
    if (kind == 1) x = sin(wave * k + phase);
    if (kind == 2) x = (k >= jump) + .01 * x;
    if (kind == 3) x = base + .01 * x;
    if (kind == 4) x = base + .3 * k * phase + .01 * x;
    f[k] = (float)(scale * x);
  }
}

// The bound of a value's error: rounding 2^-24 of the stencil's range, times at most 32 in a
// fifth difference, 4 in 1/tv^2 and 8 in the mapped weights, and the rounding of the values
// themselves. It does not depend on the scale: the same quantities round.
template <int ORD> static long check_scales(long n) {
  std::mt19937_64 g(11);
  long bad = 0;
  for (int e = -10; e <= 7; e++)
    for (int kind = 0; kind < 5; kind++)
      for (long i = 0; i < n; i++) {
        float f[ORD], o[OrdTraits<ORD>::NGLL];
        draw(g, kind, pow(10.0, e), f);
        StenV<ORD> s;
        double range = 0, top = 0;
        for (int k = 0; k < ORD; k++) {
          s.v[k] = f[k];
          range = fmax(range, fabs((double)f[k] - f[ORD / 2]));
          top = fmax(top, fabs(s.v[k]));
        }
        const GllV<ORD> r = reconstruct_gll_general<ORD>(s, true);
        weno32<ORD>(f, o);
        for (int k = 0; k < OrdTraits<ORD>::NGLL; k++)
          if (!(fabs(o[k] - r.v[k]) <= 0x1p-24 * (1024 * range + 2 * top)) && bad++ < 5)
            printf("FAIL ord %d scale 1e%d kind %d point %d: %g %g range %g\n", ORD, e, kind, k, o[k], r.v[k], range);
      }
  return bad;
}

// The same reconstruction from the scheme's matrices in FP32, sums of products in stencil order:
// what the form in differences is to be at least as accurate as.
template <int ORD> struct Matrices {
  static constexpr int HS = (ORD - 1) / 2, NG = OrdTraits<ORD>::NGLL;
  float low[HS + 1][HS + 1][HS + 1], high[ORD][ORD], gll[ORD][NG], idl[HS + 2], sigma;
  explicit Matrices(const Tables<ORD> &T) : sigma((float)T.sigma) {
    auto rec = [&](int i, int s, int ii) { return T.recon[(i * ORD + s) * ORD + ii]; };
    for (int i = 0; i <= HS; i++)
      for (int s = 0; s <= HS; s++)
        for (int ii = 0; ii <= HS; ii++) low[i][s][ii] = (float)rec(i, s, ii);
    for (int s = 0; s < ORD; s++)
      for (int ii = 0; ii < ORD; ii++) {
        double m = rec(HS + 1, s, ii);
        for (int i = 0; ii <= HS && i <= HS; i++)
          if (s >= i && s - i <= HS) m -= T.idl[i] * rec(i, s - i, ii);
        high[s][ii] = (float)(m / T.idl[HS + 1]);
      }
    for (int s = 0; s < ORD; s++)
      for (int ii = 0; ii < NG; ii++) gll[s][ii] = (float)T.c2g[s * NG + ii];
    for (int i = 0; i < HS + 2; i++) idl[i] = (float)T.idl[i];
  }
  void eval(const float (&u)[ORD], float (&out)[NG]) const {
    float a[HS + 2][ORD] = {}, w[HS + 2], tv[HS + 2], c[ORD] = {}, avg = 0, sum = 0;
    for (int i = 0; i <= HS; i++) {
      for (int ii = 0; ii <= HS; ii++)
        for (int s = 0; s <= HS; s++) a[i][ii] = fmaf(low[i][s][ii], u[i + s], a[i][ii]);
      tv[i] = HS == 2 ? awfl_tv_n3<float>(a[i]) : awfl_tv_n5<float>(a[i]);
      avg += tv[i];
    }
    for (int ii = 0; ii < ORD; ii++)
      for (int s = 0; s < ORD; s++) a[HS + 1][ii] = fmaf(high[s][ii], u[s], a[HS + 1][ii]);
    tv[HS + 1] = ORD == 5 ? awfl_tv_n5<float>(a[HS + 1]) : awfl_tv_n9<float>(a[HS + 1]);
    avg *= 1.f / (HS + 1);
    tv[HS + 1] = fmaf(tv[HS + 1] - avg, sigma, avg);
    for (int i = 0; i < HS + 2; i++) sum += w[i] = idl[i] / fmaf(tv[i], tv[i], 1e-20f);
    const float inv = 1 / (sum + 1e-20f);
    sum = 0;
    for (int i = 0; i < HS + 2; i++) {
      const float x = w[i] * inv, d = idl[i];
      sum += w[i] = x * ((d + d * d) + (x * x - (3 * d) * x)) / (d * d + x * (1 - 2 * d));
    }
    for (int i = 0; i < HS + 2; i++)
      for (int ii = 0; ii < ORD; ii++) c[ii] = fmaf(w[i] * (1 / (sum + 1e-20f)), a[i][ii], c[ii]);
    for (int k = 0; k < NG; k++) {
      out[k] = 0;
      for (int s = 0; s < ORD; s++) out[k] = fmaf(gll[s][k], c[s], out[k]);
    }
  }
};

// Errors against the general routine in FP64, over the stencil's largest value: their root mean
// square and their 99.99% quantile no larger than the matrix form's. The quantile lies 5 n / 10^4
// values from the top, 200 for random stencils: the two forms' own differ by up to 1% from sample
// to sample (the tail falls tenfold over a third of the quantile), so 5% is the margin.
template <int ORD> static long check_errors(long n, const Tables<ORD> &T) {
  constexpr int NG = OrdTraits<ORD>::NGLL;
  const Matrices<ORD> M(T);
  long bad = 0;
  for (int kind = 0; kind < 5; kind++)
    for (double scale : {1.0, 1e3, 1e6, 1e9}) {
      if (scale > 1e8 && (kind == 0 || kind == 2)) continue;  // FP32 squares of the indicators overflow
      std::mt19937_64 g(12 + kind);
      std::vector<double> e[2];
      double sq[2] = {0, 0};
      for (long i = 0; i < n; i++) {
        float f[ORD], o[2][NG];
        draw(g, kind, scale, f);
        StenV<ORD> s;
        double top = 0;
        for (int k = 0; k < ORD; k++) top = fmax(top, fabs(s.v[k] = f[k]));
        const GllV<ORD> r = reconstruct_gll_general<ORD>(s, true);
        weno32<ORD>(f, o[0]);
        M.eval(f, o[1]);
        for (int q = 0; q < 2; q++)
          for (int k = 0; k < NG; k++) {
            const double x = fabs(o[q][k] - r.v[k]) / top;
            e[q].push_back(x);
            sq[q] += x * x;
          }
      }
      double tail[2];
      for (int q = 0; q < 2; q++) {
        auto at = e[q].begin() + (long)(e[q].size() * .9999);
        std::nth_element(e[q].begin(), at, e[q].end());
        tail[q] = *at;
      }
      if (!(sq[0] <= sq[1]) || !(tail[0] <= 1.05 * tail[1])) {
        bad++;
        printf("FAIL ord %d kind %d scale %g: rms %.3g of %.3g, tail %.3g of %.3g\n", ORD, kind, scale, sqrt(sq[0] / e[0].size()),
               sqrt(sq[1] / e[1].size()), tail[0], tail[1]);
      }
    }
  return bad;
}

template <int ORD> static bool load_tables(const char *path, Tables<ORD> &T) {
  FILE *f = fopen(path, "rb");
  if (!f) return false;
  constexpr size_t n = ORD * ORD * ORD + 2 * ORD * Tables<ORD>::NG + Tables<ORD>::NG * Tables<ORD>::NG + Tables<ORD>::HS + 3 +
                       Tables<ORD>::NG;  // the struct's leading members, in its order
  const bool ok = fread(&T, sizeof(double), n, f) == n;
  fclose(f);
  return ok && host::complete_tables(T);
}

int main(int argc, char **argv) {
  if (argc < 4 || !load_tables<5>(argv[2], c_tab5) || !load_tables<9>(argv[3], c_tab9)) {
    printf("FAIL tables\n");
    return 1;
  }
  long bad = 1;
  if (!strcmp(argv[1], "scales5")) bad = check_scales<5>(20000);
  if (!strcmp(argv[1], "scales9")) bad = check_scales<9>(20000);
  if (!strcmp(argv[1], "errors5")) bad = check_errors<5>(400000, c_tab5);
  if (!strcmp(argv[1], "errors9")) bad = check_errors<9>(400000, c_tab9);
  if (!bad) printf("ok\n");
  return bad ? 1 : 0;
}
