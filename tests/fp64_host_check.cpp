// Host evaluation of the FP64 path's short forms against the general ones they replace
// (test_fp64_host.py): the pressure's pow, divisions, the WENO reconstruction.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>
#include <random>

#include "awfl_adj.h"
#include "awfl_device.cuh"
#include "awfl_recip.h"

namespace awfl {
static float fmaT(float a, float b, float c) { return fmaf(a, b, c); }
static float rcpT(float x) { return 1.f / x; }
}  // namespace awfl
#include "awfl_weno32.h"

using namespace awfl;

// pow_gamma_cr(x) == pow_cr(x, GAMMA) bit for bit: the table's range, its ends, bin edges
// and both sides of them, and values outside that take the general path
static long check_pow(long n) {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(-20.0, 30.0), in(4.0, 10.0);
  long bad = 0;
  auto one = [&](double x) {
    const double a = pow_gamma_cr(x), b = pow_cr(x, GAMMA);
    if (__double_as_longlong(a) != __double_as_longlong(b) && !(a != a && b != b)) {
      if (bad++ < 5) printf("FAIL pow %a: %a %a\n", x, a, b);
    }
  };
  for (long i = 0; i < n; i++) one(exp2(i % 8 ? in(g) : u(g)));
  for (int e = 3; e <= 11; e++)
    for (int j = 0; j < 128; j++) {
      const double x = ldexp(1.0 + j / 128.0, e);
      one(x); one(nextafter(x, 0)); one(nextafter(x, 1e9));
    }
  for (double x : {0.0, -0.0, -1.0, -300.0, 5e-324, 1e308, (double)INFINITY, -(double)INFINITY, (double)NAN}) one(x);
  return bad;
}

static bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b); }

// divp, div_known and divk against the IEEE division
static long check_div(long n) {
  std::mt19937_64 g(6);
  std::uniform_real_distribution<double> u(-60.0, 60.0), m(1.0, 2.0);
  long bad = 0;
  auto fail = [&](const char *what, double a, double b, double q) {
    if (bad++ < 10) printf("FAIL %s %a / %a = %a\n", what, a, b, q);
  };
  for (long i = 0; i < n; i++) {
    const double a = (i & 1 ? -1 : 1) * exp2(u(g)) * m(g), b = exp2(u(g)) * m(g);
    const double q = divp(a, make_rcp<double>(b));
    if (!same(q, a / b)) fail("divp", a, b, q);
    if (!same(divr(a, make_rcp<double>(-b)), a / -b)) fail("divr", a, -b, q);
    for (int k = 1; k <= 5; k++)
      if (!same(divk(a, k), a / k)) fail("divk", a, k, divk(a, k));
  }
  const double zeros[2] = {0.0, -0.0};
  for (double a : zeros)
    for (double b : {3.0, 0.7, 1e-9, 1e9}) {
      if (!same(divp(a, make_rcp<double>(b)), a / b)) fail("divp zero", a, b, divp(a, make_rcp<double>(b)));
      double h, l;
      host::split_recip(b, &h, &l);
      if (!same(div_known(a, h, l), a / b)) fail("div_known zero", a, b, div_known(a, h, l));
    }
  // known divisors: grid spacings and any significand; random dividends and the ones whose
  // quotient lies next to a midpoint, found here by another route (a = RN(b * midpoint))
  for (long i = 0; i < n / 200; i++) {
    double b = i % 3 == 0 ? 20000.0 / (1 + i / 3) : exp2(u(g)) * m(g);
    if (i % 5 == 0) b = nextafter(exp2((double)(i % 30)), i % 2 ? 0.0 : 1e30);
    double h, l;
    host::split_recip(b, &h, &l);
    for (int x = 0; x < 200; x++) {
      const double q0 = m(g), ulp = 0x1p-53 * (x % 2 ? 1 : .5);
      const double a = x < 100 ? exp2(u(g)) * m(g) : fma(q0, b, ulp * b);
      if (!same(div_known(a, h, l), a / b)) fail("div_known", a, b, div_known(a, h, l));
      if (!same(div_known(-a, -h, -l), a / b)) fail("div_known", -a, -b, div_known(a, h, l));
    }
  }
  return bad;
}

// the WENO reconstruction against weno_coefs and the GLL sums: smooth, rough and constant
// stencils, zeros of both signs, scales from 1e-150 (weights at their ideal values) to 1e150
// (the general routine), infinities and NaN
template <int ORD> static long check_weno(long n) {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> u(-1.0, 1.0), sc(-30.0, 30.0), wide(-150.0, 150.0);
  std::normal_distribution<double> nd;
  long bad = 0;
  for (long i = 0; i < n; i++) {
    StenV<ORD> s;
    const double scale = pow(10.0, i % 16 == 0 ? wide(g) : (i % 4 == 0 ? sc(g) : sc(g) / 6)), base = u(g);
    for (int k = 0; k < ORD; k++) {
      const double x = k - ORD / 2;
      switch (i % 8) {
        case 0: s.v[k] = nd(g); break;
        case 1: s.v[k] = base + 1e-3 * nd(g); break;
        case 2: s.v[k] = base + 0.1 * base * x + 0.01 * u(g) * x * x; break;
        case 3: s.v[k] = (g() % 3) ? 0.0 : nd(g); break;
        case 4: s.v[k] = base; break;
        case 5: s.v[k] = x > 0 ? base : u(g); break;
        case 6: s.v[k] = (g() % 2) ? 0.0 : -0.0; break;
        default: s.v[k] = base * (1 + 1e-14 * nd(g)); break;
      }
      s.v[k] *= scale;
    }
    if (i % 1000 == 999) s.v[g() % ORD] = (i / 1000) % 3 == 0 ? INFINITY : ((i / 1000) % 3 == 1 ? -INFINITY : NAN);
    for (int w = 0; w < 2; w++) {
      const GllV<ORD> a = reconstruct_gll_call<ORD>(s, w), b = reconstruct_gll_general<ORD>(s, w);
      for (int k = 0; k < OrdTraits<ORD>::NGLL; k++)
        if (!same(a.v[k], b.v[k])) {
          if (bad++ < 10)
            printf("FAIL weno%d case %ld weno %d point %d scale %g: %a %a\n", ORD, i % 8, w, k, scale, a.v[k], b.v[k]);
        }
    }
  }
  return bad;
}

// the ord-5 reconstruction's reverse in stencil differences against the general one (weno_vjp
// of the GLL projection's transpose): the same derivative, so equal up to rounding, which the
// weights amplify at most by the ratio of the smoothness indicators' scales: 1e-9 of the
// largest adjoint for stencils of one scale with jumps
static long check_gll5_vjp(long n) {
  std::mt19937_64 g(8);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  long bad = 0;
  for (long i = 0; i < n; i++) {
    double s[5], lo[3], la[5] = {0, 0, 0, 0, 0}, lb[5] = {0, 0, 0, 0, 0}, lc[5];
    const double scale = pow(10.0, 3 * u(g)), slope = u(g), wave = i % 3 == 0 ? 1.0 : (i % 3 == 1 ? 0.1 : 0.0);
    for (int k = 0; k < 5; k++) s[k] = scale * (slope * k + wave * u(g) + (i % 2 && k > 2 ? 1.0 : 0.0));
    for (int k = 0; k < 3; k++) lo[k] = u(g);
    for (int m = 0; m < 5; m++) {
      lc[m] = 0;
      for (int k = 0; k < 3; k++) lc[m] += c_tab5.c2g[m * 3 + k] * lo[k];
    }
    adj::gll5_vjp(s, lo, la);
    adj::weno_vjp<5>(c_tab5, s, lc, lb);
    double top = 0, off = 0;
    for (int k = 0; k < 5; k++) {
      top = fmax(top, fabs(lb[k]));
      off = fmax(off, fabs(la[k] - lb[k]));
    }
    if (!(off <= 1e-9 * top) && bad++ < 5) printf("FAIL gll5_vjp %g of %g\n", off, top);
  }
  return bad;
}

// the FP32 form's reconstruction in stencil differences against the general routine in FP64:
// rounding 2^-24 of the stencil's range, times at most 32 in a fifth difference, 4 in 1/tv^2 and
// 8 in the mapped weights, and the rounding of the values themselves
template <int ORD> static long check_weno32(long n) {
  std::mt19937_64 g(9);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::normal_distribution<double> nd;
  long bad = 0;
  for (long i = 0; i < n; i++) {
    StenV<ORD> s;
    float f[ORD], o[OrdTraits<ORD>::NGLL];
    const double scale = pow(10.0, 2 * u(g)), base = i % 2 ? u(g) : 0.0, wave = .1 + .8 * fabs(u(g)), phase = 3 * u(g);
    const int jump = (int)(g() % ORD);
    double range = 0, top = 0;
    for (int k = 0; k < ORD; k++) {
      const double x = i % 3 == 0 ? nd(g) : (i % 3 == 1 ? sin(wave * k + phase) : (k >= jump) + .01 * nd(g));
      f[k] = (float)(scale * (base + (i % 5 ? x : 0.01 * x)));
      s.v[k] = f[k];
    }
    for (int k = 0; k < ORD; k++) {
      range = fmax(range, fabs(s.v[k] - s.v[ORD / 2]));
      top = fmax(top, fabs(s.v[k]));
    }
    const GllV<ORD> r = reconstruct_gll_general<ORD>(s, true);
    if constexpr (ORD == 5) weno_gll5<float>(f, o);
    else weno_gll9<float>(f, o);
    for (int k = 0; k < OrdTraits<ORD>::NGLL; k++)
      if (!(fabs(o[k] - r.v[k]) <= 0x1p-24 * (1024 * range + 2 * top)) && bad++ < 5)
        printf("FAIL weno32 ord %d point %d: %g %g range %g\n", ORD, k, o[k], r.v[k], range);
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
  if (argc < 3 || !load_tables<5>(argv[1], c_tab5) || !load_tables<9>(argv[2], c_tab9)) {
    printf("FAIL tables\n");
    return 1;
  }
  const long scale = argc > 3 ? atol(argv[3]) : 1;
  const long bad = check_pow(2000000 * scale) + check_div(1000000 * scale) + check_weno<5>(1000000 * scale) +
                   check_weno<9>(200000 * scale) + check_gll5_vjp(200000 * scale) +
                   check_weno32<5>(400000 * scale) + check_weno32<9>(400000 * scale);
  if (!bad) printf("ok\n");
  return bad ? 1 : 0;
}
