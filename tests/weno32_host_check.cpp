// Host evaluation of the FP32 form's WENO reconstruction (awfl_weno32.h) against the general
// routine in FP64 over the values a tracer can have (test_weno32_host.py): stencils scaled by
// 1e-10 to 1e7, where the smoothness indicators' squares pass the scheme's eps of 1e-20 and,
// at the other end, their reciprocals do.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>
#include <random>

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
  if (!bad) printf("ok\n");
  return bad ? 1 : 0;
}
