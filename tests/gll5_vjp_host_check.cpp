// Host evaluation of the ord-5 WENO reconstruction's reverse in stencil differences (gll5_vjp)
// against the general one (weno_vjp of the GLL projection's transpose) for stencils of any
// size (test_gll5_vjp_host.py): from about 1e7 on the scheme's eps is large against the weights.
#include "host_cuda.h"

#include <cstdio>
#include <random>

#include "awfl_adj.h"
#include "awfl_device.cuh"

using namespace awfl;

int main(int argc, char **argv) {
  Tables<5> &T = c_tab5;
  constexpr size_t n = 125 + 2 * 15 + 9 + 4 + 1;  // recon, c2g, s2g, deriv, idl, sigma
  FILE *f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
  if (!f || fread(&T, sizeof(double), n, f) != n) return printf("FAIL tables\n"), 1;
  fclose(f);
  long bad = 0;
  for (int e = -8; e <= 14; e++) {
    std::mt19937_64 g(8);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (long i = 0; i < 20000; i++) {
      double s[5], lo[3], la[5] = {0, 0, 0, 0, 0}, lb[5] = {0, 0, 0, 0, 0}, lc[5] = {0, 0, 0, 0, 0};
      const double slope = u(g), wave = i % 3 == 0 ? 1.0 : (i % 3 == 1 ? 0.1 : 0.0);
      for (int k = 0; k < 5; k++) s[k] = pow(10.0, e) * (slope * k + wave * u(g) + (i % 2 && k > 2 ? 1.0 : 0.0));
      for (int k = 0; k < 3; k++) lo[k] = u(g);
      for (int m = 0; m < 5; m++)
        for (int k = 0; k < 3; k++) lc[m] += T.c2g[m * 3 + k] * lo[k];
      adj::gll5_vjp(s, lo, la);
      adj::weno_vjp<5>(T, s, lc, lb);
      double top = 0, off = 0;
      for (int k = 0; k < 5; k++) {
        top = fmax(top, fabs(lb[k]));
        off = fmax(off, fabs(la[k] - lb[k]));
      }
      // one derivative in two forms: rounding, amplified by the weights' sensitivity to the
      // indicators; neither depends on the scale
      if (!(off <= 1e-9 * top) && bad++ < 5) printf("FAIL scale 1e%d: %g of %g\n", e, off, top);
    }
  }
  if (!bad) printf("ok\n");
  return bad != 0;
}
