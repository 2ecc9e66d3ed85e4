// The comparison of the transform tables with the FP32 forms' compile-time constants
// (host::fp32_forms_match), for tables read from a file (test_fp32_tables_host.py): accepted as
// they are, refused with any one of the compared entries changed.
#include "host_cuda.h"

#include <cstdio>
#include <vector>

#include "awfl_recip.h"

using namespace awfl;

int main(int argc, char **argv) {
  for (int a = 1; a < argc; a++) {
    const int o = a == 1 ? 5 : 9, g = a == 1 ? 3 : 5, hs = (o - 1) / 2;
    // recon, c2g, s2g, deriv, idl, sigma
    const size_t n_rec = o * o * o, n_c2g = o * g, n_der = g * g, n = n_rec + 2 * n_c2g + n_der + hs + 3;
    std::vector<double> t(n);
    FILE *f = fopen(argv[a], "rb");
    if (!f || fread(t.data(), sizeof(double), n, f) != n) return printf("FAIL read\n"), 1;
    fclose(f);
    double *c2g = &t[n_rec], *deriv = &t[n_rec + 2 * n_c2g], *idl = deriv + n_der, *sigma = idl + hs + 2;
    auto match = [&] { return host::fp32_forms_match(o, t.data(), c2g, deriv, idl, *sigma); };
    if (!match()) printf("FAIL ord %d: the tables are refused\n", o);
    auto refused = [&](double *x, const char *what, long i) {
      const double old = *x;
      *x += 1e-9;
      if (match()) printf("FAIL ord %d: a changed %s[%ld] is accepted\n", o, what, i);
      *x = old;
    };
    for (size_t i = 0; i < n_der; i++) refused(deriv + i, "deriv", i);
    for (int i = 0; i < hs + 2; i++) refused(idl + i, "idl", i);
    refused(sigma, "sigma", 0);
    if (o == 9) {
      refused(c2g + 1 * 5 + 3, "c2g", 8);
      for (int i = 0; i < 9; i++) refused(&t[(5 * 9 + 8) * 9 + i], "recon", i);
      for (int i = 0; i < 5; i++) refused(&t[(4 * 9 + 4) * 9 + i], "recon", i);
    }
  }
  printf("done\n");
}
