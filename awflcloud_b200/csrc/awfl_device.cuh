// Device building blocks of the AWFL Euler-3D ADER/WENO step (FP64 parity path).
//
// Every function reproduces the arithmetic of the reference (mrnorman/awflCloud) in its
// evaluation order; the file:line cited is the reference code restated:
//   Spatial  = Spatial_euler3d_cons_expl_cart_fv_Agrid.h
//   Weno     = WenoLimiter.h
// The translation unit that includes this header is compiled with --fmad=false so that
// no multiply-add is contracted, like the reference's CPU build, and every pow is the
// correctly rounded pow_cr (awfl_pow.cuh), like glibc's.
#pragma once

#include <cstdint>
#include <type_traits>

#include "awfl_div.cuh"
#include "awfl_internal.h"
#include "awfl_pow.cuh"
#include "awfl_tv.h"

namespace awfl {

// One copy per translation unit that includes this header (awfl_fp64.cu, awfl_adjoint.cu);
// each is uploaded by that unit's upload function.
static __constant__ Tables<5> c_tab5;
static __constant__ Tables<9> c_tab9;

template <int ORD> __device__ __forceinline__ const Tables<ORD> &tab();
template <> __device__ __forceinline__ const Tables<5> &tab<5>() { return c_tab5; }
template <> __device__ __forceinline__ const Tables<9> &tab<9>() { return c_tab9; }

// Out-of-line forms of the two largest pieces of the per-cell FP64 code, the correctly
// rounded pow and the reconstruction of one variable (stencil and GLL values passed by
// value): one copy of their instructions in the kernel instead of one per call site. The
// fully inlined sweep outgrew the instruction cache (ncu: instruction-fetch stalls of 2.5
// cycles per issued instruction, the largest stall); out of line, the FP64 step took
// 7.38 ms instead of 9.73 ms at 256x256x128. The arithmetic is the same either way.
static __device__ __noinline__ double pow_gamma_call(double x) { return pow_gamma_cr(x); }
__device__ __forceinline__ double pow_gamma(double x) { return pow_gamma_call(x); }
template <class Sc> __device__ __forceinline__ Sc pow_gamma(const Sc &x) { return pow_cr(x, GAMMA); }

// The scalar type Sc is double for the FP64 path and Dual (awfl_dual.cuh) for the
// tangent-linear sweep; both evaluate the same expressions in the same order.
template <int N, class Sc> __device__ __forceinline__ Sc tv_eval(const Sc *a) {
  if constexpr (N == 3) return awfl_tv_n3<Sc>(a);
  else if constexpr (N == 5) return awfl_tv_n5<Sc>(a);
  else return awfl_tv_n9<Sc>(a);
}

// Weno:93-172 -- WENO polynomial coefficients of one ord-cell stencil.
template <int ORD, class Sc>
__device__ __forceinline__ void weno_coefs(const Sc (&u)[ORD], Sc (&aw)[ORD]) {
  constexpr int HS = (ORD - 1) / 2;
  const Tables<ORD> &T = tab<ORD>();
  const double eps = 1.0e-20;
  Sc a[HS + 2][ORD];
#pragma unroll
  for (int j = 0; j < HS + 2; j++)
#pragma unroll
    for (int i = 0; i < ORD; i++) a[j][i] = 0.;
#pragma unroll
  for (int i = 0; i < HS + 1; i++)
#pragma unroll
    for (int ii = 0; ii < HS + 1; ii++)
#pragma unroll
      for (int s = 0; s < HS + 1; s++) a[i][ii] += T.recon[(i * ORD + s) * ORD + ii] * u[i + s];
#pragma unroll
  for (int ii = 0; ii < ORD; ii++)
#pragma unroll
    for (int s = 0; s < ORD; s++) a[HS + 1][ii] += T.recon[((HS + 1) * ORD + s) * ORD + ii] * u[s];
#pragma unroll
  for (int i = 0; i < HS + 1; i++)
#pragma unroll
    for (int ii = 0; ii < HS + 1; ii++) a[HS + 1][ii] -= T.idl[i] * a[i][ii];
  const Rcp<double> ridl = rcp_known(T.idl[HS + 1], T.ridl);
#pragma unroll
  for (int ii = 0; ii < ORD; ii++) a[HS + 1][ii] = divd(a[HS + 1][ii], ridl);
  Sc tv[HS + 2];
#pragma unroll
  for (int i = 0; i < HS + 1; i++) tv[i] = tv_eval<HS + 1>(a[i]);
  tv[HS + 1] = tv_eval<ORD>(a[HS + 1]);
  Sc lo_avg = 0.;
#pragma unroll
  for (int i = 0; i < HS + 1; i++) lo_avg += tv[i];
  lo_avg = divk(lo_avg, HS + 1);
  tv[HS + 1] = lo_avg + (tv[HS + 1] - lo_avg) * T.sigma;
  Sc wts[HS + 2];
#pragma unroll
  for (int i = 0; i < HS + 2; i++) wts[i] = T.idl[i] / (tv[i] * tv[i] + eps);
  // convexify (Weno:20-25)
  {
    Sc sum = 0.;
#pragma unroll
    for (int i = 0; i < HS + 2; i++) sum += wts[i];
    const Rcp<Sc> rs = make_rcp<Sc>(sum + eps);
#pragma unroll
    for (int i = 0; i < HS + 2; i++) wts[i] = divr(wts[i], rs);
  }
  // map_weights (Weno:12-17)
#pragma unroll
  for (int i = 0; i < HS + 2; i++) {
    const double d = T.idl[i];
    wts[i] = wts[i] * (d + d * d - 3. * d * wts[i] + wts[i] * wts[i]) / (d * d + wts[i] * (1. - 2. * d));
  }
  {
    Sc sum = 0.;
#pragma unroll
    for (int i = 0; i < HS + 2; i++) sum += wts[i];
    const Rcp<Sc> rs = make_rcp<Sc>(sum + eps);
#pragma unroll
    for (int i = 0; i < HS + 2; i++) wts[i] = divr(wts[i], rs);
  }
#pragma unroll
  for (int i = 0; i < ORD; i++) aw[i] = 0.;
#pragma unroll
  for (int i = 0; i < HS + 2; i++)
#pragma unroll
    for (int ii = 0; ii < ORD; ii++) aw[ii] += wts[i] * a[i][ii];
}

// Spatial:1800-1833 -- ord stencil averages -> ngll GLL point values.
template <int ORD, class Sc>
__device__ __forceinline__ void reconstruct_gll(const Sc (&sten)[ORD], Sc (&out)[OrdTraits<ORD>::NGLL],
                                                bool doweno) {
  constexpr int NG = OrdTraits<ORD>::NGLL;
  const Tables<ORD> &T = tab<ORD>();
  if (doweno) {
    Sc wc[ORD];
    weno_coefs<ORD>(sten, wc);
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      Sc tmp = 0;
#pragma unroll
      for (int s = 0; s < ORD; s++) tmp += T.c2g[s * NG + ii] * wc[s];
      out[ii] = tmp;
    }
  } else {
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      Sc tmp = 0;
#pragma unroll
      for (int s = 0; s < ORD; s++) tmp += T.s2g[s * NG + ii] * sten[s];
      out[ii] = tmp;
    }
  }
}

// The WENO reconstruction on doubles with the general routine's results (weno_coefs and the
// GLL evaluation above) in about half of its FP64 instructions; the FP64 pipe bounds the
// sweep. What is left out changes no bit:
//   - products with structural zeros, and sums that start at 0 +: the sign of a zero is all
//     they can change, and the last sum of each GLL value, which does start at +0, drops it;
//   - a product by a power of two is exact, so it goes with its sum into one FMA;
//   - ord 5 shares products: u/24, u/12 and u/6 are one rounded product scaled by 2 and 4;
//   - the weights' divisions by div_near, interleaved (no branch per division), the bridge
//     polynomial's by div_known; the mapping's constants come from the tables.
// A stencil whose smoothness indicators leave the range in which these hold (tv^2 >= 2^300,
// infinities and NaN among them) is left to the general routine: these return false. Where all
// values of a stencil are below about 1e-303 the shared products round as subnormal numbers:
// the two then differ by up to 4 of the smallest one (5e-324), like quotients there
// (awfl_div.cuh). Sending such stencils to the general routine cost the FP64 step with tracers 1.5%.
// 256x256x128: ord 5 6.68 -> 4.86 ms per step; 128x128x64, ord 9: 3.99 -> 3.30 ms.
template <int ORD>
__device__ __forceinline__ bool weno_weights(const double (&tv)[(ORD + 3) / 2], double (&w)[(ORD + 3) / 2]) {
  constexpr int HS = (ORD - 1) / 2;
  const Tables<ORD> &T = tab<ORD>();
  unsigned top = 0;
#pragma unroll
  for (int i = 0; i < HS + 2; i++) {
    w[i] = tv[i] * tv[i] + 1.0e-20;
    top = max(top, (unsigned)__double2hiint(w[i]));
  }
  if (top >= ((1023u + 300u) << 20)) return false;
#pragma unroll
  for (int i = 0; i < HS + 2; i++) w[i] = div_near(T.idl[i], w[i], rcp_near(w[i]));
  auto convexify = [&]() {
    double sum = w[0];
#pragma unroll
    for (int i = 1; i < HS + 2; i++) sum += w[i];
    sum += 1.0e-20;
    const double y = rcp_near(sum);
#pragma unroll
    for (int i = 0; i < HS + 2; i++) w[i] = div_near(w[i], sum, y);
  };
  convexify();
#pragma unroll
  for (int i = 0; i < HS + 2; i++) {
    const double den = T.map_c[i] + w[i] * T.map_d[i];
    w[i] = div_near(w[i] * (T.map_a[i] - T.map_b[i] * w[i] + w[i] * w[i]), den, rcp_near(den));
  }
  convexify();
  return true;
}
// the high-order candidate's smoothness indicator relaxed towards the others' mean
template <int HS> __device__ __forceinline__ void relax_tv(double (&tv)[HS + 2], double sigma) {
  double avg = tv[0];
#pragma unroll
  for (int i = 1; i < HS + 1; i++) avg += tv[i];
  avg = divk(avg, HS + 1);
  tv[HS + 1] = avg + (tv[HS + 1] - avg) * sigma;
}
template <int ORD>
__device__ __forceinline__ bool weno_gll(const double (&u)[ORD], double (&out)[OrdTraits<ORD>::NGLL]) {
  constexpr int HS = (ORD - 1) / 2;
  constexpr int NG = OrdTraits<ORD>::NGLL;
  const Tables<ORD> &T = tab<ORD>();
  double a[HS + 1][HS + 1], h[ORD];
  if constexpr (ORD == 5) {
    const double p0 = kW24 * u[0], p1 = kW24 * u[1], p3 = kW24 * u[3], p4 = kW24 * u[4];
    const double l0 = __fma_rn(2., p1, -p0), c2 = kW2324 * u[2], t2 = 1.5 * u[2];
    const double h0 = .5 * u[0], h1 = .5 * u[1], h2 = .5 * u[2];
    a[0][0] = l0 + c2;
    a[0][1] = __fma_rn(-2., u[1], h0) + t2;
    a[0][2] = __fma_rn(.5, u[2], h0 - u[1]);
    a[1][0] = (kW1312 * u[2] - p1) - p3;
    a[1][1] = __fma_rn(.5, u[3], -h1);
    a[1][2] = __fma_rn(.5, u[3], h1 - u[2]);
    a[2][0] = __fma_rn(2., p3, c2) - p4;
    a[2][1] = __fma_rn(-.5, u[4], __fma_rn(2., u[3], -t2));
    a[2][2] = __fma_rn(.5, u[4], h2 - u[3]);
    h[0] = (((kH00 * u[0] - kH10 * u[1]) + kH20 * u[2]) - kH10 * u[3]) + kH00 * u[4];
    h[1] = ((kH01 * u[0] - kH11 * u[1]) + kH11 * u[3]) - kH01 * u[4];
    h[2] = __fma_rn(-.0625, u[4], (__fma_rn(-.0625, u[0], .75 * u[1]) - 1.375 * u[2]) + .75 * u[3]);
    h[3] = 2. * (__fma_rn(-2., p3, l0) + p4);
    h[4] = __fma_rn(-4., p3, __fma_rn(.25, u[2], __fma_rn(-4., p1, p0))) + p4;
  } else {
#pragma unroll
    for (int i = 0; i < HS + 1; i++)
#pragma unroll
      for (int ii = 0; ii < HS + 1; ii++) {
        double acc = T.recon[i * ORD * ORD + ii] * u[i];
#pragma unroll
        for (int s = 1; s < HS + 1; s++) {
          if (HS % 2 == 0 && i == HS / 2 && s == HS / 2 && ii % 2 == 1) continue;
          acc += T.recon[(i * ORD + s) * ORD + ii] * u[i + s];
        }
        a[i][ii] = acc;
      }
#pragma unroll
    for (int ii = 0; ii < ORD; ii++) {
      double acc = T.recon[(HS + 1) * ORD * ORD + ii] * u[0];
#pragma unroll
      for (int s = 1; s < ORD; s++) {
        if (s == HS && ii % 2 == 1) continue;
        acc += T.recon[((HS + 1) * ORD + s) * ORD + ii] * u[s];
      }
      h[ii] = acc;
    }
  }
#pragma unroll
  for (int i = 0; i < HS + 1; i++)
#pragma unroll
    for (int ii = 0; ii < HS + 1; ii++) h[ii] -= T.idl[i] * a[i][ii];
#pragma unroll
  for (int ii = 0; ii < ORD; ii++) h[ii] = div_known(h[ii], T.ridl_h, T.ridl_l);
  double tv[HS + 2], w[HS + 2];
#pragma unroll
  for (int i = 0; i < HS + 1; i++) tv[i] = tv_eval<HS + 1>(a[i]);
  tv[HS + 1] = tv_eval<ORD>(h);
  relax_tv<HS>(tv, T.sigma);
  if (!weno_weights<ORD>(tv, w)) return false;
#pragma unroll
  for (int ii = 0; ii < ORD; ii++) {
    if (ii <= HS) {
      double acc = w[0] * a[0][ii];
#pragma unroll
      for (int i = 1; i < HS + 1; i++) acc += w[i] * a[i][ii];
      h[ii] = acc + w[HS + 1] * h[ii];
    } else {
      h[ii] = w[HS + 1] * h[ii];
    }
  }
  const double mid = h[0] + 0.;  // +0 for a zero of either sign, as a sum from +0 gives
#pragma unroll
  for (int ii = 0; ii < NG; ii++) {
    double acc = mid;
    if (ii != NG / 2) {
#pragma unroll
      for (int s = 1; s < ORD; s++) {
        const double c = T.c2g[s * NG + ii];
        if (ii == 0 || ii == NG - 1) acc = __fma_rn((s % 2 && ii == 0) ? -1. / (1 << s) : 1. / (1 << s), h[s], acc);
        else acc += c * h[s];
      }
    }
    out[ii] = acc;
  }
  return true;
}

template <int ORD> struct StenV { double v[ORD]; };
template <int ORD> struct GllV { double v[OrdTraits<ORD>::NGLL]; };
template <int ORD> static __device__ __noinline__ GllV<ORD> reconstruct_gll_general(StenV<ORD> s, bool doweno) {
  GllV<ORD> o;
  reconstruct_gll<ORD>(s.v, o.v, doweno);
  return o;
}
template <int ORD> static __device__ __noinline__ GllV<ORD> reconstruct_gll_call(StenV<ORD> s, bool doweno) {
  GllV<ORD> o;
  if (doweno && weno_gll<ORD>(s.v, o.v)) return o;
  return reconstruct_gll_general<ORD>(s, doweno);
}
template <int ORD, class Sc>
__device__ __forceinline__ void reconstruct_gll_any(const Sc (&sten)[ORD], Sc (&out)[OrdTraits<ORD>::NGLL],
                                                    bool doweno) {
  if constexpr (std::is_same<Sc, double>::value) {
    StenV<ORD> s;
#pragma unroll
    for (int m = 0; m < ORD; m++) s.v[m] = sten[m];
    const GllV<ORD> o = reconstruct_gll_call<ORD>(s, doweno);
#pragma unroll
    for (int ii = 0; ii < OrdTraits<ORD>::NGLL; ii++) out[ii] = o.v[ii];
  } else {
    reconstruct_gll<ORD>(sten, out, doweno);
  }
}

// x + y/k for a small positive integer k: y/k is exact for a power of two, so that on doubles
// the sum is one FMA.
template <class Sc> __device__ __forceinline__ Sc add_divk(const Sc &x, const Sc &y, int k) { return x + divk(y, k); }
__device__ __forceinline__ double add_divk(const double &x, const double &y, int k) {
  if ((k & (k - 1)) == 0) return __fma_rn(1.0 / k, y, x);
  return x + divk(y, k);
}

// sum_s deriv(s, ii) x[s] on doubles, but for the sign of a zero sum: without the leading
// 0 +, and at ord 5, whose matrix is {-3 4 -1; -1 0 1; 1 -4 3}, the products by 0 and +-1; a
// product by 4 is exact and goes into an FMA.
template <int ORD> __device__ __forceinline__ double deriv_sum(const double (&x)[OrdTraits<ORD>::NGLL], int ii) {
  if constexpr (ORD == 5) {
    if (ii == 0) return __fma_rn(4., x[1], -3. * x[0]) - x[2];
    if (ii == 1) return x[2] - x[0];
    return __fma_rn(-4., x[1], x[0]) + 3. * x[2];
  } else {
    const Tables<ORD> &T = tab<ORD>();
    double d = T.deriv[ii] * x[0];
#pragma unroll
    for (int s = 1; s < OrdTraits<ORD>::NGLL; s++) d += T.deriv[s * OrdTraits<ORD>::NGLL + ii] * x[s];
    return d;
  }
}

// -(sum_s deriv(s, ii) x[s]) / dx / k: level k of a variable's time series from its flux x at
// level k-1. The sign of a zero level ends in sums that do not see it (the edge states start
// from level 0, never -0). On doubles the quotient is div_known's, a power-of-two k folded
// into the divisor's pair.
template <int ORD, class Sc>
__device__ __forceinline__ Sc deriv_term(const Sc (&x)[OrdTraits<ORD>::NGLL], int ii, int k, const SweepArgs &A) {
  if constexpr (std::is_same<Sc, double>::value) {
    const double d = deriv_sum<ORD>(x, ii);
    if ((k & (k - 1)) == 0) return div_known(d, A.nrdx_h * (1.0 / k), A.nrdx_l * (1.0 / k));
    return divk(div_known(d, A.nrdx_h, A.nrdx_l), k);
  } else {
    constexpr int NG = OrdTraits<ORD>::NGLL;
    Sc d = 0.;
#pragma unroll
    for (int s = 0; s < NG; s++) d += tab<ORD>().deriv[s * NG + ii] * x[s];
    return divk(divd(-d, rcp_known(A.dxd, A.rdxd)), k);
  }
}

// Reconstruction + ADER differential transform + edge time average of one cell
// (the K2 kernels: Spatial:665-811 x, 1028-1171 y, 1385-1552 z; diffTransformEulerConsX/Y/Z
// at Spatial:1837-2091; compute_timeAvg[_edges] at Spatial:2130-2177).
// sten(v, s) returns stencil value s of variable v. kb is the k index of the cell (z) or of
// the line (x, y). Outputs: the time-averaged left/right edge states and, for z, the
// time-averaged, GLL-weighted gravity source.
// A recorder that keeps nothing (the default): rec.level0(v, ii, x) sees every level-0
// value (after hydrostasis and the wall), for the adjoint's tape; rec.series(q) sees the
// whole ADER series q[v][kt][ii] before the edge time average, for the tracer transport.
struct NoRecord {
  template <class Sc> __device__ __forceinline__ void level0(int, int, const Sc &) const {}
  template <class Q> __device__ __forceinline__ void series(const Q &) const {}
};

template <int ORD, int DIR, class Sten, class Sc, class Rec = NoRecord>
__device__ __forceinline__ void cell_recon(const Sten &sten, int kb, const SweepArgs &A, Sc (&eL)[5], Sc (&eR)[5],
                                           Sc &src_avg, const Rec &rec = Rec()) {
  constexpr int HS = (ORD - 1) / 2;
  constexpr int NG = OrdTraits<ORD>::NGLL;
  constexpr int NA = NG;  // nAder = ngll (Temporal_ader.h:8)
  constexpr int NM = 1 + DIR;  // normal momentum
  const Tables<ORD> &T = tab<ORD>();

  Sc q[5][NA][NG];
#pragma unroll
  for (int v = 0; v < 5; v++) {
    Sc s[ORD];
#pragma unroll
    for (int m = 0; m < ORD; m++) s[m] = sten(v, m);
    const bool doweno = (v == idR || v == idT) ? A.weno_s : A.weno_w;
    reconstruct_gll_any<ORD>(s, q[v][0], doweno);
  }
  // add hydrostasis back on (x/y: cell averages, Spatial:680,697; z: GLL values, :1400,:1421)
#pragma unroll
  for (int ii = 0; ii < NG; ii++) {
    if (DIR == 2) {
      q[idR][0][ii] += A.dens_g[kb * NG + ii];
      q[idT][0][ii] += A.denstheta_g[kb * NG + ii];
    } else {
      q[idR][0][ii] += A.dens_c[HS + kb];
      q[idT][0][ii] += A.denstheta_c[HS + kb];
    }
  }
  if (DIR == 2 && A.bc == BC_WALL) {  // Spatial:1413-1416
    if (kb == A.nz - 1) q[idW][0][NG - 1] = 0;
    if (kb == 0) q[idW][0][0] = 0;
  }
#pragma unroll
  for (int v = 0; v < 5; v++)
#pragma unroll
    for (int ii = 0; ii < NG; ii++) rec.level0(v, ii, q[v][0][ii]);
  // level-0 flux products (Spatial:704-715 and y/z equivalents)
  Sc f[4][NA][NG];
  Sc g[NA][NG];
  Sc srcfill = 0;
  Rcp<Sc> rr[NG];  // the density of each GLL point: divisor of its velocities and products
#pragma unroll
  for (int ii = 0; ii < NG; ii++) {
    const Sc r = q[idR][0][ii];
    rr[ii] = make_rcp<Sc>(r);
    const Sc u = divp(q[idU][0][ii], rr[ii]);
    const Sc v = divp(q[idV][0][ii], rr[ii]);
    const Sc w = divp(q[idW][0][ii], rr[ii]);
    const Sc t = divp(q[idT][0][ii], rr[ii]);
    const Sc vn = NM == 1 ? u : (NM == 2 ? v : w);
    f[0][0][ii] = r * vn * u;
    f[1][0][ii] = r * vn * v;
    f[2][0][ii] = r * vn * w;
    f[3][0][ii] = r * vn * t;
    g[0][ii] = pow_gamma(r * t);
    if (DIR == 2) srcfill = -(q[idR][0][ii] - A.dens_g[kb * NG + ii]) * GRAV;
  }
  // The z source SArray is filled by a scalar assignment inside the kk loop, so every entry
  // holds the kk = ngll-1 value (Spatial:1439).
  Sc sr[NA][NG];
#pragma unroll
  for (int kt = 0; kt < NA; kt++)
#pragma unroll
    for (int ii = 0; ii < NG; ii++) sr[kt][ii] = srcfill;

  // diffTransformEulerCons{X,Y,Z}. Level kt+1 of f and g is still zero where the reference's
  // Cauchy products read it: those terms are left out. The quotients that share no divisor
  // (here and the flux's sound speed) still go through a reciprocal of their own: the compiler's
  // division may call a slow path, and keeping 128 registers across that call cost 32-88
  // bytes of spills (256x256x128 step 4.25 -> 4.08 ms).
#pragma unroll
  for (int kt = 0; kt < NA - 1; kt++) {
    Sc fl[5][NG];  // the flux of each variable
#pragma unroll
    for (int s = 0; s < NG; s++) {
      fl[idR][s] = q[NM][kt][s];
#pragma unroll
      for (int m = 1; m <= 4; m++) fl[m][s] = f[m - 1][kt][s];
      if (DIR == 2 && kt == 0) fl[NM][s] = fl[NM][s] + C0 * g[kt][s] - A.pres_g[kb * NG + s];
      else fl[NM][s] = add_divk(fl[NM][s], C0 * g[kt][s], kt == 0 ? 1 : 2);
    }
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
#pragma unroll
      for (int m = 0; m < 5; m++) q[m][kt + 1][ii] = deriv_term<ORD>(fl[m], ii, kt + 1, A);
      if (DIR == 2) {
        q[idW][kt + 1][ii] = add_divk(q[idW][kt + 1][ii], sr[kt][ii], kt + 1);
        if (A.bc == BC_WALL) {
          if (kb == A.nz - 1) q[idW][kt + 1][NG - 1] = 0;
          if (kb == 0) q[idW][kt + 1][0] = 0;
        }
        sr[kt + 1][ii] = -q[idR][kt + 1][ii] * GRAV;
      }
    }
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      Sc tot[4];
#pragma unroll
      for (int x = 0; x < 4; x++) tot[x] = q[NM][0][ii] * q[x + 1][kt + 1][ii];
#pragma unroll
      for (int ir = 1; ir <= kt + 1; ir++) {
#pragma unroll
        for (int x = 0; x < 4; x++)
          tot[x] += q[NM][ir][ii] * q[x + 1][kt + 1 - ir][ii] - q[idR][ir][ii] * f[x][kt + 1 - ir][ii];
      }
#pragma unroll
      for (int x = 0; x < 4; x++) f[x][kt + 1][ii] = divp(tot[x], rr[ii]);
      const Sc g0 = GAMMA * g[0][ii] * q[idT][kt + 1][ii];
      Sc tg = (kt + 1.) * g0;
#pragma unroll
      for (int ir = 1; ir <= kt; ir++)
        tg += (kt + 1. - ir) * (GAMMA * g[ir][ii] * q[idT][kt + 1 - ir][ii] - q[idT][ir][ii] * g[kt + 1 - ir][ii]);
      g[kt + 1][ii] = divp(g0 + divk(tg, kt + 1), make_rcp<Sc>(q[idT][0][ii]));
    }
  }
  rec.series(q);
  // compute_timeAvg_edges (Spatial:2153-2177)
#pragma unroll
  for (int v = 0; v < 5; v++) {
    Sc l = q[v][0][0], r = q[v][0][NG - 1];
    double dtmult = A.dt;
#pragma unroll
    for (int kt = 1; kt < NA; kt++) {
      l = add_divk(l, q[v][kt][0] * dtmult, kt + 1);
      r = add_divk(r, q[v][kt][NG - 1] * dtmult, kt + 1);
      dtmult *= A.dt;
    }
    eL[v] = l;
    eR[v] = r;
  }
  src_avg = 0.;
  if (DIR == 2) {  // compute_timeAvg (Spatial:2130-2138) + GLL quadrature (Spatial:1489-1496)
    double dtmult = A.dt;
#pragma unroll
    for (int kt = 1; kt < NA; kt++) {
#pragma unroll
      for (int ii = 0; ii < NG; ii++) sr[0][ii] = add_divk(sr[0][ii], sr[kt][ii] * dtmult, kt + 1);
      dtmult *= A.dt;
    }
    Sc sa = 0.;
#pragma unroll
    for (int ii = 0; ii < NG; ii++) sa += sr[0][ii] * T.wts[ii];
    src_avg = sa;
  }
}

// Upwind characteristic Riemann flux at one interface (K4: Spatial:842-902 x, 1202-1260 y,
// 1583-1644 z). The y-direction averages are not divided by density (Spatial:1210-1214).
// kf is the interface's k index for the z hydrostatic pressure subtraction (x, y: the
// line's k, unused).
template <int DIR, int NG, class Sc>
__device__ __forceinline__ void riemann(const Sc (&qL)[5], const Sc (&qR)[5], int kf, const SweepArgs &A,
                                        Sc (&F)[5]) {
  constexpr int TA = DIR == 0 ? 1 : 0;  // first tangential velocity slot
  constexpr int TB = DIR == 2 ? 1 : 2;  // second tangential velocity slot
  constexpr int QN = 1 + DIR, QA = 1 + TA, QB = 1 + TB;
  const Sc r = 0.5 * (qL[0] + qR[0]);
  Sc vel[3], t;
  if (DIR == 1) {
    vel[0] = 0.5 * (qL[1] + qR[1]);
    vel[1] = 0.5 * (qL[2] + qR[2]);
    vel[2] = 0.5 * (qL[3] + qR[3]);
    t = 0.5 * (qL[4] + qR[4]);
  } else {
    const Rcp<Sc> rl = make_rcp<Sc>(qL[0]), rg = make_rcp<Sc>(qR[0]);
    vel[0] = 0.5 * (divp(qL[1], rl) + divp(qR[1], rg));
    vel[1] = 0.5 * (divp(qL[2], rl) + divp(qR[2], rg));
    vel[2] = 0.5 * (divp(qL[3], rl) + divp(qR[3], rg));
    t = 0.5 * (divp(qL[4], rl) + divp(qR[4], rg));
  }
  const Sc p = C0 * pow_gamma(r * t);
  const Sc cs2 = divp(GAMMA * p, make_rcp<Sc>(r));
  const Sc cs = sqrt(cs2);
  const Sc vn = vel[DIR], va = vel[TA], vb = vel[TB];
  const Rcp<Sc> rt = make_rcp<Sc>(t), rt2 = rcp_twice(rt), rc2 = make_rcp<Sc>(2. * cs);
  Sc w1, w2, w3;
  if (vn > 0) {
    w1 = qL[0] - divp(qL[4], rt);
    w2 = qL[QA] - divp(va * qL[4], rt);
    w3 = qL[QB] - divp(vb * qL[4], rt);
  } else {
    w1 = qR[0] - divp(qR[4], rt);
    w2 = qR[QA] - divp(va * qR[4], rt);
    w3 = qR[QB] - divp(vb * qR[4], rt);
  }
  const Sc w5 = divp(vn * qR[0], rc2) - divp(qR[QN], rc2) + divp(qR[4], rt2);
  const Sc w6 = divp(-vn * qL[0], rc2) + divp(qL[QN], rc2) + divp(qL[4], rt2);
  Sc q[5];
  q[0] = w1 + w5 + w6;
  q[QN] = vn * w1 + (vn - cs) * w5 + (vn + cs) * w6;
  q[QA] = w2 + va * w5 + va * w6;
  q[QB] = w3 + vb * w5 + vb * w6;
  q[4] = t * w5 + t * w6;
  const Rcp<Sc> r0 = make_rcp<Sc>(q[0]);
  F[0] = q[QN];
  F[QN] = divp(q[QN] * q[QN], r0) + C0 * pow_gamma(q[4]);
  F[QA] = divp(q[QN] * q[QA], r0);
  F[QB] = divp(q[QN] * q[QB], r0);
  F[4] = divp(q[QN] * q[4], r0);
  if (DIR == 2) {  // Spatial:1628-1629
    if (kf < A.nz) F[idW] -= A.pres_g[kf * NG + 0];
    if (kf == A.nz) F[idW] -= A.pres_g[(A.nz - 1) * NG + NG - 1];
  }
}

}  // namespace awfl
