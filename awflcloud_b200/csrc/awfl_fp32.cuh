// FP32 precision form of the AWFL Euler-3D ADER/WENO step: device functions and the
// sweep policy P32, sm_100a.
//
// Same scheme as the reference (Spatial_euler3d_cons_expl_cart_fv_Agrid.h, WenoLimiter.h,
// Temporal_ader.h), same line-sweep kernel skeleton as the FP64 path (awfl_sweep.cuh), but
// FP32 arithmetic (FMA contraction and fast division/sqrt allowed) with the scheme's
// cancellation-prone pieces rewritten in perturbation form, so that single precision
// keeps its ~1e-7 relative accuracy on the perturbation fields:
//
//  * State: FP32 perturbations from the hydrostatic background (rho', rho*u, rho*v, rho*w,
//    (rho*theta)'), like the reference's own state, plus a second FP32 plane holding the
//    Kahan compensation of every stage update (state += dt*tend, Temporal_ader.h:63-65).
//  * Background: computed in FP64 on the host (the reference's profiles) and used as FP32
//    per-row (x/y: cell averages) or per-GLL-point/per-face (z) constants.
//  * Pressure: C0*(rho*theta)^gamma = P_h * (1 + B(x)), x = (rho*theta)'/(rho*theta)_h,
//    B(x) = (1+x)^gamma - 1 by its binomial series (|x| < 0.05; expm1(gamma*log1p(x))
//    otherwise), P_h = C0*(rho*theta)_h^gamma in FP64. Only P_h*B enters derivatives and
//    fluxes: a row-constant P_h cancels exactly in the x/y divergence, and in z it is the
//    reference's own hydrostatic subtraction (Spatial:2042, :1628-1629).
//  * (rho*theta)^gamma time derivatives are carried scaled by (rho*theta)_h^gamma.
//  * Edge states are carried as perturbations; the Riemann mass flux is evaluated as
//    vn*q1 + cs*(w6 - w5) with w6 - w5 expressed through L-R differences of perturbations,
//    instead of vn*w1 + (vn-cs)*w5 + (vn+cs)*w6 whose O(rho*cs) terms cancel.
//  * The CFL time step reads the FP32 state but computes in FP64.
// Every expression equals the reference's in exact arithmetic, including its quirks (y
// averages not divided by density, the filled z gravity source, the z wall).
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "awfl_internal.h"
#include "awfl_fp32_args.h"
#include "awfl_pow.cuh"
#include "awfl_recip.h"
#include "awfl_sweep.cuh"

namespace awfl {

// Fast reciprocal (MUFU-based, ~1 ulp): the FP32 form's divisions.
__device__ __forceinline__ float frcp(float x) { return __fdividef(1.f, x); }

constexpr float GAMMAF = (float)GAMMA;
constexpr float GRAVF = (float)GRAV;

// Binomial coefficients C(gamma, n), n = 1..6, of (1+x)^gamma.
constexpr double kB1 = GAMMA;
constexpr double kB2 = kB1 * (GAMMA - 1.0) / 2.0;
constexpr double kB3 = kB2 * (GAMMA - 2.0) / 3.0;
constexpr double kB4 = kB3 * (GAMMA - 3.0) / 4.0;
constexpr double kB5 = kB4 * (GAMMA - 4.0) / 5.0;
constexpr double kB6 = kB5 * (GAMMA - 5.0) / 6.0;

// (1+x)^gamma - 1
__device__ __forceinline__ float binom_gamma_m1(float x) {
  if (fabsf(x) < 0.05f) {
    float p = (float)kB6;
    p = fmaf(p, x, (float)kB5);
    p = fmaf(p, x, (float)kB4);
    p = fmaf(p, x, (float)kB3);
    p = fmaf(p, x, (float)kB2);
    p = fmaf(p, x, (float)kB1);
    return p * x;
  }
  return expm1f(GAMMAF * log1pf(x));
}

template <int ORD> struct Tables32 {
  static constexpr int NG = OrdTraits<ORD>::NGLL;
  float s2g[ORD * NG];
  float deriv[NG * NG];
  float wts[NG];
};
// One copy per translation unit that includes this header (awfl_fp32.cu, awfl_ens32.cu),
// each uploaded by upload_tables32_here.
static __constant__ Tables32<5> c32_tab5;
static __constant__ Tables32<9> c32_tab9;
template <int ORD> __device__ __forceinline__ const Tables32<ORD> &tab32();
template <> __device__ __forceinline__ const Tables32<5> &tab32<5>() { return c32_tab5; }
template <> __device__ __forceinline__ const Tables32<9> &tab32<9>() { return c32_tab9; }

// Two independent FP32 lanes evaluated with the paired sm_100 instructions (FFMA2, FMUL2,
// FADD2: one instruction, two results, each rounded like the scalar operation), so that
// two variables' reconstructions issue half the instructions. Divisions stay per lane.
struct F2 {
  float2 v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(float2 x) : v(x) {}
  __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
  __device__ __forceinline__ explicit F2(double c) : v(make_float2((float)c, (float)c)) {}
  __device__ __forceinline__ explicit F2(float c) : v(make_float2(c, c)) {}
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {  // FADD2 with a negated operand (no intrinsic for it)
  unsigned long long x, y, z;
  __builtin_memcpy(&x, &a.v, 8);
  __builtin_memcpy(&y, &b.v, 8);
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
  F2 r;
  __builtin_memcpy(&r.v, &z, 8);
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator*(float c, F2 b) { return F2(__fmul2_rn(make_float2(c, c), b.v)); }
__device__ __forceinline__ F2 operator*(F2 a, float c) { return F2(__fmul2_rn(a.v, make_float2(c, c))); }
__device__ __forceinline__ F2 operator+(F2 a, float c) { return F2(__fadd2_rn(a.v, make_float2(c, c))); }
__device__ __forceinline__ F2 operator+(float c, F2 a) { return F2(__fadd2_rn(make_float2(c, c), a.v)); }
__device__ __forceinline__ F2 &operator+=(F2 &a, F2 b) { return a = a + b; }

// fma / reciprocal / quotient on either scalar type
__device__ __forceinline__ float fmaT(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ F2 fmaT(float a, F2 b, F2 c) { return F2(__ffma2_rn(make_float2(a, a), b.v, c.v)); }
__device__ __forceinline__ F2 fmaT(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ F2 fmaT(F2 a, float b, F2 c) { return F2(__ffma2_rn(a.v, make_float2(b, b), c.v)); }
__device__ __forceinline__ float rcpT(float x) { return frcp(x); }
__device__ __forceinline__ F2 rcpT(F2 x) { return F2(frcp(x.v.x), frcp(x.v.y)); }

}  // namespace awfl

#include "awfl_weno32.h"

namespace awfl {

template <int ORD, class T>
__device__ __forceinline__ void reconstruct_gll32(const T (&sten)[ORD], T (&out)[OrdTraits<ORD>::NGLL], bool doweno) {
  constexpr int NG = OrdTraits<ORD>::NGLL;
  const Tables32<ORD> &Tb = tab32<ORD>();
  if (doweno) {
    if constexpr (ORD == 5) weno_gll5(sten, out);
    else weno_gll9(sten, out);
  } else {
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      T tmp = T(0.f);
#pragma unroll
      for (int s = 0; s < ORD; s++) tmp = fmaT(Tb.s2g[s * NG + ii], sten[s], tmp);
      out[ii] = tmp;
    }
  }
}

// (1+x)^gamma - 1 on two lanes
__device__ __forceinline__ F2 binom_gamma_m1(F2 x) {
  if (fmaxf(fabsf(x.v.x), fabsf(x.v.y)) < 0.05f) {
    F2 p = fmaT(F2((float)kB6), x, F2((float)kB5));
    p = fmaT(p, x, F2((float)kB4));
    p = fmaT(p, x, F2((float)kB3));
    p = fmaT(p, x, F2((float)kB2));
    p = fmaT(p, x, F2((float)kB1));
    return p * x;
  }
  return F2(binom_gamma_m1(x.v.x), binom_gamma_m1(x.v.y));
}

// The values of one quantity at a cell's GLL points: the mirror points (ii, NG-1-ii) as the
// two lanes of the paired FP32 instructions, the centre alone. All points of a cell go
// through the same operations, so the time series takes 2 instructions where it took 3 (ord
// 5; 3 for 5 at ord 9), with no lane to broadcast.
template <int NG> struct Pts {
  F2 p[NG / 2];
  float c;
  __device__ __forceinline__ float get(int ii) const {
    return ii == NG / 2 ? c : (ii < NG / 2 ? p[ii].v.x : p[NG - 1 - ii].v.y);
  }
  __device__ __forceinline__ void set(int ii, float x) {
    if (ii == NG / 2) c = x;
    else if (ii < NG / 2) p[ii].v.x = x;
    else p[NG - 1 - ii].v.y = x;
  }
};
template <int NG, class F> __device__ __forceinline__ Pts<NG> each(const F &f) {
  Pts<NG> r;
#pragma unroll
  for (int i = 0; i < NG / 2; i++) r.p[i] = f([i](const Pts<NG> &x) -> const F2 & { return x.p[i]; });
  r.c = f([](const Pts<NG> &x) -> const float & { return x.c; });
  return r;
}
template <int NG> __device__ __forceinline__ Pts<NG> operator+(const Pts<NG> &a, const Pts<NG> &b) {
  return each<NG>([&](auto e) { return e(a) + e(b); });
}
template <int NG> __device__ __forceinline__ Pts<NG> operator*(const Pts<NG> &a, const Pts<NG> &b) {
  return each<NG>([&](auto e) { return e(a) * e(b); });
}
template <int NG> __device__ __forceinline__ Pts<NG> operator*(float a, const Pts<NG> &b) {
  return each<NG>([&](auto e) { return a * e(b); });
}
template <int NG> __device__ __forceinline__ Pts<NG> operator-(const Pts<NG> &a, const Pts<NG> &b) {
  return each<NG>([&](auto e) { return e(a) - e(b); });
}
template <int NG> __device__ __forceinline__ Pts<NG> fmaT(const Pts<NG> &a, const Pts<NG> &b, const Pts<NG> &c) {
  return each<NG>([&](auto e) { return fmaT(e(a), e(b), e(c)); });
}
template <int NG> __device__ __forceinline__ Pts<NG> fmaT(float a, const Pts<NG> &b, const Pts<NG> &c) {
  return each<NG>([&](auto e) { return fmaT(a, e(b), e(c)); });
}
template <int NG> __device__ __forceinline__ Pts<NG> rcpT(const Pts<NG> &a) {
  return each<NG>([&](auto e) { return rcpT(e(a)); });
}
template <int NG> __device__ __forceinline__ Pts<NG> binom_gamma_m1(const Pts<NG> &a) {
  return each<NG>([&](auto e) { return binom_gamma_m1(e(a)); });
}
template <int NG> __device__ __forceinline__ Pts<NG> same(float x) {
  return each<NG>([&](auto e) { return std::decay_t<decltype(e(Pts<NG>()))>(x); });
}
// sum_s deriv(s, ii) x[s], times sc, at every point (the matrix has no centre weight at the
// centre; at ord 5 it is {-3 4 -1; -1 0 1; 1 -4 3})
template <int ORD> __device__ __forceinline__ Pts<OrdTraits<ORD>::NGLL> deriv32(const Pts<OrdTraits<ORD>::NGLL> &x, float sc) {
  constexpr int NG = OrdTraits<ORD>::NGLL;
  Pts<NG> r;
  if constexpr (ORD == 5) {
    const float x0 = x.get(0), x1 = x.c, x2 = x.get(2);
    r.set(0, fmaf(4.f, x1, fmaf(-3.f, x0, -x2)));
    r.set(1, x2 - x0);
    r.set(2, fmaf(-4.f, x1, fmaf(3.f, x2, x0)));
  } else {
    // the rows of mirror points are each other's reverse negated: lane y takes the same
    // coefficients on the reversed values, and -sc (128x128x64 step 0.483 -> 0.476 ms)
    constexpr w9::Deriv kD = w9::kD;
    auto rev = [](F2 a) { return F2(a.v.y, a.v.x); };
    const F2 p0 = x.p[0], p1 = x.p[1], m0 = rev(p0), m1 = rev(p1), cc = F2(x.c), pm = F2(sc, -sc);
    r.p[0] = pm * fmaT((float)kD.d[0][0], p0, fmaT((float)kD.d[0][1], p1, fmaT((float)kD.d[0][2], cc, fmaT((float)kD.d[0][3], m1, (float)kD.d[0][4] * m0))));
    r.p[1] = pm * fmaT((float)kD.d[1][0], p0, fmaT((float)kD.d[1][2], cc, fmaT((float)kD.d[1][3], m1, (float)kD.d[1][4] * m0)));
    const F2 h = fmaT((float)kD.d[2][0], p0, (float)kD.d[2][1] * p1);
    r.c = sc * (h.v.x - h.v.y);
    return r;
  }
  return sc * r;
}

// A recorder that keeps nothing (the default of cell_recon32): rec.series32(q, rtot) sees
// the whole ADER series q[v][kt] (level 0 as perturbations) and the total density of the GLL
// points before the edge time average, for the tracer transport.
struct NoRecord32 {
  template <class Q, class Rt> __device__ __forceinline__ void series32(const Q &, const Rt &) const {}
};

template <int ORD, int DIR, class Sten, class Rec = NoRecord32>
__device__ __forceinline__ void cell_recon32(const Sten &sten, int kb, const SweepArgs32 &A, float (&eL)[5],
                                             float (&eR)[5], float &src_avg, const Rec &rec = Rec()) {
  constexpr int HS = (ORD - 1) / 2;
  constexpr int NG = OrdTraits<ORD>::NGLL;
  constexpr int NA = NG;
  constexpr int NM = 1 + DIR;
  using V = Pts<NG>;
  const Tables32<ORD> &T = tab32<ORD>();

  V q[5][NA];  // level 0: rho' (perturbation), rho*u/v/w, (rho*theta)' (perturbation)
  // (rho', (rho theta)') and (rho u, rho v) in pairs on the paired FP32 instructions
#pragma unroll
  for (int pr = 0; pr < 2; pr++) {
    const int va = pr == 0 ? idR : idU, vb = pr == 0 ? idT : idV;
    F2 s2[ORD], o2[NG];
#pragma unroll
    for (int m = 0; m < ORD; m++) s2[m] = F2(sten(va, m), sten(vb, m));
    reconstruct_gll32<ORD>(s2, o2, pr == 0 ? A.weno_s : A.weno_w);
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      q[va][0].set(ii, o2[ii].v.x);
      q[vb][0].set(ii, o2[ii].v.y);
    }
  }
  {
    float s[ORD], o[NG];
#pragma unroll
    for (int m = 0; m < ORD; m++) s[m] = sten(idW, m);
    reconstruct_gll32<ORD>(s, o, A.weno_w);
#pragma unroll
    for (int ii = 0; ii < NG; ii++) q[idW][0].set(ii, o[ii]);
  }
  const bool wall0 = DIR == 2 && A.bc == BC_WALL && kb == 0, wallN = DIR == 2 && A.bc == BC_WALL && kb == A.nz - 1;
  auto wall = [&](V &w) {  // Spatial:1413-1416
    if (wallN) w.set(NG - 1, 0.f);
    if (wall0) w.set(0, 0.f);
  };
  if (DIR == 2) wall(q[idW][0]);
  V rb, rtb, irtb, Pbg;  // background
  if (DIR == 2) {
#pragma unroll
    for (int ii = 0; ii < NG; ii++) {
      rb.set(ii, A.bg.rho_g[kb * NG + ii]);
      rtb.set(ii, A.bg.rt_g[kb * NG + ii]);
      irtb.set(ii, A.bg.irt_g[kb * NG + ii]);
      Pbg.set(ii, A.bg.p_g[kb * NG + ii]);
    }
  } else {
    rb = same<NG>(A.bg.rho_c[HS + kb]);
    rtb = same<NG>(A.bg.rt_c[HS + kb]);
    irtb = same<NG>(A.bg.irt_c[HS + kb]);
    Pbg = same<NG>(A.bg.p_c[HS + kb]);
  }
  const V rtot = rb + q[idR][0], rttot = rtb + q[idT][0];
  const V ir = rcpT(rtot);
  V f[4][NA];
  V g[NA];  // (rho theta)^gamma series / (rho theta)_h^gamma
#pragma unroll
  for (int m = 1; m <= 3; m++) f[m - 1][0] = q[NM][0] * (q[m][0] * ir);
  f[3][0] = q[NM][0] * (rttot * ir);
  g[0] = binom_gamma_m1(q[idT][0] * irtb);  // B(x); the scaled series starts at 1 + B
  // z gravity source: every entry of the first level holds the kk = ngll-1 value (Spatial:1439)
  const float srcfill = DIR == 2 ? -q[idR][0].get(NG - 1) * GRAVF : 0.f;
  float sa = srcfill;  // its time average, GLL-weighted (the weights sum to one)
  float dtm = A.dt;

  // diffTransformEulerCons{X,Y,Z} (Spatial:1837-2091)
#pragma unroll
  for (int kt = 0; kt < NA - 1; kt++) {
    const float sc = -A.inv_dxd * (1.0f / (kt + 1));
    q[idR][kt + 1] = deriv32<ORD>(q[NM][kt], sc);
#pragma unroll
    for (int m = 1; m <= 4; m++) {
      V fl = f[m - 1][kt];
      if (m == NM) fl = fmaT(kt == 0 ? Pbg : 0.5f * Pbg, g[kt], fl);
      q[m][kt + 1] = deriv32<ORD>(fl, sc);
    }
    if (DIR == 2) {
      if (kt == 0) q[idW][1] = q[idW][1] + same<NG>(srcfill);
      else q[idW][kt + 1] = fmaT(-GRAVF / (kt + 1), q[idR][kt], q[idW][kt + 1]);
      wall(q[idW][kt + 1]);
      float w = 0.f;
#pragma unroll
      for (int ii = 0; ii < NG; ii++) w = fmaf(T.wts[ii], q[idR][kt + 1].get(ii), w);
      sa = fmaf(dtm * (-GRAVF / (kt + 2)), w, sa);
      dtm *= A.dt;
    }
    if (kt + 1 < NA - 1) {  // products needed by the next level only
      auto Q = [&](int m, int l) -> const V & { return l == 0 && m == idR ? rtot : (l == 0 && m == idT ? rttot : q[m][l]); };
      // Cauchy products of the series; the not-yet-known level kt+1 of f and g enters
      // with a zero coefficient and is left out (an IEEE multiply by zero is not
      // removed by the compiler)
#pragma unroll
      for (int x = 0; x < 4; x++) {
        V tot = q[NM][0] * Q(x + 1, kt + 1);
        V sub = q[idR][1] * f[x][kt];
#pragma unroll
        for (int i = 1; i <= kt + 1; i++) {
          tot = fmaT(q[NM][i], Q(x + 1, kt + 1 - i), tot);
          if (i > 1) sub = fmaT(q[idR][i], f[x][kt + 1 - i], sub);
        }
        f[x][kt + 1] = (tot - sub) * ir;
      }
      // scaled (rho theta)^gamma: g~(0) = 1 + B
      const V one = same<NG>(1.f);
      auto Gs = [&](int l) -> V { return l == 0 ? one + g[0] : g[l]; };
      V tg = (2.f * GAMMAF) * (Gs(0) * q[idT][kt + 1]);  // the leading term of the sum, and outside it
#pragma unroll
      for (int i = 1; i <= kt; i++) {
        const V term = GAMMAF * (g[i] * q[idT][kt + 1 - i]) - q[idT][i] * Gs(kt + 1 - i);
        tg = fmaT((kt + 1.f - i) / (kt + 1.f), term, tg);
      }
      g[kt + 1] = tg * rcpT(rttot);
    }
  }
  rec.series32(q, rtot);
  // compute_timeAvg_edges on perturbations (Spatial:2153-2177): both edges as one pair
#pragma unroll
  for (int v = 0; v < 5; v++) {
    F2 e = q[v][0].p[0];
    float dtmult = A.dt;
#pragma unroll
    for (int kt = 1; kt < NA; kt++) {
      e = fmaT(dtmult * (1.0f / (kt + 1)), q[v][kt].p[0], e);
      dtmult *= A.dt;
    }
    eL[v] = e.v.x;
    eR[v] = e.v.y;
  }
  src_avg = sa;
}

// Upwind Riemann flux in FP32 perturbation form (Spatial:842-902, 1202-1260, 1583-1644).
template <int DIR, int NG>
__device__ __forceinline__ void riemann32(const float (&qL)[5], const float (&qR)[5], int kf, const SweepArgs32 &A,
                                          float (&F)[5]) {
  constexpr int TA = DIR == 0 ? 1 : 0;
  constexpr int TB = DIR == 2 ? 1 : 2;
  constexpr int QN = 1 + DIR, QA = 1 + TA, QB = 1 + TB;
  constexpr int HS = NG == 3 ? 2 : 4;
  // side backgrounds (rho, rho*theta) and the face's pressure background
  float bLr, bLt, bRr, bRt, rtf, irtf, pf;
  if (DIR == 2) {
    const int fL = (kf == 0 && A.bc == BC_PERIODIC) ? A.nz : kf;
    const int fR = (kf == A.nz && A.bc == BC_PERIODIC) ? 0 : kf;
    bLr = A.bg.rho_f[fL]; bLt = A.bg.rt_f[fL];
    bRr = A.bg.rho_f[fR]; bRt = A.bg.rt_f[fR];
    rtf = A.bg.rt_f[kf]; irtf = A.bg.irt_f[kf]; pf = A.bg.p_f[kf];
  } else {
    (void)HS;
    const int k = kf;  // x/y sweeps: the line's k
    bLr = bRr = A.bg.rho_c[HS + k];
    bLt = bRt = A.bg.rt_c[HS + k];
    rtf = bLt; irtf = A.bg.irt_c[HS + k]; pf = A.bg.p_c[HS + k];
  }
  const float rL = bLr + qL[0], rR = bRr + qR[0];
  const float tL = bLt + qL[4], tR = bRt + qR[4];  // total rho*theta
  const float irL = frcp(rL), irR = frcp(rR);
  const float r = 0.5f * (rL + rR);
  float vel[3], t, uL = 0.f, uR = 0.f;
  if (DIR == 1) {  // y: averages not divided by density (Spatial:1210-1214)
    vel[0] = 0.5f * (qL[1] + qR[1]);
    vel[1] = 0.5f * (qL[2] + qR[2]);
    vel[2] = 0.5f * (qL[3] + qR[3]);
    t = 0.5f * (tL + tR);
  } else {
    uL = qL[QN] * irL;
    uR = qR[QN] * irR;
#pragma unroll
    for (int m = 0; m < 3; m++) vel[m] = m == DIR ? 0.5f * (uL + uR) : 0.5f * fmaf(qL[1 + m], irL, qR[1 + m] * irR);
    t = 0.5f * fmaf(tL, irL, tR * irR);
  }
  // cs^2 = gamma*C0*(r t)^gamma / r with (r t)^gamma = (rho theta)_f^gamma (1 + B)
  const float rt = r * t;
  const float cs2 = GAMMAF * pf * (1.f + binom_gamma_m1((rt - rtf) * irtf)) * frcp(r);
  const float cs = sqrtf(cs2);
  const float ics2 = 0.5f * frcp(cs), it2 = 0.5f * frcp(t);
  const float vn = vel[DIR], va = vel[TA], vb = vel[TB];
  float w1, w2, w3;
  if (vn > 0) {
    const float a = tL * (2.f * it2);
    w1 = rL - a;
    w2 = qL[QA] - va * a;
    w3 = qL[QB] - vb * a;
  } else {
    const float a = tR * (2.f * it2);
    w1 = rR - a;
    w2 = qR[QA] - va * a;
    w3 = qR[QB] - vb * a;
  }
  const float dq1 = (bRr - bLr) + (qR[0] - qL[0]);  // q1R - q1L
  const float dqn = qR[QN] - qL[QN];
  const float dq5 = (bLt - bRt) + (qL[4] - qR[4]);  // q5L - q5R
  const float S = fmaf(vn, dq1, -dqn) * ics2 + (tL + tR) * it2;  // w5 + w6
  float d65;                                                        // w6 - w5
  if (DIR == 1) d65 = fmaf(-vn, rL + rR, qL[QN] + qR[QN]) * ics2 + dq5 * it2;
  else d65 = (-dq1) * (uL - uR) * 0.5f * ics2 + dq5 * it2;
  const float q1 = w1 + S;
  const float qn = fmaf(vn, q1, cs * d65);
  const float qa = fmaf(va, S, w2);
  const float qb = fmaf(vb, S, w3);
  const float q5 = t * S;
  // (rho theta) perturbation of the upwind state relative to the face background
  const float q5p = t * fmaf(vn, dq1, -dqn) * ics2 + (0.5f * ((bLt + bRt) - 2.f * rtf) + 0.5f * (qL[4] + qR[4]));
  const float iq1 = frcp(q1);
  F[0] = qn;
  F[QN] = fmaf(qn * qn, iq1, pf * binom_gamma_m1(q5p * irtf));
  F[QA] = qn * qa * iq1;
  F[QB] = qn * qb * iq1;
  F[4] = qn * q5 * iq1;
}

struct P32 {
  using Real = float;
  static constexpr int kWdiv = 1;
  static constexpr bool kAsyncRing = true;
  // interior chunks are staged by tiled TMA: the single-grid sweep reads the tensor map
  // from its kernel parameter, the ensemble's persistent sweep from the work list in
  // global memory (its shared-memory copy of the arguments is no place for one)
  static constexpr bool kTmaRing = true;
  static constexpr bool kSlab = true;  // awfl_split_slab
  static bool prepare_tma(SweepArgs32 &A, int ord, int dir, int C, int W) {
    return prepare_sweep_map32(A, ord, dir, C, W);
  }
  static __device__ __forceinline__ const void *tma_map(const SweepArgs32 &A) { return &A.tmap; }
  static __device__ __forceinline__ const void *tma_map_global(const SweepArgs32 &shared_copy,
                                                               const SweepArgs32 *in_global) {
    return shared_copy.tma ? (const void *)&in_global->tmap : nullptr;
  }
  static __device__ __forceinline__ void flag_timeout(const SweepArgs32 &A) {
    if (A.err) atomicOr(A.err, 1u);
  }
  // ord 5: five CTAs of 128 threads per SM (86-93 registers): 256x256x128 step 1.160 ms,
  // against 1.200 at the compiler's 115 (four) and 1.177 at six (80); the small-grid shapes
  // and the x-slab sweep at four (awfl_sweep.cuh)
  // ord 9: three (168 registers by cp.async: the large grids' shapes spill nothing, the small
  // ones' and the x-slab sweep 24-52 bytes): 128x128x64 step 0.476 ms at two CTAs, 0.433 at
  // three. The ensembles' TMA kernels take the same bound for 128-thread tiles (40-60 bytes of
  // spills, 230 registers at 64 threads; awfl_ensemble_tune picks)
  static constexpr int min_blocks(int ord) { return ord == 5 ? 5 : 3; }
  using Args = SweepArgs32;
  // where the base shape's rows come by TMA (`tma`), those that it cannot address (16-byte
  // pitch) come by cp.async: 107 instead of about 85 us for the x split of 130x100x70
  static double base_factor(const Args &A, bool tma) { return tma && A.nx % 4 ? 1.25 : 1.0; }
  // the Kahan compensations of the cell's five variables, loaded before the reconstruction
  struct Aux {
    float c[5];
  };
  static __device__ __forceinline__ void load_aux(const Args &A, long g0, long sv, Aux &aux) {
#pragma unroll
    for (int v = 0; v < 5; v++) aux.c[v] = A.comp[g0 + v * sv];
  }

  template <int ORD, int DIR, class S>
  static __device__ __forceinline__ void recon(const S &sten, int kb, const Args &A, float (&eL)[5], float (&eR)[5],
                                               float &src, long) {
    cell_recon32<ORD, DIR>(sten, kb, A, eL, eR, src);
  }
  template <int DIR, int NG>
  static __device__ __forceinline__ void flux(const float (&qL)[5], const float (&qR)[5], int kf, const Args &A,
                                              float (&F)[5]) {
    riemann32<DIR, NG>(qL, qR, kf, A, F);
  }
  template <int DIR>
  static __device__ __forceinline__ float tendency(int v, float Fl, float Fr, float sa, const Args &A) {
    const float d = (Fl - Fr) * A.inv_dxd;
    if (DIR == 0) return (A.sim2d && v == idV) ? 0.f : d;
    if (DIR == 1) return d;
    return (A.sim2d && v == idV) ? 0.f : (v == idW ? sa + d : d);
  }
  // Kahan-compensated stage update: s += dt*tnd with the running compensation c.
  static __device__ __forceinline__ void apply(const Args &A, long g, float orig, float tnd, const Aux &aux, int v) {
    const float y = A.dt * tnd - aux.c[v];
    const float t = orig + y;
    A.comp[g] = __fsub_rn(__fsub_rn(t, orig), y);
    A.state[g] = t;
  }
  static __device__ __forceinline__ float load(const Args &A, long g) { return A.state[g]; }
  static __device__ __forceinline__ void store(const Args &A, long g, float x) { A.state[g] = x; }
  static __device__ __forceinline__ void store_tend(const Args &A, long g, float x) { A.tend[g] = x; }
};

// Single-grid sweep shapes of the FP32 form, ord 5 (chunk C x lines W, 128 threads): x 8 x 16,
// y 8 x 16, z 4 x 32 (y/z: a warp = 32/C lines x C positions). Measured at 256x256x128, five
// CTAs per SM, us per split: x 8x16 374, 16x8 372, 8x8 (64 threads) 425; y 8x16 385, 4x32
// 401, 8x8 385, 4x16 418; z 4x32 388, 8x16 408, 4x64 511, 4x16 438.
// (z at 254x256x128, whose rows TMA could not address: 385, 8x16 428.)
template <> struct PolicyShape<P32, 5, 0> { static constexpr int C = 8, W = 16; };
template <> struct PolicyShape<P32, 5, 1> { static constexpr int C = 8, W = 16; };
// Ord 9, three CTAs of 128 threads (128x128x64, us): x 32 x 4 138, 8 x 16 154; y 16 x 8 141,
// 8 x 16 157; z 8 x 16 141, 16 x 8 149. With the shapes for small grids, against 32 x 2, 8 x 16
// and 8 x 16 for all: step 32x32x16 45 -> 33 us, 64x64x32 92 -> 77, 97x61x45 197 (two CTAs) -> 150,
// 400x1x200 184 (two) -> 48, 128x128x64 433 -> 418.
template <> struct PolicyShape<P32, 9, 0> { static constexpr int C = 32, W = 4; };
template <> struct PolicyShape<P32, 9, 1> { static constexpr int C = 16, W = 8; };
// The shapes for small grids (PolicyShapes, awfl_sweep.cuh).
template <int DIR> struct PolicyShapes<P32, 9, DIR> {
  static constexpr int n = DIR == 0 ? 2 : 3;
  static constexpr int C[3] = {DIR == 1 ? 8 : 16, DIR == 0 ? 128 : 32, 128}, W[3] = {DIR == 1 ? 16 : 8, DIR == 0 ? 1 : 4, 1};
  static constexpr double factor[3] = {DIR == 0 ? 1.0 : (DIR == 1 ? 0.92 : 1.12), DIR == 0 ? 1.15 : (DIR == 1 ? 1.12 : 1.25),
                                       1.4};
};
template <int DIR> struct PolicyShapes<P32, 5, DIR> {
  static constexpr int n = 4;
  static constexpr int C[4] = {DIR == 2 ? 8 : 4, 16, 32, 128}, W[4] = {DIR == 2 ? 16 : 32, 8, 4, 1};
  static constexpr double factor[4] = {DIR == 2 ? 1.1 : 1.0, DIR == 0 ? 1.15 : (DIR == 1 ? 1.15 : 1.3),
                                       DIR == 0 ? 1.25 : (DIR == 1 ? 1.6 : 1.8), DIR == 0 ? 1.5 : 2.5};
};

// Uploads the FP32 tables into this translation unit's constant memory.
static inline cudaError_t upload_tables32_here(int ord, const double *recon, const double *c2g, const double *s2g,
                                               const double *deriv, const double *idl, double sigma,
                                               const double *wts) {
  auto fill = [&](auto &t, int o, int g) {
    for (int i = 0; i < o * g; i++) t.s2g[i] = (float)s2g[i];
    for (int i = 0; i < g * g; i++) t.deriv[i] = (float)deriv[i];
    for (int i = 0; i < g; i++) t.wts[i] = (float)wts[i];
  };
  if (!host::fp32_forms_match(ord, recon, c2g, deriv, idl, sigma)) return cudaErrorInvalidValue;
  if (ord == 5) {
    Tables32<5> t;
    fill(t, 5, 3);
    return cudaMemcpyToSymbol(c32_tab5, &t, sizeof t);
  }
  Tables32<9> t;
  fill(t, 9, 5);
  return cudaMemcpyToSymbol(c32_tab9, &t, sizeof t);
}

}  // namespace awfl
