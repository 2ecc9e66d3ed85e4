// IEEE division by a divisor shared by several quotients, for the FP64 parity path.
//
// The reference divides with the CPU's correctly rounded division everywhere. Several of
// its quotients share a divisor: the four velocity-like ratios and the eight Cauchy-
// product quotients of a GLL point all divide by its density, the WENO normalisations
// divide all weights by one sum, and every tendency divides by dx. Each IEEE division on
// the GPU is a reciprocal-approximation sequence of ~10 FP64 instructions; here the
// correctly rounded reciprocal y = RN(1/b) is formed once, and each quotient a/b costs one
// multiply and four FMAs:
//
//   q0 = RN(a*y);  q1 = RN(q0 + RN(a - b*q0)*y);  q2 = RN(q1 + (a - b*q1)*y)
//
// q1 is within one ulp of a/b (q0 is within 1.5 ulp, and the first correction leaves
// half an ulp plus ~2^-52 ulp), so b*q1 differs from a by an exactly representable
// remainder, and by Markstein's theorem (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990: with y
// within half an ulp of 1/b and q within one ulp of a/b, RN(q + (a - bq)y) = RN(a/b)) q2
// is the correctly rounded quotient -- the IEEE result bit for bit, for operands whose
// quotient, remainder and reciprocal stay in the normal range (the path's values are
// physical quantities of order 1e-20 .. 1e20). A zero dividend returns RN(a*y), which
// carries IEEE's sign of zero. Tested against the GPU's IEEE division on random and
// edge-case operands (tests/test_pow_gpu.py) and through the bit-exact parity tests.
//
// The reciprocal itself comes from Newton iterations on the GPU's reciprocal seed
// (rcp.approx.ftz.f64, 20 bits), one cubic step and one with the residual b*y - 1 exact
// (Markstein, ibid.): RN(1/b) for every significand but all ones, where y is the value on
// the other side of the midpoint that 1/b all but is. No branch, unlike 1.0/b, so that the
// divisions of independent points overlap. Shorter forms where they suffice:
//   divp        divr without the test for a zero dividend: forming the remainder as
//               b*q - a keeps a zero's sign through the corrections for b > 0
//   div_known   a divisor known on the host, 1/b = h + l: two instructions (awfl_recip.h)
//   div_near    one correction instead of two: q0 is within 1.5 ulp, and the corrected
//               value before its rounding within 2^-104 of a/b, so that the quotient is
//               the IEEE one unless a/b lies that close to a rounding midpoint (one pair of
//               operands in ~2^50); for the WENO weights, whose divisions do not share a
//               divisor
//
// The scalar type may also be the tangent-linear Dual; its quotients keep the plain
// division (their value parts are bit-identical either way).
#pragma once

namespace awfl {

template <class Sc> struct Rcp {
  Sc b;
};
template <> struct Rcp<double> {
  double b, y;  // divisor and RN(1/b)
};

__device__ __forceinline__ double rcp_seed(double b) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else  // a host build of this header: a seed of the same 20 bits
  return __hiloint2double(__double2hiint(1.0 / b), 0);
#endif
}
// 1/b within 2^-53 (1 + 2^-5) of itself
__device__ __forceinline__ double rcp_near(double b) {
  const double y = rcp_seed(b), e = __fma_rn(-b, y, 1.0);
  return __fma_rn(__fma_rn(e, e, e), y, y);
}

template <class Sc> __device__ __forceinline__ Rcp<Sc> make_rcp(const Sc &b) { return Rcp<Sc>{b}; }
template <> __device__ __forceinline__ Rcp<double> make_rcp(const double &b) {
  const double y = rcp_near(b);
  return Rcp<double>{b, __fma_rn(__fma_rn(-b, y, 1.0), y, y)};
}
// a divisor whose reciprocal RN(1/b) is already known (host-computed, or a folded constant)
__host__ __device__ __forceinline__ Rcp<double> rcp_known(double b, double y) { return Rcp<double>{b, y}; }

__device__ __forceinline__ double div_markstein(double a, double b, double y) {
  const double q0 = __dmul_rn(a, y);
  const double q1 = __fma_rn(__fma_rn(-q0, b, a), y, q0);
  const double q2 = __fma_rn(__fma_rn(-q1, b, a), y, q1);
  return a == 0.0 ? q0 : q2;
}

__device__ __forceinline__ double div_near(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(q, b, -a), -y, q);
}
__device__ __forceinline__ double div_known(double a, double h, double l) { return __fma_rn(a, h, __dmul_rn(a, l)); }

// a / r.b, correctly rounded, for r.b > 0
template <class Sc> __device__ __forceinline__ Sc divp(const Sc &a, const Rcp<Sc> &r) { return a / r.b; }
__device__ __forceinline__ double divp(const double &a, const Rcp<double> &r) {
  const double q0 = __dmul_rn(a, r.y);
  const double q1 = __fma_rn(__fma_rn(q0, r.b, -a), -r.y, q0);
  return __fma_rn(__fma_rn(q1, r.b, -a), -r.y, q1);
}

// a / r.b, correctly rounded
template <class Sc> __device__ __forceinline__ Sc divr(const Sc &a, const Rcp<Sc> &r) { return a / r.b; }
__device__ __forceinline__ double divr(const double &a, const Rcp<double> &r) { return div_markstein(a, r.b, r.y); }
// The divisions of transported tracer values, correctly rounded for every dividend: nonzero
// ones below 2^-900 in magnitude (where the quotient or the remainder could leave the normal
// range, as values that decay towards zero can) and those from 2^900 on (infinities among
// them, of which the remainder would make a NaN) take the IEEE division itself; a zero
// dividend stays on the short path, whose quotient is IEEE's signed zero
// (the test on the bit pattern, off the FP64 pipe)
__device__ __forceinline__ bool is_extreme(double a) {
  const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
  return h - ((1023u - 900u) << 20) >= (1800u << 20) && (h | (unsigned)__double2loint(a)) != 0;
}
// for r.b > 0, and for a divisor b known on the host as 1/b = h + l
__device__ __forceinline__ double divp_any(double a, const Rcp<double> &r) { return is_extreme(a) ? a / r.b : divp(a, r); }
__device__ __forceinline__ double div_known_any(double a, double b, double h, double l) {
  return is_extreme(a) ? a / b : div_known(a, h, l);
}
// any scalar divided by a double divisor with a known reciprocal
template <class Sc> __device__ __forceinline__ Sc divd(const Sc &a, const Rcp<double> &r) { return a / r.b; }
__device__ __forceinline__ double divd(const double &a, const Rcp<double> &r) { return div_markstein(a, r.b, r.y); }

// a / k for a small positive integer k that is a constant once loops are unrolled: 1 and
// powers of two are exact multiplications; others use the constant-folded reciprocal.
template <class Sc> __device__ __forceinline__ Sc divk(const Sc &a, int k) {
  if (k == 1) return a;
  if ((k & (k - 1)) == 0) return a * (1.0 / k);
  return divd(a, rcp_known((double)k, 1.0 / k));
}
// the same on doubles by div_known (k of two bits: exact for every dividend)
__device__ __forceinline__ double divk(const double &a, int k) {
  if (k == 1) return a;
  if ((k & (k - 1)) == 0) return a * (1.0 / k);
  return k == 3 ? div_known(a, 0x1.5555555555555p-2, 0x1.5555555555555p-56)
                : div_known(a, 0x1.9999999999999p-3, 0x1.3333333333333p-56);  // k == 5
}

// divk for dividends of any magnitude
__device__ __forceinline__ double divk_any(double a, int k) {
  if (k == 1) return a;
  if ((k & (k - 1)) == 0) return a * (1.0 / k);
  return is_extreme(a) ? a / k : divk(a, k);
}

// the reciprocal of 2b from that of b (exact: a power-of-two scaling)
template <class Sc> __device__ __forceinline__ Rcp<Sc> rcp_twice(const Rcp<Sc> &r) { return Rcp<Sc>{2. * r.b}; }
__device__ __forceinline__ Rcp<double> rcp_twice(const Rcp<double> &r) { return Rcp<double>{2. * r.b, 0.5 * r.y}; }

}  // namespace awfl
