// Internal declarations shared by the library's translation units (not part of the ABI).
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

namespace awfl {

namespace adj {
struct SplitArgs;
}
template <class Args> struct EnsList;
struct SweepArgs32;
struct SweepArgs;

// phys_params.h:4-10
constexpr double GRAV = 9.81;
constexpr double C0 = 27.5629410929725921310572974482;
constexpr double GAMMA = 1.40027894002789400278940027894;

enum { idR = 0, idU = 1, idV = 2, idW = 3, idT = 4 };
enum { BC_PERIODIC = 0, BC_WALL = 1 };
enum { MODE_TEND = 0, MODE_APPLY = 1 };

template <int ORD> struct OrdTraits;
template <> struct OrdTraits<5> { static constexpr int NGLL = 3; };
template <> struct OrdTraits<9> { static constexpr int NGLL = 5; };

// Ideal weights and relaxation of ord 5 (WenoLimiter.h:28-90) as compile-time constants (the
// uploaded tables are compared with them), and what the reconstruction in stencil
// differences (FP32: weno_gll5, adjoint: gll5_vjp) derives from them: with d_i = u[i+1] -
// u[i], s_i = d[i+1] - d[i], S = s_0 + s_2, g = s_2 - s_0, the parabolas are u[2] - s_i/24 +
// a_i x + (s_i/2) x^2 with a = (d_1 + s_0/2, d_1 + s_1/2, d_2 - s_2/2).
namespace w5 {
constexpr double kSum = 2 * 1. + 73.564225445964 + 1584.89319246111;
// the weights of the side parabolas, of the centred one and of the bridge polynomial
constexpr double kD0 = 1. / kSum, kD1 = 73.564225445964 / kSum, kD3 = 1584.89319246111 / kSum;
constexpr double kSigma = 0.73564225445964;
// the bridge polynomial (quartic minus the idl-weighted parabolas, over idl[3]) in the
// differences: u[2] + e0, then h1..h4, with e0 = E0S*S + E01*s1, h1 = a_1 + H1*g,
// h2 = H2S*S + H21*s1, h3 = H3*g, h4 = H4*(S - 2 s1)
constexpr double kE0S = (3. / 640 + kD0 / 24) / kD3, kE01 = (-1. / 24 - 6. / 640 + kD1 / 24) / kD3;
constexpr double kH1 = (-5. / 48 + kD0 / 2) / kD3;
constexpr double kH2S = (-1. / 16 - kD0 / 2) / kD3, kH21 = (.625 - kD1 / 2) / kD3;
constexpr double kH3 = 1 / (12 * kD3), kH4 = 1 / (24 * kD3);
}  // namespace w5
// The same for ord 9 (weno_gll9). D_j is the fifth difference over cells j..j+5 of the nine;
// P_i the quartic through the averages of cells i..i+4.
namespace w9 {
constexpr double kSum = 2 * 1. + 2 * 2.15766927997459 + 2.40224886796286 + 1136.12697719888;
constexpr double kSigma = 0.0288539981181442;
__host__ __device__ constexpr double ideal(int i) {
  return (i == 5 ? 1136.12697719888 : (i == 2 ? 2.40224886796286 : (i % 2 ? 2.15766927997459 : 1.))) / kSum;
}
constexpr double kX1 = 0.32732683535398857;  // sqrt(3/7)/2: the GLL points are 0, +-kX1, +-1/2
struct Poly {
  double c[9];
  __host__ __device__ constexpr double even(double x) const { return c[0] + x * x * (c[2] + x * x * (c[4] + x * x * (c[6] + x * x * c[8]))); }
  __host__ __device__ constexpr double odd(double x) const { return x * (c[1] + x * x * (c[3] + x * x * (c[5] + x * x * c[7]))); }
};
// P_3 - P_2 = D_2 N(x), P_4 - P_3 = D_3 M(x), P_1 - P_2 = -D_1 N(-x), P_0 - P_1 = -D_0 M(-x)
constexpr Poly kN = {{3. / 640, 5. / 48, -1. / 16, -1. / 12, 1. / 24, 0, 0, 0, 0}};
constexpr Poly kM = {{-71. / 1920, -3. / 16, 7. / 16, -1. / 4, 1. / 24, 0, 0, 0, 0}};
// The octic less P_2: coefficient i is kFa[i] (D_2 -+ D_1) + kFb[i] (D_3 -+ D_0), minus for
// even i; the bridge polynomial less P_2 (the octic minus the ideal(0..4)-weighted P_i, over
// ideal(5)) likewise with kHa, kHb.
constexpr Poly kFa = {{-725. / 688128, 5911. / 215040, 1889. / 129024, -701. / 23040, -127. / 9216, 11. / 1920, 1. / 384,
                       -1. / 10080, -1. / 13440}};
constexpr Poly kFb = {{35. / 294912, -3229. / 645120, -3229. / 1935360, 47. / 7680, 47. / 27648, -1. / 640, -7. / 17280,
                       1. / 10080, 1. / 40320}};
constexpr Poly bridge(const Poly &f, double d, const Poly &p) {
  Poly r = {};
  for (int i = 0; i < 9; i++) r.c[i] = (f.c[i] - d * p.c[i]) / ideal(5);
  return r;
}
// d/dx at the GLL points -1/2, -kX1, 0 from the values at all five; those of the mirror points
// are each other's reverse negated
struct Deriv {
  double d[3][5];
};
constexpr Deriv kD = {{{-10, 13.51300497744848, -16. / 3, 2.8203283558848535, -1},
                       {-2.4819805060619657, 0, 3.4914862437758787, -1.5275252316519454, 0.5180194939380343},
                       {.75, -2.6731691553909065, 0, 2.6731691553909065, -.75}}};
constexpr Poly kHa = bridge(kFa, ideal(0) + ideal(1), kN), kHb = bridge(kFb, ideal(0), kM);
}  // namespace w9

// Constant tables (Spatial:274-315), one set per order, uploaded once per device.
template <int ORD> struct Tables {
  static constexpr int HS = (ORD - 1) / 2;
  static constexpr int NG = OrdTraits<ORD>::NGLL;
  double recon[ORD * ORD * ORD];  // weno_sten_to_coefs(i, s, ii)
  double c2g[ORD * NG];            // coefs_to_gll(s, ii)
  double s2g[ORD * NG];            // sten_to_gll(s, ii)
  double deriv[NG * NG];          // derivMatrix(s, ii)
  double idl[HS + 2];
  double sigma;
  double wts[NG];                 // gllWts_ngll
  double ridl;                    // RN(1/idl[HS+1]), the bridge polynomial's divisor
  // derived (host::complete_tables, awfl_recip.h): 1/idl[HS+1] = ridl_h + ridl_l, and the
  // constants of the weights' mapping, d + d*d, 3d, d*d and 1 - 2d for d = idl[i]
  double ridl_h, ridl_l;
  double map_a[HS + 2], map_b[HS + 2], map_c[HS + 2], map_d[HS + 2];
};

// Entries of the ord-5 reconstruction tables that the FP64 kernels hold as literals
// (compared with the tables when they are uploaded): the others are zero or a power of two
// times one of these.
constexpr double kW24 = 0x1.5555555555555p-5;     // 1/24
constexpr double kW2324 = 0x1.eaaaaaaaaaaabp-1;   // 23/24
constexpr double kW1312 = 0x1.1555555555555p+0;   // 13/12
constexpr double kH00 = 0x1.3333333333333p-8;     // 3/640
constexpr double kH10 = 0x1.eeeeeeeeeeeefp-5;     // 29/480
constexpr double kH20 = 0x1.1c88888888889p+0;     // 1067/960
constexpr double kH01 = 0x1.aaaaaaaaaaaabp-4;     // 5/48
constexpr double kH11 = 0x1.6aaaaaaaaaaabp-1;     // 17/24

// Per-line constants of one sweep.
struct SweepArgs {
  double *state;   // (5, nz+2hs, ny+2hs, nx+2hs)
  double *tend;    // (5, nz, ny, nx) for MODE_TEND
  long plane;      // tangent-linear sweep: offset of the tangent plane in state (else 0)
  int nx, ny, nz;
  int bc;          // BC along the sweep direction
  int weno_s, weno_w, sim2d, mode;
  int nsm;         // SMs of the device (the launch picks the tile shape by it)
  double dxd;      // dx, dy or dz
  double rdxd;     // RN(1/dxd)
  double nrdx_h, nrdx_l;  // -1/dxd = nrdx_h + nrdx_l (div_known's pair, awfl_recip.h)
  double dt;
  const double *dens_c, *denstheta_c;             // hyDensCells, hyDensThetaCells (nz+2hs)
  const double *dens_g, *denstheta_g, *pres_g;    // hyDensGLL, hyDensThetaGLL, hyPressureGLL (nz*ngll)
  // x sweeps of a slab of a larger grid: the halo columns of a slab end that borders
  // another slab, [5][nz][ny][hs+1] values per side (side 0: positions -(hs+1)..-1, the
  // lower neighbour's last columns; side 1: positions nx..nx+hs, the upper neighbour's
  // first); nullptr for an end with the grid's own boundary condition
  const double *xh[2];
};


struct InitLaunch {
  void *state;
  float *state32, *comp32;  // FP32 contexts: value and Kahan planes (state unused)
  int nx, ny, nz, hs, ord;
  int xoff, nx_global;  // a slab: its first cell's global x index; the grid's nx (0: not a slab)
  double dx, dy, dz, xlen, ylen, zlen;
  int data_spec, sim2d, kind, shape;
  double x0, y0, z0, xrad, yrad, zrad, amp, pwr, noise_amp;
  unsigned long long seed;
  int noise_kind;
  const double *dens_c;
  double pts[9], wts[9];
};

// FP32 form (awfl_fp32.cu)
struct SweepArgs32;
cudaError_t launch_sweep_fp32(int ord, int dir, const SweepArgs32 &A, cudaStream_t st);
// The tile shape that a sweep's launch takes (chunk C x lines W) and its staging, for the plain
// sweeps, the tracer splits' and the adjoint's recording ones.
struct SweepChoice {
  int C, W, tma;
};
SweepChoice sweep_choice_fp32(int ord, int dir, const SweepArgs32 &A);
SweepChoice sweep_choice_tracers32(int ord, int dir, const SweepArgs32 &A);
SweepChoice sweep_choice_fp64(int ord, int dir, const SweepArgs &A);
SweepChoice sweep_choice_tracers(int ord, int dir, const SweepArgs &A);
SweepChoice sweep_choice_rec(int ord, int dir, const SweepArgs &A);
cudaError_t launch_apply_fp32(float *state, float *comp, const float *tend, float dt, int nx, int ny, int nz, int hs,
                              cudaStream_t st);
cudaError_t upload_tables_fp32(int ord, const double *recon, const double *c2g, const double *s2g,
                               const double *deriv, const double *idl, double sigma, const double *wts);

// Ensemble sweeps (awfl_ens32.cu, awfl_ens64.cu): launch (occ == nullptr) or query the
// occupancy of tile shape `shape` (awfl_ens.cuh).
cudaError_t ens_run_fp32(int ord, int dir, int shape, const EnsList<SweepArgs32> *E, int grid, int *occ,
                         cudaStream_t st);
cudaError_t ens_run_fp64(int ord, int dir, int shape, const EnsList<SweepArgs> *E, int grid, int *occ,
                         cudaStream_t st);
cudaError_t upload_tables_ens32(int ord, const double *recon, const double *c2g, const double *s2g,
                                const double *deriv, const double *idl, double sigma, const double *wts);
cudaError_t upload_tables_ens64(int ord, const void *tab, size_t bytes);

// Error message for entry points without a context (awfl_capi.cu).
void set_unbound_error(const char *msg);

// FP64 translation unit (awfl_fp64.cu)
cudaError_t upload_tables_fp64(int ord, const void *tab, size_t bytes);
cudaError_t launch_sweep_fp64(int ord, int dir, const SweepArgs &A, cudaStream_t st);
// Differentiation TU (awfl_adjoint.cu)
cudaError_t launch_sweep_tlm(int ord, int dir, const SweepArgs &A, cudaStream_t st);
// FP64 sweep that also records level-0 values and edges of every cell into A.tend
cudaError_t launch_sweep_rec(int ord, int dir, const SweepArgs &A, cudaStream_t st);
cudaError_t upload_tables_adj(int ord, const void *tab, size_t bytes);
// Tracer transport of the FP64 path (awfl_tracers.cu): one split of state (fused, MODE_APPLY
// arithmetic of awfl_split) and tracers; scratch holds tracer_scratch_bytes(..., 8) bytes.
// io: TRC_IN_DIVIDED, the tracers arrive divided by the current density (no division at
// the start); TRC_OUT_DIVIDED, the update leaves the interior divided by the post-split
// density (for the next split of the same step).
enum { TRC_IN_DIVIDED = 1, TRC_OUT_DIVIDED = 2 };
cudaError_t launch_split_tracers(int ord, int dir, const SweepArgs &A, double *tracers, int ntr,
                                 unsigned long long pos, double *scratch, int io, cudaStream_t st);
// Record layout of a tracer split (both precisions; planes of ncell cells, then of nfmax
// faces): R (NG*(NG-1): levels 0..NG-2 of the density series), U (NG*(NG-1): the same of
// the normal-momentum series), D (1: the pre-split rho', the stencil centre), Y (NG: 1/rho
// of the GLL points), then per face F0 (the Riemann mass flux), VN (the velocity that
// picks the upwind side), UN (the limiter's velocity), RUP (the upwind side's density),
// YUP (1/RUP). The series' last level only enters the tracer series' last momentum-flux
// level, which no edge reads, so it is not recorded. The FP32 form recomputes Y and YUP
// (its reciprocals are single fast-reciprocal instructions) and leaves their planes unused.
template <int NG> __host__ __device__ constexpr long trc_series_planes() { return (long)NG * (NG - 1); }
template <int NG> __host__ __device__ constexpr long trc_cell_planes() { return 2 * trc_series_planes<NG>() + 1 + NG; }
// scratch of one tracer split: records and fluxes of elem bytes each, and the line flags
size_t tracer_scratch_bytes(int ord, int nx, int ny, int nz, int ntr, int elem);
cudaError_t upload_tables_tracers(int ord, const void *tab, size_t bytes);
// The same in the FP32 form (awfl_tracers32.cu): the FP32 state split with FP64 tracers;
// scratch holds tracer_scratch_bytes(..., 4) bytes; dens_c: rho_h rows (FP64).
cudaError_t launch_split_tracers32(int ord, int dir, const SweepArgs32 &A, const double *dens_c, double dt,
                                   double dxd, double *tracers, int ntr, unsigned long long pos, float *scratch,
                                   int io, cudaStream_t st);
cudaError_t upload_tables_tracers32(int ord, const double *recon, const double *c2g, const double *s2g,
                                    const double *deriv, const double *idl, double sigma, const double *wts);
// Adjoint reverse sweeps (awfl_adjrev.cu)
cudaError_t launch_adjoint_split(int ord, int dir, const adj::SplitArgs &A, int need_edges, cudaStream_t st);
cudaError_t launch_zero_halo(double *lam, int nx, int ny, int nz, int hs, cudaStream_t st);
cudaError_t upload_tables_adjrev(int ord, const void *tab, size_t bytes);
cudaError_t launch_apply_fp64(double *state, const double *tend, double dt, int nx, int ny, int nz, int hs,
                              cudaStream_t st);
// x += dt*0 on the interior of nplanes planes (the sim2d y split's apply of zero tendencies)
cudaError_t launch_add_zero_fp64(double *p, int nplanes, int nx, int ny, int nz, int hs, cudaStream_t st);
// The largest max|u +- cs|, |v +- cs|, |w +- cs| of a state into result[0..2]; acc: four
// device words, zero before the first call and after each.
cudaError_t launch_cfl(const void *state, int fp32, const double *dens_c, const double *denstheta_c, int nx, int ny,
                       int nz, int hs, int nsm, unsigned long long *acc, double *result, cudaStream_t st);
cudaError_t launch_init_state_fp64(const InitLaunch &L, cudaStream_t st);
cudaError_t launch_init_tracers_fp64(const InitLaunch &L, int ntr, cudaStream_t st);
cudaError_t launch_tracer_fields(const void *state, int fp32, long plane, const double *dens_c,
                                 const double *tracers, int ntr, int nx, int ny, int nz, int hs, int nsm, double *out,
                                 cudaStream_t st);
// interior sums x dV (partials[nblk*5] -> out[5], fixed order) and the bad-cell count
cudaError_t launch_state_sums(const void *state, int fp32, long plane, int nx, int ny, int nz, int hs, double dv,
                              double *partials, int nblk, double *out, cudaStream_t st);
cudaError_t launch_check_state(const void *state, int fp32, long plane, const double *dens_c, int nx, int ny,
                               int nz, int hs, int nsm, unsigned long long *count, cudaStream_t st);
cudaError_t run_fma_peak(int kind, int nsm, double *tflops);  // 0 FP64, 1 FP32, 2 paired FP32
cudaError_t launch_output_fields(const void *state, int fp32, long plane, const double *dens_c,
                                 const double *denstheta_c, const double *pres_c, int nx, int ny, int nz, int hs,
                                 int nsm, double *out, cudaStream_t st);
cudaError_t launch_selftest_pow(const double *x, double y, double *out, long n, int mode, cudaStream_t st);
// The hs+1 first and last interior x columns of every variable of a state (value plane)
// into send = [2][5][nz][ny][hs+1] elements of the state's type (esz 8 or 4).
cudaError_t launch_slab_pack(const void *state, int esz, int nx, int ny, int nz, int hs, void *send, cudaStream_t st);

}  // namespace awfl
