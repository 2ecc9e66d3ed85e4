// FP64 sweep policy P64 (the reference's arithmetic) over the line-sweep skeleton.
// Included by the translation units that instantiate FP64 sweeps (awfl_fp64.cu,
// awfl_ens64.cu); each has its own copy of the constant tables (awfl_device.cuh).
#pragma once

#include "awfl_device.cuh"
#include "awfl_internal.h"
#include "awfl_sweep.cuh"

namespace awfl {

// ------------------------------------------------------------------------------------
// FP64 physics policy of the line sweep (awfl_sweep.cuh): the reference's arithmetic.
// ------------------------------------------------------------------------------------

struct P64 {
  using Real = double;
  static constexpr int kWdiv = 1;
  static constexpr bool kAsyncRing = true;
  static constexpr bool kTmaRing = false;
  static constexpr bool kSlab = true;  // awfl_split_slab
  // ord 5: 4 CTAs per SM (<= 128 registers), more warps to hide the FP64 latency
  // (measured +17%); ord 9 would spill heavily at that budget
#ifndef AWFL_P64_MIN_BLOCKS_ORD5
#define AWFL_P64_MIN_BLOCKS_ORD5 4
#endif
  static constexpr int min_blocks(int ord) { return ord == 5 ? AWFL_P64_MIN_BLOCKS_ORD5 : 1; }
  using Args = SweepArgs;
  static double base_factor(const Args &, bool) { return 1.0; }
  struct Aux {};
  static __device__ __forceinline__ void load_aux(const Args &, long, long, Aux &) {}

  template <int ORD, int DIR, class S>
  static __device__ __forceinline__ void recon(const S &sten, int kb, const Args &A, double (&eL)[5],
                                               double (&eR)[5], double &src, long) {
    cell_recon<ORD, DIR>(sten, kb, A, eL, eR, src);
  }

  template <int DIR, int NG>
  static __device__ __forceinline__ void flux(const double (&qL)[5], const double (&qR)[5], int kf, const Args &A,
                                              double (&F)[5]) {
    riemann<DIR, NG>(qL, qR, kf, A, F);
  }

  // K5 divergence (Spatial:940-956, 1298-1310, 1680-1696): z adds onto the gravity source.
  template <int DIR>
  static __device__ __forceinline__ double tendency(int v, double Fl, double Fr, double sa, const Args &A) {
    const double d = div_known(Fr - Fl, A.nrdx_h, A.nrdx_l);  // -(Fr - Fl) / dx
    if (DIR == 0) return (A.sim2d && v == idV) ? 0.0 : d;
    if (DIR == 1) return d;
    return (A.sim2d && v == idV) ? 0.0 : (v == idW ? sa : 0.0) + d;
  }

  // K6 apply (Temporal_ader.h:63-65)
  static __device__ __forceinline__ void apply(const Args &A, long g, double orig, double tnd, const Aux &, int) {
    A.state[g] = orig + A.dt * tnd;
  }
  static __device__ __forceinline__ double load(const Args &A, long g) { return A.state[g]; }
  static __device__ __forceinline__ void store(const Args &A, long g, double x) { A.state[g] = x; }
  static __device__ __forceinline__ void store_tend(const Args &A, long g, double x) { A.tend[g] = x; }
};

// Single-grid sweep shapes of the FP64 path, ord 5 (chunk x lines; measured at
// 256x256x128 with the current kernel against x 32 x 4 / 8 x 16 and y, z 4 x 32 / 16 x 8,
// which took 1-2% longer): x 16 x 8, y and z 8 x 16. The macros let a build try others.
#ifndef AWFL_P64_XC
#define AWFL_P64_XC 16
#define AWFL_P64_XW 8
#endif
#ifndef AWFL_P64_YC
#define AWFL_P64_YC 8
#define AWFL_P64_YW 16
#endif
#ifndef AWFL_P64_ZC
#define AWFL_P64_ZC 8
#define AWFL_P64_ZW 16
#endif
template <> struct PolicyShape<P64, 5, 0> { static constexpr int C = AWFL_P64_XC, W = AWFL_P64_XW; };
template <> struct PolicyShape<P64, 5, 1> { static constexpr int C = AWFL_P64_YC, W = AWFL_P64_YW; };
template <> struct PolicyShape<P64, 5, 2> { static constexpr int C = AWFL_P64_ZC, W = AWFL_P64_ZW; };

// The shapes for small grids, x, y and z alike (PolicyShapes, awfl_sweep.cuh).
template <int ORD, int DIR> struct SmallShapes { static constexpr int n = 0; };
template <int DIR> struct SmallShapes<5, DIR> {
  static constexpr int n = 3;
  static constexpr int C[3] = {DIR == 0 ? 8 : 16, 32, 128}, W[3] = {DIR == 0 ? 16 : 8, 4, 1};
  static constexpr double factor[3] = {1.0, 1.0, 1.1};
};
// Ord 9: x 32 x 4 (128x128x64, us: 734; 32 x 2 770, 16 x 8 761), and for y and z 8 x 16
// (840 873), 16 x 8 (795 828) or 32 x 4 (756 826), whichever pads the lines less and fills the
// chip. Step, all in 32 x 2 (x) or 8 x 16 -> the rule, us: 32x32x16 172 -> 94, 64x64x32 408
// -> 341, 97x61x45 1004 -> 753, 400x1x200 805 -> 207, 128x128x64 2494 -> 2295, 256x256x64
// 10130 -> 9415; 80x50x48 571 -> 576.
template <> struct PolicyShape<P64, 9, 0> { static constexpr int C = 32, W = 4; };
template <int DIR> struct SmallShapes<9, DIR> {
  static constexpr int n = DIR == 0 ? 2 : 3;
  static constexpr int C[3] = {16, DIR == 0 ? 128 : 32, 128}, W[3] = {8, DIR == 0 ? 1 : 4, 1};
  static constexpr double factor[3] = {DIR == 2 ? 0.99 : 1.0, DIR == 0 ? 1.1 : (DIR == 1 ? 1.0 : 0.93), 1.2};
};
template <int ORD, int DIR> struct PolicyShapes<P64, ORD, DIR> : SmallShapes<ORD, DIR> {};
// The same for the recording policies, whose 20-odd record planes are written along x: a y
// or z shape of few lines spreads each store over as many rows as it has cells of a line
// (128x128x64 with tracers, y split, 8 x 16 / 16 x 8 / 32 x 4: 445 / 467 / 497 us; 64x64x32:
// 121 / 107 / 98).
template <int ORD, int DIR> struct RecordShapes { static constexpr int n = 0; };
template <int DIR> struct RecordShapes<5, DIR> : SmallShapes<5, DIR> {
  static constexpr double factor[3] = {DIR == 0 ? 1.0 : (DIR == 1 ? 1.1 : 1.2), DIR == 0 ? 1.0 : (DIR == 1 ? 1.2 : 1.3),
                                       DIR == 0 ? 1.1 : 1.5};
};

}  // namespace awfl
