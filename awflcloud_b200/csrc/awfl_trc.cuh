// Tracer transport kernels shared by the FP64 path (awfl_tracers.cu) and the FP32 form
// (awfl_tracers32.cu): the along-line geometry of a split, the in-place division of the
// tracers by the pre-split density (Spatial:624-627), the positivity limiter with the
// result of the reference's serial face order (Spatial:904-935, 1262-1293, 1646-1677) and
// the tendency and update (Spatial:948-955; Temporal_ader.h:67-69).
//
// The including translation unit defines, before including this header, its tracer
// argument struct TA with
//   A                the split's sweep arguments (nx, ny, nz, bc),
//   using Flux       the flux type (double: FP64 path; float: FP32 form),
//   tr               double*, (ntr, nz+2hs, ny+2hs, nx+2hs): the tracers,
//   ntr, pos         the tracer count and the positive-definite bits,
//   D                const Flux*, (ncell): the recorded pre-split rho',
//   F0, VN, UN       const Flux*, (nface) each: per face, recorded by the state's sweep, the
//                    Riemann mass flux, the velocity that picks the upwind side and the
//                    limiter's velocity,
//   TF, TF2          Flux*, (ntr, nface): the unscaled and the limited tracer fluxes,
//   flag, list, count  int*: per line, whether the limiter redoes it in serial order; the
//                    list of those lines and its length (zeroed with the flags before
//                    the limiter runs),
// and these overloads for it:
//   trc_divisor(T, hs, k, g)        the divisor of the division: rho' + rho_h (double)
//   trc_dens(T, hs, k)              rho_h of row k as the limiter adds it to a recorded rho'
//   limit_face(T, F, f1, f2, q, d)  a face's scaled flux from its upwind cell's two faces
//   trc_div_up(T, a, fi)            a divided by the upwind density of face fi (recorded)
//   trc_update(T, q, hs, k, c, Fl, Fr)
//                                   the updated tracer of cell c (row k) from its divided
//                                   value q and its limited face fluxes: q*rho + dt*tend
// Everything here sits in an anonymous namespace: each translation unit compiles its own
// copy with its own floating-point flags.
#pragma once

#include <cuda_runtime.h>

#include "awfl_div.cuh"
#include "awfl_internal.h"

namespace awfl {
namespace {

template <class R> __device__ __forceinline__ R dmax(R a, R b) { return a > b ? a : b; }
template <class R> __device__ __forceinline__ R dmin(R a, R b) { return a < b ? a : b; }

// Along-direction geometry of one split: cells (k, j, i); p = the index along DIR.
template <int DIR> struct Geo {
  int nx, ny, nz, hs;
  long sy, sz, sv;  // state strides (halo-inclusive)
  template <class SA> __device__ Geo(const SA &A, int hs_) : nx(A.nx), ny(A.ny), nz(A.nz), hs(hs_) {
    sy = nx + 2 * hs;
    sz = (long)(ny + 2 * hs) * sy;
    sv = (long)(nz + 2 * hs) * sz;
  }
  __device__ int n() const { return DIR == 0 ? nx : (DIR == 1 ? ny : nz); }
  __device__ long cell(int k, int j, int i) const { return ((long)k * ny + j) * nx + i; }
  // state offset of interior cell (k, j, i)
  __device__ long g(int k, int j, int i) const { return (long)(hs + k) * sz + (long)(hs + j) * sy + hs + i; }
  // face index (faces along DIR: n+1 per line)
  __device__ long face(int k, int j, int i) const {
    if (DIR == 0) return ((long)k * ny + j) * (nx + 1) + i;
    if (DIR == 1) return ((long)k * (ny + 1) + j) * nx + i;
    return ((long)k * ny + j) * nx + i;
  }
  __device__ long nface() const {
    return (long)(nz + (DIR == 2)) * (ny + (DIR == 1)) * (nx + (DIR == 0));
  }
  __device__ long nlines() const {
    return DIR == 0 ? (long)nz * ny : (DIR == 1 ? (long)nz * nx : (long)ny * nx);
  }
  // cell (k, j, i) moved to index p along DIR
  __device__ void at(int k, int j, int i, int p, int &kk, int &jj, int &ii) const {
    kk = DIR == 2 ? p : k;
    jj = DIR == 1 ? p : j;
    ii = DIR == 0 ? p : i;
  }
};

// Index p (possibly in the halo) -> the interior index whose value the halo holds, and
// whether it is a wall halo (normal momentum zero).
__device__ __forceinline__ int halo_src(int p, int n, int bc, bool &wall) {
  wall = false;
  if (p >= 0 && p < n) return p;
  if (bc == BC_PERIODIC) return p < 0 ? p + n : p - n;
  wall = true;
  return p < 0 ? 0 : n - 1;
}

// (k, j, i) of a flat index over extents ex (fastest) and ey, in 32-bit arithmetic: the
// tracer path's grids hold fewer than 2^31 cells and faces (the launchers check)
__device__ __forceinline__ void unflat(unsigned x, unsigned ex, unsigned ey, int &k, int &j, int &i) {
  const unsigned r = x / ex;
  const unsigned kk = r / ey;
  i = (int)(x - r * ex);
  j = (int)(r - kk * ey);
  k = (int)kk;
}

// The tracer kernels walk a grid of cells or faces plane by plane: a block's 128 threads on
// consecutive indices of a plane (x fastest), blockIdx.y on the planes (all of them but the
// 65536th plane of faces, which the loop brings back): one 32-bit division per thread where a
// flat index took two, and flat indices in 32 bits. With the pointers stepped from tracer to
// tracer, integer instructions, which were 40% of these kernels', are halved (128x128x64,
// three tracers, us per split: limiter 35.6 -> 26.6, update 27.4 -> 24.7).
inline dim3 plane_grid(long plane, int planes) { return dim3((unsigned)((plane + 127) / 128), (unsigned)(planes < 65535 ? planes : 65535)); }

template <int DIR> __device__ __forceinline__ long line_of(int k, int j, int i, int ny, int nx) {
  return DIR == 0 ? (long)k * ny + j : (DIR == 1 ? (long)k * nx + i : (long)j * nx + i);
}

// The tracer fluxes (Spatial:891-901, 1249-1259, 1633-1643) of the faces cell p of a line
// is upwind of, from its time-averaged tracer edges tl (left) and tr (right): face flux =
// the state's mass flux F0 times the upwind edge over the upwind density RUP, both recorded
// by the sweep at the face; VN > 0 makes the left cell upwind. Edge BCs (Spatial:816-837):
// periodic faces 0 and n both see (right edge of cell n-1, left edge of cell 0); at a wall
// both sides of face 0 see cell 0's left edge, of face n cell n-1's right edge. Every face
// of the line is written by exactly one cell (face 0 and face n of a periodic line by one
// cell each). fl: this cell's left face, fs: the face stride along the line, f0: face 0.
// Which faces those are, decided once per cell for all its tracers: the left face (fed by
// tl), the right face (tr), and on a periodic line face 0 (tr of cell n-1) and face n
// (tl of cell 0).
struct UpwindFaces {
  long fl, fr, f0, fn;
  bool pl, pr, p0, pn;
};
template <class TA>
__device__ __forceinline__ UpwindFaces upwind_faces(const TA &T, int p, int n, bool periodic, long fl, long fs,
                                                    long f0) {
  UpwindFaces U;
  U.fl = fl;
  U.fr = fl + fs;
  U.f0 = f0;
  U.fn = f0 + (long)n * fs;
  U.pl = (p == 0 && !periodic) || !(T.VN[fl] > 0);
  U.pr = (p == n - 1 && !periodic) || T.VN[U.fr] > 0;
  U.p0 = periodic && p == n - 1 && T.VN[f0] > 0;      // face 0, across the wrap
  U.pn = periodic && p == 0 && !(T.VN[U.fn] > 0);     // face n, likewise
  return U;
}
template <class Fx, class TA>
__device__ __forceinline__ void put_upwind_fluxes(const TA &T, Fx *TF, const UpwindFaces &U, Fx tl, Fx tr) {
  auto put = [&](long fi, Fx t) { TF[fi] = trc_div_up(T, T.F0[fi] * t, fi); };
  if (U.pl) put(U.fl, tl);
  if (U.pr) put(U.fr, tr);
  if (U.p0) put(U.f0, tr);
  if (U.pn) put(U.fn, tl);
}
template <class Fx, class TA>
__device__ __forceinline__ void write_upwind_fluxes(const TA &T, Fx *TF, int p, int n, bool periodic, long fl,
                                                    long fs, long f0, Fx tl, Fx tr) {
  put_upwind_fluxes<Fx>(T, TF, upwind_faces(T, p, n, periodic, fl, fs, f0), tl, tr);
}

// tracers /= (rho' + rho_h) on the interior cells, with the state before the split
// (Spatial:624-627). The halos are not touched: every kernel of the split maps a halo
// position to the interior cell whose value it holds.
#ifndef AWFL_TRC_DIVIDE_MINB
#define AWFL_TRC_DIVIDE_MINB 1
#endif
template <class TA>
__global__ void __launch_bounds__(128, AWFL_TRC_DIVIDE_MINB) tracer_divide_kernel(TA T, int hs) {
  const Geo<0> G(T.A, hs);
  const unsigned q = blockIdx.x * 128u + threadIdx.x;
  if (q >= (unsigned)G.nx * G.ny) return;
  const int j = (int)(q / (unsigned)G.nx), i = (int)(q - (unsigned)j * G.nx);
  for (int k = blockIdx.y; k < G.nz; k += gridDim.y) {
    const long g = G.g(k, j, i);
    const Rcp<double> r = make_rcp<double>(trc_divisor(T, hs, k, idR * G.sv + g));  // shared by the tracers
    double *t = T.tr + g;
    for (int l = 0; l < T.ntr; l++, t += G.sv) *t = divp_any(*t, r);
  }
}

// Positivity limiter in the reference's serial loop order: along each line the faces are
// visited in increasing order and each is scaled in place by its upwind cell's factor,
// computed from that cell's two faces as they stand at that moment (the face behind
// already scaled, the face itself and the ones ahead not yet) -- the one defined result of
// the reference's in-place parallel_for, the one its CPU build gives when the loop runs in
// order. Faces of other lines are never read.
//
// The serial order matters only where a face reads a face that has been scaled: face f > 0
// with un > 0 reads face f-1 (as min(., 0)), and face n with un < 0 reads faces 0 (min) and
// 1 (max). So tracer_limit_faces_kernel limits every face at once with all reads unscaled,
// and flags the lines where some scaled face changed a value another face reads; on the
// other lines that result is the serial one, face by face (by induction along the line:
// every read sees the value the serial loop would). tracer_limit_lines_kernel redoes the
// flagged lines serially. Equal reads are compared as values: a read that differs only in
// the sign of a zero leaves the factor unchanged (it enters as f2 - f1 + eps).
#ifndef AWFL_TRC_LIMIT_MINB
#define AWFL_TRC_LIMIT_MINB 1
#endif
template <class TA, int DIR>
__global__ void __launch_bounds__(128, AWFL_TRC_LIMIT_MINB) tracer_limit_faces_kernel(TA T, int hs) {
  using Fx = typename TA::Flux;
  const Geo<DIR> G(T.A, hs);
  const int nf = (int)G.nface();  // < 2^31 (the launchers check)
  const unsigned fx = G.nx + (DIR == 0), fy = G.ny + (DIR == 1), fz = G.nz + (DIR == 2);
  const unsigned pq = blockIdx.x * 128u + threadIdx.x;
  if (pq >= fx * fy) return;
  const int j = (int)(pq / fx), i = (int)(pq - (unsigned)j * fx);
  const int n = G.n();
  // strides along the line: faces and cells (flat), state (halo-inclusive)
  const int fs = DIR == 0 ? 1 : (DIR == 1 ? G.nx : G.nx * G.ny);
  const long gsd = DIR == 0 ? 1 : (DIR == 1 ? G.sy : G.sz);
  for (int k = blockIdx.y; k < (int)fz; k += gridDim.y) {
    const int fi = (int)(k * (fx * fy) + pq);
    const int f = DIR == 0 ? i : (DIR == 1 ? j : k);
    const int f0 = fi - f * fs;  // the line's face 0
    int k0, j0, i0;
    G.at(k, j, i, 0, k0, j0, i0);
    const Fx un = T.UN[fi];
    // the upwind cell and the two faces that bound it (as offsets from this one)
    int c = -1;
    if (un > 0) c = f == 0 ? n - 1 : f - 1;
    else if (un < 0) c = f == n ? 0 : f;
    const int ia = (c - f) * fs, ib = ia + fs;
    Fx dens = 0;
    if (c >= 0) dens = T.D[(int)G.cell(k0, j0, i0) + c * fs] + trc_dens(T, hs, DIR == 2 ? c : k);
    // the faces that read this one: f+1 when it is upwinded from cell f; face n reads
    // faces 0 (min) and 1 (max) when it is upwinded from cell 0 -- through the factor of
    // the reader's upwind cell (f, resp. 0), which is zero whatever it reads when the cell
    // holds no tracer
    const bool read_next = f < n && T.UN[fi + fs] > 0;
    const bool read_by_n = (f == 0 || (f == 1 && n >= 2)) && T.UN[f0 + n * fs] < 0;
    bool chained = false;
    const Fx *TF = T.TF + fi;
    Fx *TF2 = T.TF2 + fi;
    const double *t0 = T.tr + G.g(k0, j0, i0), *tc = t0 + (c > 0 ? c * gsd : 0L);
    for (int l = 0; l < T.ntr; l++) {
      const Fx F = *TF;
      Fx out = F;
      if (((T.pos >> l) & 1ull) && c >= 0) {
        const double q = *tc;
        if (F == Fx(0) && ((unsigned)__double2hiint(q) & 0x7fffffffu) < ((1023u + 100u) << 20)) {
          // a zero times the factor, whose sign is the tracer's: a tracer absent here reads no
          // other face and divides nothing (not so an infinite one or a NaN, which the FP32
          // form's clamped edges turn into zero fluxes: their factor makes it a NaN again)
          out = __double2hiint(q) < 0 ? -F : F;
        } else {
          const Fx Fa = ia == 0 ? F : TF[ia], Fb = ib == 0 ? F : TF[ib];
          out = limit_face(T, F, dmin(Fa, Fx(0)), dmax(Fb, Fx(0)), q, dens);
          if (read_next || read_by_n) {
            const bool neg = !(dmin(out, Fx(0)) == dmin(F, Fx(0))), posv = !(dmax(out, Fx(0)) == dmax(F, Fx(0)));
            if ((read_next && neg && t0[f * gsd] != 0.) || (read_by_n && (f == 0 ? neg : posv) && *t0 != 0.))
              chained = true;
          }
        }
      }
      *TF2 = out;
      TF += nf;
      TF2 += nf;
      tc += G.sv;
      t0 += G.sv;
    }
    if (chained) {
      const long line = line_of<DIR>(k, j, i, G.ny, G.nx);
      if (atomicExch(&T.flag[line], 1) == 0) T.list[atomicAdd(T.count, 1)] = (int)line;
    }
  }
}

// The flagged lines in the serial order, one warp per line and tracer: walking the faces
// in order, a face keeps the first pass's value unless a face it reads (min of face f-1 for
// un > 0; min of face 0 and max of face 1 for face n with un < 0) now holds a value other
// than the unscaled one the first pass read; only those faces are limited again. The warp
// loads 32 faces at a time (one per lane) and knows by ballot which of them read a face that
// changed, so it steps from one such face to the next instead of through all of them
// (128x128x64, three tracers: 14 -> 7 us per split).
template <class TA, int DIR>
__global__ void __launch_bounds__(128) tracer_limit_lines_kernel(TA T, int hs) {
  using Fx = typename TA::Flux;
  constexpr unsigned kAll = 0xffffffffu;
  const Geo<DIR> G(T.A, hs);
  const int n = G.n();
  const int lane = threadIdx.x & 31;
  const long nwarps = (long)gridDim.x * (blockDim.x / 32);
  const long items = (long)(*T.count) * T.ntr;
  const long nf = G.nface();
  for (long item = (blockIdx.x * (long)blockDim.x + threadIdx.x) / 32; item < items; item += nwarps) {
    const int l = (int)(item % T.ntr);
    if (!((T.pos >> l) & 1ull)) continue;  // unlimited: the first pass copied the fluxes
    const unsigned ln = (unsigned)T.list[item / T.ntr];
    int k0, j0, i0;  // the line's cell 0
    if (DIR == 0) { i0 = 0; j0 = (int)(ln % (unsigned)G.ny); k0 = (int)(ln / (unsigned)G.ny); }
    else if (DIR == 1) { j0 = 0; i0 = (int)(ln % (unsigned)G.nx); k0 = (int)(ln / (unsigned)G.nx); }
    else { k0 = 0; i0 = (int)(ln % (unsigned)G.nx); j0 = (int)(ln / (unsigned)G.nx); }
    auto face = [&](int p) {
      int kk, jj, ii;
      G.at(k0, j0, i0, p, kk, jj, ii);
      return G.face(kk, jj, ii);
    };
    const Fx *TF = T.TF + l * nf;
    Fx *TF2 = T.TF2 + l * nf;
    auto redo = [&](Fx F, Fx f1, Fx f2, int c) {  // face flux F limited by its upwind cell c
      int ck, cj, ci;
      G.at(k0, j0, i0, c, ck, cj, ci);
      return limit_face(T, F, f1, f2, T.tr[l * G.sv + G.g(ck, cj, ci)], T.D[G.cell(ck, cj, ci)] + trc_dens(T, hs, ck));
    };
    Fx sprev = 0, uprev = 0;            // the face behind the chunk: serial (scaled) and unscaled
    Fx s0 = 0, u0 = 0, s1 = 0, u1 = 0;  // faces 0 and 1, likewise
    for (int base = 0; base <= n; base += 32) {
      const int fme = base + lane;
      const bool in = fme <= n;
      long fim = 0;
      Fx Fm = 0, Tm = 0, Um = 0;
      if (in) {
        fim = face(fme);
        Fm = TF[fim];
        Tm = TF2[fim];
        Um = T.UN[fim];
      }
      // readers: faces upwinded from the cell behind; changed: faces whose min moved
      const unsigned readers = __ballot_sync(kAll, in && Um > 0 && fme > 0);
      unsigned changed = __ballot_sync(kAll, !(dmin(Tm, Fx(0)) == dmin(Fm, Fx(0))));
      const unsigned carry = !(dmin(sprev, Fx(0)) == dmin(uprev, Fx(0)));
      unsigned from = 0;  // lanes below it are done
      for (;;) {
        const unsigned need = readers & ((changed << 1) | carry) & (from < 32 ? kAll << from : 0u);
        if (!need) break;
        const int i = __ffs(need) - 1;
        const Fx sb = __shfl_sync(kAll, Tm, i > 0 ? i - 1 : 0);
        const Fx F = __shfl_sync(kAll, Fm, i);
        const Fx out = redo(F, dmin(i > 0 ? sb : sprev, Fx(0)), dmax(F, Fx(0)), base + i - 1);
        if (lane == i) {
          Tm = out;
          TF2[fim] = out;
        }
        changed = (changed & ~(1u << i)) | ((unsigned)!(dmin(out, Fx(0)) == dmin(F, Fx(0))) << i);
        from = (unsigned)i + 1;
      }
      if (base == 0) {
        s0 = __shfl_sync(kAll, Tm, 0);
        u0 = __shfl_sync(kAll, Fm, 0);
        s1 = __shfl_sync(kAll, Tm, 1);
        u1 = __shfl_sync(kAll, Fm, 1);
      }
      if (n - base < 32) {  // face n: upwinded from cell 0, it reads faces 0 and 1
        const int i = n - base;
        const Fx un = __shfl_sync(kAll, Um, i), F = __shfl_sync(kAll, Fm, i);
        if (un < 0 && (!(dmin(s0, Fx(0)) == dmin(u0, Fx(0))) || (n >= 2 && !(dmax(s1, Fx(0)) == dmax(u1, Fx(0)))))) {
          const Fx out = redo(F, dmin(s0, Fx(0)), dmax(n == 1 ? F : s1, Fx(0)), 0);
          if (lane == i) TF2[fim] = out;
        }
      }
      sprev = __shfl_sync(kAll, Tm, 31);
      uprev = __shfl_sync(kAll, Fm, 31);
    }
  }
}

// Per cell: the tendency of the limited fluxes, density multiplied back and the update
// (Spatial:948-955; Temporal_ader.h:67-69), and the halo cells of this direction left
// holding tracer/density, as the reference's in-place halo fill leaves them. out_divided:
// the interior is left divided by the post-split density (the state's split is done), as
// the next split's tracer_divide_kernel would divide it.
#ifndef AWFL_TRC_UPDATE_MINB
#define AWFL_TRC_UPDATE_MINB 1
#endif
template <class TA, int DIR>
__global__ void __launch_bounds__(128, AWFL_TRC_UPDATE_MINB) tracer_update_kernel(TA T, int hs, bool out_divided) {
  const Geo<DIR> G(T.A, hs);
  const unsigned pq = blockIdx.x * 128u + threadIdx.x;
  if (pq >= (unsigned)G.nx * G.ny) return;
  const int j = (int)(pq / (unsigned)G.nx), i = (int)(pq - (unsigned)j * G.nx);
  const int n = G.n();
  const long nf = G.nface();
  const int fs = DIR == 0 ? 1 : (DIR == 1 ? G.nx : G.nx * G.ny);
  const long gsd = DIR == 0 ? 1 : (DIR == 1 ? G.sy : G.sz);
  const bool periodic = T.A.bc == BC_PERIODIC;
  for (int k = blockIdx.y; k < G.nz; k += gridDim.y) {
    const int p = DIR == 0 ? i : (DIR == 1 ? j : k);
    const long gg = G.g(k, j, i), c = (long)k * ((unsigned)G.nx * G.ny) + pq;
    const Rcp<double> r = make_rcp<double>(out_divided ? trc_divisor(T, hs, k, idR * G.sv + gg) : 1.);
    double *t = T.tr + gg;
    const typename TA::Flux *TF2 = T.TF2 + G.face(k, j, i);
    for (int l = 0; l < T.ntr; l++, t += G.sv, TF2 += nf) {
      const double q = *t;  // tracer / density (tracer_divide_kernel)
      const double tn = trc_update(T, q, hs, k, c, TF2[0], TF2[fs]);
      *t = out_divided ? divp_any(tn, r) : tn;
      // the halo cells along DIR that copy this one
      if (periodic) {
        if (p >= n - hs) t[-n * gsd] = q;
        if (p < hs) t[n * gsd] = q;
      } else {
        if (p == 0)
          for (int h = 1; h <= hs; h++) t[-h * gsd] = q;
        if (p == n - 1)
          for (int h = 1; h <= hs; h++) t[h * gsd] = q;
      }
    }
  }
}

}  // namespace
}  // namespace awfl
