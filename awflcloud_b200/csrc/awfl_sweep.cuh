// The line-sweep kernel skeleton shared by the FP64 and FP32 forms.
//
// A CTA owns W whole lines along the sweep direction DIR and marches along them in
// chunks of C cells. Because no other CTA touches those lines, the tendency can be
// applied in place (MODE_APPLY) with no race: every stencil value a chunk reads comes
// from a shared-memory ring holding the ORIGINAL values of positions
// [base-HS, base+C+HS), refilled one chunk ahead of the updates, and the first HS rows
// (needed again by the periodic wrap at the end of the line) are saved before they are
// overwritten.
//
// Per chunk: (A) the chunk's ring rows are in place (landed by TMA or cp.async, or stored
// from registers); the next chunk's rows are requested; reconstruct cells base..base+C-1
// -> left/right edge states; Riemann flux at their left faces (the left state of the
// first face is carried from the previous chunk); divergence and update of cells
// base-1..base+C-2 (the last cell's right face is computed in the next chunk). Where a
// line's C cells are consecutive lanes of one warp (SHFL) the edge states and fluxes move
// between neighbouring cells by warp shuffles and (A) is the chunk's only CTA barrier;
// otherwise they go through shared memory with barriers (B), (C), (D) between the steps.
// The last cell of the line is finished after the loop.
//
// Boundary handling reproduces the reference's halo fill (Spatial_euler3d_cons_expl_
// cart_fv_Agrid.h:631-662, 994-1025, 1351-1382) and edge-value BCs (:816-837, 1176-1197,
// 1557-1578): periodic wraps; a wall copies the edge cell with zero normal momentum, and
// its boundary face uses the interior state on both sides. The halo values are also
// written to the state's halo cells, as the reference does in place.
// An x sweep of a slab of a larger grid (A.xh[side] != nullptr) takes an end's halo
// values from the neighbouring slab's columns instead (hs+1 of them: the neighbour's edge
// cell is reconstructed here, so the face between the slabs gets the same left and right
// states, hence the same flux, as in the undivided grid).
//
// The physics policy P supplies the element type, the per-cell reconstruction (+ADER +
// time average), the face flux, the tendency and the in-place update:
//   using Real; using Args;                         Args has state/tend/nx/ny/nz/bc/mode/sim2d
//   template <int ORD, int DIR, class S> recon(sten, kb, A, eL[5], eR[5], src, cell)
//                                          (cell: the cell's (k,j,i) index, -1 for a
//                                          cell of a neighbouring slab)
//   template <int DIR, int NG>            flux(qL[5], qR[5], kf, A, F[5])
//                                          (kf: the face's k for z, the line's k for x, y)
//   template <int DIR>                    tendency(v, Fl, Fr, src, A) -> Real
//   struct Aux; load_aux(A, g0, sv, aux)   per-cell inputs of the update (variable v at
//                                          g0 + v*sv), loaded a reconstruction ahead
//   apply(A, gidx, orig, tnd, aux, v)      state[gidx] = orig "+" dt*tnd (MODE_APPLY)
//   kAsyncRing                             next-chunk rows by cp.async into a 4C ring
//   kTmaRing, prepare_tma(A, ord, dir, C, W) (host), tma_map(A), tma_map_global(a, g),
//   flag_timeout(A)                        next-chunk rows of interior chunks by tiled TMA
//                                          boxes through a tensor map (kernel parameter
//                                          for single-grid sweeps, the work list in
//                                          global memory for ensembles)
//   min_blocks(ORD)                        CTAs per SM the register budget must allow
//   kSlab                                  the policy runs x splits of slabs (A.xh)
//   base_factor(A, tma)                    (host) what keeps PolicyShape from its usual speed
//   load(A, gidx) / store(A, gidx, x)      state element access (halo writes)
//   store_tend(A, tidx, x)                 tendency output (MODE_TEND)
#pragma once

#include <algorithm>
#include <type_traits>

#include "awfl_internal.h"

namespace awfl {

// Asynchronous global -> shared copy of one element (cp.async, sm_80+; 4 or 8 bytes).
template <class T> __device__ __forceinline__ void cp_async_row(T *dst_smem, const T *src_gmem) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "cp.async of 4 or 8 bytes");
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src_gmem), "n"(sizeof(T)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Tiled TMA loads (cp.async.bulk.tensor) completing on a shared-memory mbarrier. The
// destination is the CTA's own shared memory (128-byte aligned boxes), the source this
// GPU's global memory through a tensor map held in the kernel parameter; no multicast.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *mb, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(mb)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long *mb) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(mb)) : "memory");
}
__device__ __forceinline__ void mbar_arm(unsigned long long *mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(mb)), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity, giving up after a bounded number of polls
// (each poll may suspend the thread for a while); returns false then.
__device__ __forceinline__ bool mbar_wait(unsigned long long *mb, unsigned parity) {
  const unsigned a = smem_addr(mb);
  for (int i = 0; i < (1 << 20); i++) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// One 3-D box of the tensor map at element coordinates (x, y, z) into shared memory.
__device__ __forceinline__ void tma_load_3d(void *dst_smem, const void *tmap, int x, int y, int z,
                                            unsigned long long *mb) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(smem_addr(dst_smem)),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_addr(mb))
      : "memory");
}
// Warp shuffle up by `delta` lanes within segments of `width` lanes, for a value of any
// type made of 4-byte words (float, double, a dual number); every lane of the warp calls it.
template <class T> __device__ __forceinline__ T shfl_up_any(const T &x, int delta, int width) {
  static_assert(sizeof(T) % 4 == 0, "shuffled types are made of 4-byte words");
  constexpr int N = (int)(sizeof(T) / 4);
  unsigned u[N];
  __builtin_memcpy(u, &x, sizeof(T));
#pragma unroll
  for (int i = 0; i < N; i++) u[i] = __shfl_up_sync(0xffffffffu, u[i], delta, width);
  T y;
  __builtin_memcpy(&y, u, sizeof(T));
  return y;
}

// the value of lane `lane` of the segment, likewise
template <class T> __device__ __forceinline__ T shfl_idx_any(const T &x, int lane, int width) {
  static_assert(sizeof(T) % 4 == 0, "shuffled types are made of 4-byte words");
  constexpr int N = (int)(sizeof(T) / 4);
  unsigned u[N];
  __builtin_memcpy(u, &x, sizeof(T));
#pragma unroll
  for (int i = 0; i < N; i++) u[i] = __shfl_sync(0xffffffffu, u[i], lane, width);
  T y;
  __builtin_memcpy(&y, u, sizeof(T));
  return y;
}

// orders this thread's generic-proxy shared-memory accesses before later async-proxy ones
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// Row pitch (elements) of the ring of a y/z sweep fed by TMA: the box starts at the
// 16-byte-aligned x = bx*W of the halo-inclusive row (the tile's first line sits at
// column HS), spans at least W + HS columns in a multiple of 4, and a chunk's C rows
// (one box) are a multiple of 128 bytes so that every box lands 128-byte aligned.
__host__ __device__ constexpr int tma_ring_pitch_of(int ord, int C, int W, int esz) {
  int rw = (W + (ord - 1) / 2 + 3) / 4 * 4;
  while ((C * rw * esz) % 128 != 0) rw += 4;
  return rw;
}
template <int ORD, int C, int W, int ESZ> __host__ __device__ constexpr int tma_ring_pitch() {
  return tma_ring_pitch_of(ORD, C, W, ESZ);
}

// A policy with `static constexpr bool kFaceRec = true` sees every face the sweep computes:
// P::face_rec<ORD, DIR>(A, face, kf, qL, qR, F) with the face's index in the tracer path's
// face numbering (faces along DIR: n+1 per line), the k passed to the flux, the face's two
// states after the edge BCs and its flux (the tracer transport records them).
template <class P, class = void> struct PolicyFaceRec : std::false_type {};
template <class P> struct PolicyFaceRec<P, std::void_t<decltype(P::kFaceRec)>> : std::bool_constant<P::kFaceRec> {};

// One CTA's tile: lines bx*W .. bx*W+W-1 of plane `by` (x, y sweeps: by = k; z: by = j).
// tmap: the tensor map of the TMA path (a kernel-parameter or global address), or nullptr
// (the instantiation with TMA = true then stages every chunk by cp.async).
// SLAB: the x sweep of a slab of a larger grid, whose ends may take their halo values from
// the neighbouring slabs (A.xh); a separate instantiation, so that the plain sweeps carry
// none of its registers.
// ENDS: the line's last face takes a spare lane (below): for the small-grid shapes, since
// the large grids' sweeps, with many chunks to a line, lose more by the registers.
template <class P, int ORD, int DIR, int C, int W, bool TMA = false, bool SLAB = false, bool ENDS = false>
__device__ __forceinline__ void sweep_tile(const typename P::Args &A, const int bx, const int by,
                                           const void *tmap = nullptr) {
  using Real = typename P::Real;
  constexpr int HS = (ORD - 1) / 2;
  constexpr int NG = OrdTraits<ORD>::NGLL;
  // Next-chunk rows: policies with kAsyncRing copy them global -> shared with cp.async one
  // chunk ahead (issued before the reconstruction, no registers held), which needs a ring
  // of 4C so that the rows in flight never share a slot with rows still being read;
  // otherwise they are loaded into registers and stored at the next chunk's start.
  constexpr bool ASYNC = P::kAsyncRing;
  constexpr int R = ASYNC ? 4 * C : 2 * C;  // ring length (power of two, >= C + 2*HS)
  // TMA path (TMA, with the async ring): a chunk whose rows are all interior arrives as
  // five tiled TMA boxes, one per variable, issued by one thread and completing on an
  // mbarrier -- x sweep: box {C positions, W lines}, landing as one page [W][C] of the
  // ring; y/z sweeps: box {RW columns from x = bx*W, C positions}, landing as C ring rows
  // of pitch RW with line w at column HS + w. Other chunks (and a tile whose wait gave
  // up) use cp.async. Out-of-range box elements (the last tile's missing lines) read as
  // zero and are never used.
  // The C cells of a chunk of one line are C consecutive lanes of one warp (x sweep: a
  // warp holds 32/C lines along x; y/z sweeps: 32/C neighbouring lines, so that a warp's
  // global accesses are 32/C consecutive x cells in each of C rows), so the interface
  // states, fluxes and z sources pass between neighbouring cells by warp shuffles (the
  // first cell's left neighbour is the previous chunk's last cell, carried per line in
  // shared memory); the chunk needs no CTA barrier besides the ring's (A). The y/z sweeps
  // of the register-staged path keep a warp along x across lines (32/W positions) and
  // trade through shared memory between barriers: a warp's next-chunk loads from global
  // memory would otherwise touch C rows instead of 32/W (FP64 z split measured 3.61 ->
  // 3.71 ms with the shuffles).
  constexpr bool SHFL = C <= 32 && (C * W) % 32 == 0 && (DIR == 0 || ASYNC);
  static_assert(!TMA || ASYNC, "the TMA path feeds the async ring");
  // Row pitch of a y/z ring. A warp of the shuffle path reads LW = 32/C neighbouring words of
  // each of C rows; with the pitch an odd multiple of LW the rows start in different banks
  // (at pitch W, a multiple of the banks, all C of them in the same ones: FP64 256x256x128,
  // y 1343 -> 1299 us, z 1420 -> 1376; ord 9, 128x128x64, y 875 -> 837, z 909 -> 862).
  constexpr int LW = C <= 32 ? 32 / C : 1;
  constexpr int RW = DIR == 0 ? W
                     : TMA    ? tma_ring_pitch<ORD, C, W, (int)sizeof(Real)>()
                     : (SHFL && W % LW == 0) ? (W / LW % 2 ? W : W + LW) : W;
  static_assert(!TMA || DIR != 0 || ((C * W * (int)sizeof(Real)) % 128 == 0 && (2 * HS * (int)sizeof(Real)) % 16 == 0 &&
                                     (C * (int)sizeof(Real)) % 16 == 0),
                "x-sweep TMA pages must be 128-byte multiples starting at 16-byte-aligned x");
  static_assert(!TMA || DIR == 0 || (W * (int)sizeof(Real)) % 16 == 0, "y/z-sweep TMA boxes start at x = bx*W");
  constexpr int NM = 1 + DIR;
  static_assert((C & (C - 1)) == 0 && C >= 2 * HS, "chunk must be a power of two >= 2*HS");
  // Register path: load the next chunk's rows before the reconstruction (latency hidden
  // behind it, at the cost of 5 live registers) for the z sweep, whose loads stride over
  // whole planes; after the updates for x and y, where occupancy matters more (measured).
  constexpr bool EARLY_PREFETCH = !ASYNC && DIR == 2;
  __shared__ __align__(128) Real ring[5][R * RW];
  __shared__ __align__(8) unsigned long long mbar;  // TMA path only
  __shared__ int sAbort;                            // TMA path: a wait of this tile gave up
  constexpr int ES = SHFL ? 1 : C + 1;  // edge slots of a line: the carry alone, or every face
  __shared__ Real sEL[5][ES * W];
  __shared__ Real sER[5][ES * W];
  __shared__ Real sF[5][ES * W];
  __shared__ Real sSrc[DIR == 2 ? ES * W : 1];
  __shared__ Real sWrap[5][HS * W];
  __shared__ Real sEL0[5][W];
  __shared__ Real sF1[5][W];  // periodic lines: the flux of face 1 and the source of cell 0
  __shared__ Real sSrc0[DIR == 2 ? W : 1];

  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  // position in chunk, line within CTA
  const int c = DIR == 0 ? (int)threadIdx.x : (SHFL ? (tid & (C - 1)) : (int)threadIdx.y);
  const int w = DIR == 0 ? (int)threadIdx.y : (SHFL ? tid / C : (int)threadIdx.x);
  // edge/flux slot (0..C) of this line: consecutive threads of a warp hit consecutive words
  auto E = [&](int slot) { return DIR == 0 ? w * ES + slot : slot * W + w; };

  const int nx = A.nx, ny = A.ny, nz = A.nz;
  const long sx = 1, sy = nx + 2 * HS, sz = (long)(ny + 2 * HS) * sy, sv = (long)(nz + 2 * HS) * sz;
  int L, kline = 0;
  bool valid;
  long lb;  // offset of (v=0, position 0 along DIR) of this line, halo-inclusive frame
  long sd;  // stride along DIR
  long tb;  // tendency offset of position 0
  long tsd;
  long fb, fsd;  // face index of position 0 and its stride along DIR (face records only)
  if (DIR == 0) {
    const int k = by, j = bx * W + w;
    L = nx; valid = j < ny; kline = k;
    lb = (HS + k) * sz + (HS + (valid ? j : 0)) * sy + HS * sx; sd = sx;
    tb = ((long)k * ny + (valid ? j : 0)) * nx; tsd = 1;
    fb = ((long)k * ny + (valid ? j : 0)) * (nx + 1); fsd = 1;
  } else if (DIR == 1) {
    const int k = by, i = bx * W + w;
    L = ny; valid = i < nx; kline = k;
    lb = (HS + k) * sz + HS * sy + HS + (valid ? i : 0); sd = sy;
    tb = (long)k * ny * nx + (valid ? i : 0); tsd = nx;
    fb = (long)k * (ny + 1) * nx + (valid ? i : 0); fsd = nx;
  } else {
    const int j = by, i = bx * W + w;
    L = nz; valid = i < nx;
    lb = HS * sz + (HS + j) * sy + HS + (valid ? i : 0); sd = sz;
    tb = (long)j * nx + (valid ? i : 0); tsd = (long)ny * nx;
    fb = (long)j * nx + (valid ? i : 0); fsd = (long)ny * nx;
  }
  const long tv = (long)nz * ny * nx;
  const bool periodic = A.bc == BC_PERIODIC;
  // x sweep of a slab: the ends bordering another slab, and that slab's columns
  // ([5][nz][ny][HS+1] per side: side 0 holds positions -(HS+1)..-1, side 1 L..L+HS)
  static_assert(!SLAB || DIR == 0, "slabs are cut along x");
  bool xlo = false, xhi = false;
  int jline = 0;
  if constexpr (SLAB) {
    xlo = A.xh[0] != nullptr;
    xhi = A.xh[1] != nullptr;
    jline = bx * W + w;
  }
  auto XH = [&](int side, int v, int col) -> Real {
    return Real(A.xh[side][(((long)v * nz + kline) * ny + jline) * (HS + 1) + col]);
  };

  auto G = [&](int v, int p) -> Real { return P::load(A, lb + v * sv + p * sd); };
  // ring slot of position p: the async ring counts from p = HS so that a chunk's rows
  // (positions base+HS .. base+C+HS-1) fill one aligned run of C slots. The x sweep's
  // async ring is paged: page s/C holds [line][slot % C], so the lines of a warp read
  // 32 consecutive words (no bank conflict) and a chunk is one TMA box.
  auto ringAt = [&](int v, int p) -> Real & {
    if constexpr (ASYNC) {
      const int s = (p - HS) & (R - 1);
      if constexpr (DIR == 0) return ring[v][(s / C) * (W * C) + w * C + (s & (C - 1))];
      else return ring[v][s * RW + (TMA ? HS : 0) + w];
    } else {
      const int s = p & (R - 1);
      return DIR == 0 ? ring[v][w * R + s] : ring[v][s * W + w];
    }
  };
  auto topval = [&](int v, int p, bool first) -> Real {  // p >= L
    const int q = p - L;
    if (q >= HS) return Real(0);  // beyond the last cell's stencil: never read
    if (xhi) return XH(1, v, q);
    if (periodic) return first ? G(v, q) : sWrap[v][q * W + w];
    return v == NM ? Real(0) : G(v, L - 1);
  };
  auto finish_as = [&](int cell, auto orig, const Real *Fl, const Real *Fr, Real sa, const typename P::Aux &aux) {
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const Real tnd = P::template tendency<DIR>(v, Fl[v], Fr[v], sa, A);
      if (A.mode == MODE_APPLY) P::apply(A, lb + v * sv + cell * sd, orig(v), tnd, aux, v);
      else P::store_tend(A, tb + v * tv + cell * tsd, tnd);
    }
  };
  auto finish = [&](int cell, const Real *Fl, const Real *Fr, Real sa, const typename P::Aux &aux) {
    finish_as(cell, [&](int v) -> Real { return ringAt(v, cell); }, Fl, Fr, sa, aux);
  };
  // a row value into its ring slot: asynchronously when it is a load of an interior cell
  auto stage = [&](int v, int p, bool first) {
    if constexpr (ASYNC) {
      if (p < L) cp_async_row(&ringAt(v, p), &A.state[lb + v * sv + p * sd]);
      else ringAt(v, p) = topval(v, p, first);
    }
  };
  // the chunk whose rows start at position p0 comes by TMA (uniform in the CTA)
  auto chunk_tma = [&](int p0) { return TMA && tmap != nullptr && p0 + C <= L; };
  constexpr unsigned kTmaBytes = 5u * C * (DIR == 0 ? W : RW) * (unsigned)sizeof(Real);
  auto issue_tma = [&](int p0) {  // thread 0 only
    if constexpr (TMA) {
      const int s0 = (p0 - HS) & (R - 1);  // a multiple of C
      const int zp = nz + 2 * HS;          // the map's z extent per variable
      mbar_arm(&mbar, kTmaBytes);
#pragma unroll
      for (int v = 0; v < 5; v++) {
        if (DIR == 0) tma_load_3d(&ring[v][(s0 / C) * (W * C)], tmap, HS + p0, HS + bx * W, v * zp + HS + by, &mbar);
        else if (DIR == 1) tma_load_3d(&ring[v][s0 * RW], tmap, bx * W, HS + p0, v * zp + HS + by, &mbar);
        else tma_load_3d(&ring[v][s0 * RW], tmap, bx * W, HS + by, v * zp + HS + p0, &mbar);
      }
    }
  };

  // ---- prologue: the first chunk's rows are requested, then the bottom halo, the wrap rows and
  // the top halo are loaded, all of them before the first store: the halo stores go to the
  // state's own array, so the compiler keeps every later load behind them, and five variables
  // in turn were five round trips to L2 (FP32 64x64x32: 50.2 -> 46.9 us per step).
  Real pre[ASYNC ? 1 : 5];
  bool cur_tma = false;  // this chunk's rows come by TMA (uniform in the CTA)
  unsigned phase = 0;    // TMA phases of the mbarrier issued so far
  if constexpr (TMA) {
    cur_tma = chunk_tma(HS);
    if (tid == 0) {
      mbar_init(&mbar, 1);
      sAbort = 0;
      if (cur_tma) issue_tma(HS);
    }
    if (cur_tma) phase++;
  }
  if (ASYNC && valid && !cur_tma) {
#pragma unroll
    for (int v = 0; v < 5; v++) stage(v, HS + c, true);
  }
  if (valid && c < HS) {
    Real bot[5], top[5], orig[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
      bot[v] = xlo ? XH(0, v, c + 1) : (periodic ? G(v, L + c - HS) : (v == NM ? Real(0) : G(v, 0)));
      top[v] = xhi ? XH(1, v, c) : (periodic ? G(v, c) : (v == NM ? Real(0) : G(v, L - 1)));
      // position c of a wall line shorter than HS is a top halo cell: its stencil value is
      // the wall copy (read from the interior, never from a halo cell another thread of
      // this prologue is writing); periodic lines are at least HS long (awfl_create)
      orig[v] = c < L ? G(v, c) : top[v];
    }
#pragma unroll
    for (int v = 0; v < 5; v++) {
      ringAt(v, c - HS) = bot[v];
      ringAt(v, c) = orig[v];
      sWrap[v][c * W + w] = orig[v];
      P::store(A, lb + v * sv + (c - HS) * sd, bot[v]);
      P::store(A, lb + v * sv + (L + c) * sd, top[v]);
    }
  }
  if constexpr (TMA) {
    fence_proxy_async();  // the prologue's generic writes to ring slots before any TMA write to them
    __syncthreads();      // the mbarrier is initialised before the other threads wait on it
  }
  if constexpr (!ASYNC) {
    if (valid) {
      const int p = HS + c;
#pragma unroll
      for (int v = 0; v < 5; v++) pre[v] = p < L ? G(v, p) : topval(v, p, true);
    }
  }
  // A periodic line's face 0 is its face L: its left state, the right edge of cell L-1, is
  // known when the line ends, so the flux of face 0 and the update of cell 0 wait until
  // then (cell 0's right flux and source are kept, its original value is in the wrap rows).
  // The sweep used to reconstruct cell L-1 a second time up front, on one lane of C: 1/L
  // more work, and a whole chunk's latency per tile (FP64 ord 9, 128x128x64: 2.91 -> 2.66 ms
  // per step; FP32 ord 9: 0.76 -> 0.64).
  const bool late0 = periodic && !xlo;
  // a periodic line's cell 0 from the states and the flux of face L: the same states as face
  // 0, so the same flux, but for z's per-face background
  auto finish_first = [&](const Real (&qL)[5], const Real (&qR)[5], const Real (&FL)[5]) {
    Real F[5], F1[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
      F[v] = FL[v];
      F1[v] = sF1[v][w];
    }
    if constexpr (DIR == 2) P::template flux<DIR, NG>(qL, qR, 0, A, F);
    if constexpr (PolicyFaceRec<P>::value) P::template face_rec<ORD, DIR>(A, fb, DIR == 2 ? 0 : kline, qL, qR, F);
    typename P::Aux aux;
    if (A.mode == MODE_APPLY) P::load_aux(A, lb, sv, aux);
    finish_as(0, [&](int v) -> Real { return sWrap[v][w]; }, F, F1, DIR == 2 ? sSrc0[w] : Real(0), aux);
  };
  // a slab bordering another below: the left state of face 0 is the right edge of that
  // slab's last cell (position -1)
  if constexpr (SLAB) if (valid && xlo && c == 0) {
    auto wrapSten = [&](int v, int m) -> Real {
      const int p = -1 - HS + m;
      return p < 0 ? XH(0, v, p + HS + 1) : G(v, p);
    };
    Real eL[5], eR[5], sa;
    P::template recon<ORD, DIR>(wrapSten, kline, A, eL, eR, sa, -1L);
#pragma unroll
    for (int v = 0; v < 5; v++) sER[v][E(0)] = eR[v];
  }

  const int nchunk = (L + C - 1) / C;
  // ENDS: face L takes a lane of its own in the last chunk where that has one to spare, so
  // that the line ends with the chunk instead of one more flux on one lane of C (the
  // epilogue; a third of a short line's time). A periodic x or y line of one full chunk has its faces
  // 0 and L as one: lane 0 takes it, its left state from the last lane (ROT).
  const bool ends = ENDS && L % C != 0 && !xhi;
  const bool rot = ENDS && SHFL && DIR != 2 && late0 && L == C;
  for (int t = 0; t < nchunk; t++) {
    const int base = t * C;
    const int nvalid = min(C, L - base);
    const int nface = nvalid + (ends && t + 1 == nchunk ? 1 : 0);  // faces base .. of this chunk
    if constexpr (TMA) {
      // the chunk's boxes have landed; a wait that gives up flags the error and ends the
      // tile's use of TMA (the rest of the tile's chunks come by cp.async)
      if (cur_tma && !mbar_wait(&mbar, (phase - 1) & 1u)) {
        P::flag_timeout(A);
        sAbort = 1;
      }
      // (generic reads of a slot, then a TMA write into it after barrier (A): ordered by
      // the barrier. Within a tile, generic writes into slots that a TMA box fills later
      // happen only in the prologue, which fences them, and the first chunk's boxes, issued
      // before that fence, fill none of the prologue's slots. What a tile leaves behind, its
      // last chunks' cp.async rows and halo values among it, is fenced at its end.)
    }
    if constexpr (ASYNC) {
      cp_async_wait_all();  // this thread's rows of the chunk have landed
    } else if (valid) {
#pragma unroll
      for (int v = 0; v < 5; v++) ringAt(v, base + HS + c) = pre[v];
    }
    __syncthreads();  // (A)
    if constexpr (ASYNC) {  // the next chunk's rows, a chunk ahead
      bool next_tma = false;
      if constexpr (TMA) {
        next_tma = t + 1 < nchunk && chunk_tma(base + C + HS) && !*(volatile int *)&sAbort;
        if (next_tma && tid == 0) issue_tma(base + C + HS);
        if (next_tma) phase++;
      }
      if (!next_tma && valid && t + 1 < nchunk) {
#pragma unroll
        for (int v = 0; v < 5; v++) stage(v, base + C + HS + c, false);
      }
      cur_tma = next_tma;
    }
    // the compensation (or other per-cell input) of the cell this thread updates below
    typename P::Aux aux;
    if (valid && c < nface && (rot || base + c >= 1) && A.mode == MODE_APPLY)
      P::load_aux(A, lb + (rot && c == 0 ? L - 1 : base + c - 1) * sd, sv, aux);
    // next chunk's rows (stored into the ring at the next (A); the updates of this chunk
    // never reach them)
    if (EARLY_PREFETCH && valid && t + 1 < nchunk) {
      const int p = base + C + HS + c;
#pragma unroll
      for (int v = 0; v < 5; v++) pre[v] = p < L ? G(v, p) : topval(v, p, false);
    }
    Real eL[5], eR[5], sa;
    if constexpr (SHFL) {  // defined values on the lanes that reconstruct nothing
#pragma unroll
      for (int v = 0; v < 5; v++) eL[v] = eR[v] = Real(0);
      sa = Real(0);
    }
    if (valid && c < nvalid) {
      const int p = base + c;
      auto sten = [&](int v, int m) -> Real { return ringAt(v, p - HS + m); };
      P::template recon<ORD, DIR>(sten, DIR == 2 ? p : kline, A, eL, eR, sa, tb + p * tsd);
      if constexpr (!SHFL) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
          sEL[v][E(c)] = eL[v];
          sER[v][E(c + 1)] = eR[v];
        }
        if (DIR == 2) sSrc[E(c + 1)] = sa;
      }
      if (p == 0) {
#pragma unroll
        for (int v = 0; v < 5; v++) sEL0[v][w] = eL[v];
      }
    }
    if constexpr (SHFL) {
      const bool act = valid && c < nface;
      // face base+c: left state = right edge of cell base+c-1 (the lane below, or the carry;
      // ROT: lane 0 takes the last lane's)
      Real qL[5], F[5];
#pragma unroll
      for (int v = 0; v < 5; v++) {
        const Real up = shfl_up_any(eR[v], 1, C);
        qL[v] = c == 0 ? sER[v][E(0)] : up;
      }
      if (rot) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
          const Real top = shfl_idx_any(eR[v], C - 1, C);
          if (c == 0) qL[v] = top;
        }
      }
      if (ENDS && nface > nvalid) {
        __syncwarp();  // sEL0 may be this chunk's
        if (c == nvalid) {
#pragma unroll
          for (int v = 0; v < 5; v++) eL[v] = late0 ? sEL0[v][w] : qL[v];
        }
      }
      if (act && (rot || !(late0 && base + c == 0))) {
        if (base + c == 0 && !periodic && !xlo) {
#pragma unroll
          for (int v = 0; v < 5; v++) qL[v] = eL[v];
        }
        P::template flux<DIR, NG>(qL, eL, DIR == 2 ? base + c : kline, A, F);
        if constexpr (PolicyFaceRec<P>::value) {
          P::template face_rec<ORD, DIR>(A, fb + (base + c) * fsd, DIR == 2 ? base + c : kline, qL, eL, F);
          if (rot && c == 0) P::template face_rec<ORD, DIR>(A, fb + L * fsd, kline, qL, eL, F);
        }
      } else {
#pragma unroll
        for (int v = 0; v < 5; v++) F[v] = Real(0);
      }
      // cell base+c-1: its left face's flux from the lane below (or the carry), its right
      // face's from this lane; ROT: lane 0 finishes cell L-1
      Real Fl[5];
#pragma unroll
      for (int v = 0; v < 5; v++) {
        const Real up = shfl_up_any(F[v], 1, C);
        Fl[v] = c == 0 ? sF[v][E(0)] : up;
      }
      if (rot) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
          const Real top = shfl_idx_any(F[v], C - 1, C);
          if (c == 0) Fl[v] = top;
        }
      }
      Real sl = Real(0);  // z: the source term of cell base+c-1
      if constexpr (DIR == 2) {
        const Real up = shfl_up_any(sa, 1, C);
        sl = c == 0 ? sSrc[E(0)] : up;
      }
      if (act && late0 && !rot && base + c == 1) {
#pragma unroll
        for (int v = 0; v < 5; v++) sF1[v][w] = F[v];
        if (DIR == 2) sSrc0[w] = sl;
      } else if (act && (rot || base + c >= 1)) {
        finish(rot && c == 0 ? L - 1 : base + c - 1, Fl, F, sl, aux);
      }
      if (!ASYNC && valid && t + 1 < nchunk) {
        const int p = base + C + HS + c;
#pragma unroll
        for (int v = 0; v < 5; v++) pre[v] = p < L ? G(v, p) : topval(v, p, false);
      }
      __syncwarp();  // the line's reads of its ring rows and carry are done
      if (valid && c == nvalid - 1) {  // the carry: last cell's right edge, right-face flux, source
#pragma unroll
        for (int v = 0; v < 5; v++) {
          sER[v][E(0)] = eR[v];
          sF[v][E(0)] = F[v];
        }
        if (DIR == 2) sSrc[E(0)] = sa;
      }
      if constexpr (ENDS)
        if (late0 && act && c == nvalid) finish_first(qL, eL, F);  // the lane of face L
      __syncwarp();
      continue;
    }
    __syncthreads();  // (B)
    if (valid && c < nface && !(late0 && base + c == 0)) {
      const int f = base + c;  // face index = left face of cell f
      Real qL[5], qR[5], F[5];
#pragma unroll
      for (int v = 0; v < 5; v++) qR[v] = c < nvalid ? sEL[v][E(c)] : (late0 ? sEL0[v][w] : sER[v][E(c)]);
#pragma unroll
      for (int v = 0; v < 5; v++) qL[v] = (f == 0 && !periodic && !xlo) ? qR[v] : sER[v][E(c)];
      P::template flux<DIR, NG>(qL, qR, DIR == 2 ? f : kline, A, F);
      if constexpr (PolicyFaceRec<P>::value) P::template face_rec<ORD, DIR>(A, fb + f * fsd, DIR == 2 ? f : kline, qL, qR, F);
#pragma unroll
      for (int v = 0; v < 5; v++) sF[v][E(c + 1)] = F[v];
    }
    __syncthreads();  // (C)
    if (valid && c < nface) {
      const int cell = base + c - 1;
      if (cell >= 0) {
        Real Fl[5], Fr[5];
#pragma unroll
        for (int v = 0; v < 5; v++) {
          Fl[v] = sF[v][E(c)];
          Fr[v] = sF[v][E(c + 1)];
        }
        if (late0 && cell == 0) {
#pragma unroll
          for (int v = 0; v < 5; v++) sF1[v][w] = Fr[v];
          if (DIR == 2) sSrc0[w] = sSrc[E(c)];
        } else {
          finish(cell, Fl, Fr, DIR == 2 ? sSrc[E(c)] : Real(0), aux);
        }
      }
    }
    if (!ASYNC && !EARLY_PREFETCH && valid && t + 1 < nchunk) {
      const int p = base + C + HS + c;
#pragma unroll
      for (int v = 0; v < 5; v++) pre[v] = p < L ? G(v, p) : topval(v, p, false);
    }
    __syncthreads();  // (D)
    if (ENDS && late0 && valid && c == nvalid && nface > nvalid) {  // the lane of face L
      Real qL[5], qR[5], F[5];
#pragma unroll
      for (int v = 0; v < 5; v++) {
        qL[v] = sER[v][E(nvalid)];
        qR[v] = sEL0[v][w];
        F[v] = sF[v][E(nvalid + 1)];
      }
      finish_first(qL, qR, F);
    }
    if (valid && c == 0) {
#pragma unroll
      for (int v = 0; v < 5; v++) {
        sER[v][E(0)] = sER[v][E(nvalid)];
        sF[v][E(0)] = sF[v][E(nvalid)];
      }
      if (DIR == 2) sSrc[E(0)] = sSrc[E(nvalid)];
    }
  }
  // ---- epilogue, where no lane was left for it: face L and the last cell (same thread that
  // wrote the carry), then a periodic line's face 0 and cell 0
  if (valid && c == 0 && !ends && !rot) {
    Real qL[5], qR[5], F[5], Fl[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
      qL[v] = sER[v][E(0)];
      qR[v] = periodic ? sEL0[v][w] : qL[v];
      Fl[v] = sF[v][E(0)];
    }
    if (xhi) {  // a slab bordering another above: the left edge of that slab's first cell
      auto hiSten = [&](int v, int m) -> Real {
        const int p = L - HS + m;
        return p >= L ? XH(1, v, p - L) : ringAt(v, p);
      };
      Real hL[5], hR[5], hs_;
      P::template recon<ORD, DIR>(hiSten, kline, A, hL, hR, hs_, -1L);
#pragma unroll
      for (int v = 0; v < 5; v++) qR[v] = hL[v];
    }
    P::template flux<DIR, NG>(qL, qR, DIR == 2 ? L : kline, A, F);
    if constexpr (PolicyFaceRec<P>::value) P::template face_rec<ORD, DIR>(A, fb + L * fsd, DIR == 2 ? L : kline, qL, qR, F);
    typename P::Aux aux;
    if (A.mode == MODE_APPLY) P::load_aux(A, lb + (L - 1) * sd, sv, aux);
    finish(L - 1, Fl, F, DIR == 2 ? sSrc[E(0)] : Real(0), aux);
    if (late0) finish_first(qL, qR, F);
  }
  if constexpr (TMA) {  // every issued phase has completed (or been given up on, flagged)
    // a persistent CTA's next tile issues its first boxes straight away: this tile's generic
    // accesses to the ring (all of them where it had no tensor map) come before those
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      // after a give-up, a last bounded wait so that no box is still landing in this
      // CTA's shared memory when the tile ends
      if (sAbort && phase > 0) (void)mbar_wait(&mbar, (phase - 1) & 1u);
      mbar_inval(&mbar);
    }
  }
}

// CTAs per SM the register budget must allow: the policy's figure, or for the x-slab sweeps
// and the small-grid shapes of ord 5 AWFL_SMALL_MINB_ORD5 (the FP32 slab sweep at 4: 142 ->
// 107 registers and its x split of a 128x256x128 slab 0.442 -> 0.408 ms; the FP32 z split
// of 64x64x32 at 4 / 5: 17.4 / 18.5 us)
#ifndef AWFL_SMALL_MINB_ORD5
#define AWFL_SMALL_MINB_ORD5 4
#endif
template <class P, int ORD, bool CAP> constexpr int sweep_min_blocks() {
  return CAP && ORD == 5 ? AWFL_SMALL_MINB_ORD5 : P::min_blocks(ORD);
}

// TMA: the policy's single-grid TMA path; its tensor map lives in the (grid-constant)
// kernel parameter, the only place besides global memory a TMA copy may read it from.
template <class P, int ORD, int DIR, int C, int W, bool TMA, bool SLAB = false, bool ENDS = false>
__global__ void __launch_bounds__(C *W, (sweep_min_blocks<P, ORD, SLAB || ENDS>())) sweep_kernel(const __grid_constant__ typename P::Args A) {
  if constexpr (TMA) sweep_tile<P, ORD, DIR, C, W, true, SLAB, ENDS>(A, blockIdx.x, blockIdx.y, P::tma_map(A));
  else sweep_tile<P, ORD, DIR, C, W, false, SLAB, ENDS>(A, blockIdx.x, blockIdx.y);
}
template <class P, int ORD, int DIR, int C, int W, bool TMA, bool SLAB, bool ENDS>
cudaError_t launch_sweep_kernel(const typename P::Args &A, dim3 grid, cudaStream_t st) {
  const dim3 block(DIR == 0 ? C : W, DIR == 0 ? W : C);
  sweep_kernel<P, ORD, DIR, C, W, TMA, SLAB, ENDS><<<grid, block, 0, st>>>(A);
  return cudaGetLastError();
}

template <int ORD, int DIR> struct SweepShape;
template <> struct SweepShape<5, 0> { static constexpr int C = 32, W = 4; };
template <> struct SweepShape<5, 1> { static constexpr int C = 4, W = 32; };
template <> struct SweepShape<5, 2> { static constexpr int C = 4, W = 32; };
template <> struct SweepShape<9, 0> { static constexpr int C = 32, W = 2; };
template <> struct SweepShape<9, 1> { static constexpr int C = 8, W = 16; };
template <> struct SweepShape<9, 2> { static constexpr int C = 8, W = 16; };

// Shape of a policy's single-grid sweep: SweepShape unless the policy specialises it
// (measured per form at 256x256x128).
template <class P, int ORD, int DIR> struct PolicyShape : SweepShape<ORD, DIR> {};

// Policies with wider elements (P::kWdiv > 1) use fewer lines per CTA to stay within the
// 48 KB of static shared memory.
template <class P, int ORD, int DIR, int C> constexpr bool stages_by_tma() {
  return P::kTmaRing && ORD == 5 && DIR != 2 && C == PolicyShape<P, ORD, DIR>::C;
}
template <class P, int ORD, int DIR, int C, int W>
cudaError_t launch_sweep_shape(const typename P::Args &A, cudaStream_t st) {
  dim3 grid;
  if (DIR == 0) grid = dim3((A.ny + W - 1) / W, A.nz);
  else if (DIR == 1) grid = dim3((A.nx + W - 1) / W, A.nz);
  else grid = dim3((A.nx + W - 1) / W, A.ny);
  constexpr bool base = C == PolicyShape<P, ORD, DIR>::C;
  // the x split of a slab with neighbouring slabs' columns: the SLAB instantiation
  bool slab = false;
  if constexpr (DIR == 0 && P::kSlab && base) slab = A.xh[0] != nullptr || A.xh[1] != nullptr;
  if constexpr (stages_by_tma<P, ORD, DIR, C>()) {
    // the policy encodes this launch's tensor map (box = one chunk of one variable); a
    // layout TMA cannot address (alignment) leaves tma off and the cp.async path runs. TMA only
    // where it is the faster: the x and y shapes of large grids (FP32 256x256x128, us, TMA
    // 370 384, by cp.async 377 392). The z sweep needs 79 registers by cp.async instead of 89
    // (383 us, TMA 390); small grids' shapes start sooner (64x64x32 x split 12.4 us, TMA
    // 14.1) and TMA's pitch puts a narrow shape's rows in the same banks (y 16.6, TMA 17.4);
    // at ord 9 TMA's bookkeeping spills at three CTAs per SM (128x128x64, 32 x 2, 8 x 16 and
    // 8 x 16: 148 168 155 us, by cp.async 138 158 140)
    typename P::Args a = A;
    if (P::prepare_tma(a, ORD, DIR, C, W)) {
      if constexpr (DIR == 0 && P::kSlab)
        if (slab) return launch_sweep_kernel<P, ORD, DIR, C, W, true, true, false>(a, grid, st);
      return launch_sweep_kernel<P, ORD, DIR, C, W, true, false, false>(a, grid, st);
    }
  }
  if constexpr (DIR == 0 && P::kSlab && base)
    if (slab) return launch_sweep_kernel<P, ORD, DIR, C, W, false, true, false>(A, grid, st);
  return launch_sweep_kernel<P, ORD, DIR, C, W, false, false, !base>(A, grid, st);
}

// Time of a sweep of `tiles` CTAs marching along lines of L cells in chunks of C, in units of
// the chunk latency of an SM's only CTA: ceil(L/C) chunks, and an epilogue where no lane of
// the last one is free, each as long as the CTAs that share an SM make it. Measured with the
// FP64 ord-5 sweep: 5.9 us for one CTA per SM, 8 for two, 10.5 for three, 13 for four, the
// most; the tiles of a grid take equally long, so an SM runs its share `slots` (4) at a time,
// each CTA after the first adding `share` (0.4) to the latency. Ord 9, two CTAs (FP64) or
// three (FP32) per SM: 20.5 us for one FP64 CTA, 24.6 for two; FP32 4.4, 5.2 and 6.
inline double sweep_cost(int C, int L, long tiles, int nsm, bool ends, int slots, double share) {
  const long k = (tiles + nsm - 1) / nsm;  // of the busiest SM
  const double full = 1 + share * (slots - 1), rest = k % slots ? 1 + share * (k % slots - 1) : 0.0;
  return ((L + C - 1) / C + (ends && L % C ? 0.0 : 0.35)) * (k / slots * full + rest);
}

// The single-grid sweep of a policy whose PolicyShapes lists further shapes takes its first
// one (PolicyShape, the best on large grids) unless another is 5% cheaper by sweep_cost
// times its own factor: a small grid has too few lines to fill the chip W at a time, and
// marches along them in ceil(L/C) dependent chunks, so it wants more cells of a line at once
// (C up to 128) and fewer lines per CTA. The factor is what a shape's narrower rows (y, z:
// W elements) or its barriers (C > 32) cost on a full chip. Measured, us for the x, y and z
// splits, PolicyShape -> the rule: FP64 32x32x16 18.6 32.9 22.7 -> 13.8 14.4 14.6, 64x64x32
// 37.3 57.7 43.3 -> 35.2 37.2 37.8, 97x61x45 (walls) 78.4 90.7 75.8 -> 76.5 62.0 72.2,
// 400x1x200 150 - 190 -> 37.3 - 28.9; FP32 64x64x32 25.0 43.3 29.0 -> 16.8 20.8 18.9,
// 97x61x45 39.4 49.6 41.5 -> 33.4 25.2 31.2, 400x1x200 120 - 129 -> 18.6 - 18.7.
template <class P, int ORD, int DIR, class = void> struct PolicyShapes { static constexpr int n = 0; };

// the index in PolicyShapes of the shape that a sweep takes, -1 for PolicyShape
template <class P, int ORD, int DIR> int sweep_shape(const typename P::Args &A) {
  using B = PolicyShape<P, ORD, DIR>;
  constexpr int BW = B::W / P::kWdiv > 0 ? B::W / P::kWdiv : 1;
  using S = PolicyShapes<P, ORD, DIR>;
  int best = -1;
  if constexpr (S::n > 0) {
    const int L = DIR == 0 ? A.nx : (DIR == 1 ? A.ny : A.nz);
    const int across = DIR == 0 ? A.ny : A.nx;  // lines of one plane, W to a tile
    const long planes = DIR == 2 ? A.ny : A.nz;
    constexpr int slots = ORD == 5 ? 4 : (P::min_blocks(ORD) > 2 ? P::min_blocks(ORD) : 2);
    constexpr double share = ORD == 5 ? 0.4 : 0.2;
    double cost = 0.95 * P::base_factor(A, stages_by_tma<P, ORD, DIR, B::C>()) *
                  sweep_cost(B::C, L, (across + BW - 1) / BW * planes, A.nsm, false, slots, share);
    for (int i = 0; i < S::n; i++) {
      const double c = S::factor[i] * sweep_cost(S::C[i], L, (across + S::W[i] - 1) / S::W[i] * planes, A.nsm, true, slots, share);
      if (c < cost) { best = i; cost = c; }
    }
    if constexpr (DIR == 0 && P::kSlab) {
      if (A.xh[0] != nullptr || A.xh[1] != nullptr) best = -1;
    }
  }
  return best;
}

template <class P, int ORD, int DIR>
cudaError_t launch_sweep_t(const typename P::Args &A, cudaStream_t st) {
  using B = PolicyShape<P, ORD, DIR>;
  constexpr int BW = B::W / P::kWdiv > 0 ? B::W / P::kWdiv : 1;
  using S = PolicyShapes<P, ORD, DIR>;
  if constexpr (S::n > 0) {
    const int best = sweep_shape<P, ORD, DIR>(A);
    if (best == 0) return launch_sweep_shape<P, ORD, DIR, S::C[0], S::W[0]>(A, st);
    if constexpr (S::n > 1) if (best == 1) return launch_sweep_shape<P, ORD, DIR, S::C[1], S::W[1]>(A, st);
    if constexpr (S::n > 2) if (best == 2) return launch_sweep_shape<P, ORD, DIR, S::C[2], S::W[2]>(A, st);
    if constexpr (S::n > 3) if (best == 3) return launch_sweep_shape<P, ORD, DIR, S::C[3], S::W[3]>(A, st);
    static_assert(S::n <= 4, "shape dispatch");
  }
  return launch_sweep_shape<P, ORD, DIR, B::C, BW>(A, st);
}

template <class P>
cudaError_t launch_sweep_any(int ord, int dir, const typename P::Args &A, cudaStream_t st) {
  if (ord == 5) {
    if (dir == 0) return launch_sweep_t<P, 5, 0>(A, st);
    if (dir == 1) return launch_sweep_t<P, 5, 1>(A, st);
    return launch_sweep_t<P, 5, 2>(A, st);
  }
  if (dir == 0) return launch_sweep_t<P, 9, 0>(A, st);
  if (dir == 1) return launch_sweep_t<P, 9, 1>(A, st);
  return launch_sweep_t<P, 9, 2>(A, st);
}

// What a launch with these arguments takes (diagnostics): C, W, and whether its rows come by TMA.
template <class P, int ORD, int DIR> SweepChoice sweep_choice_t(typename P::Args A) {
  using B = PolicyShape<P, ORD, DIR>;
  using S = PolicyShapes<P, ORD, DIR>;
  const int i = sweep_shape<P, ORD, DIR>(A);
  if constexpr (S::n > 0) if (i >= 0) return SweepChoice{S::C[i], S::W[i], 0};
  SweepChoice c{B::C, B::W / P::kWdiv > 0 ? B::W / P::kWdiv : 1, 0};
  if constexpr (stages_by_tma<P, ORD, DIR, B::C>()) c.tma = P::prepare_tma(A, ORD, DIR, c.C, c.W);
  return c;
}
template <class P> SweepChoice sweep_choice_any(int ord, int dir, const typename P::Args &A) {
  if (ord == 5) return dir == 0 ? sweep_choice_t<P, 5, 0>(A) : (dir == 1 ? sweep_choice_t<P, 5, 1>(A) : sweep_choice_t<P, 5, 2>(A));
  return dir == 0 ? sweep_choice_t<P, 9, 0>(A) : (dir == 1 ? sweep_choice_t<P, 9, 1>(A) : sweep_choice_t<P, 9, 2>(A));
}

}  // namespace awfl
