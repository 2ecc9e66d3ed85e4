// Ensemble (batched) sweeps of the FP32 form: the persistent kernels of awfl_ens.cuh
// instantiated for the P32 policy, sm_100a. Same flags as awfl_fp32.cu.
#include <cuda_runtime.h>

// 640 threads' registers per SM at ord 5 (at most 102 a thread): the persistent sweeps then
// hold 5 CTAs of 128 threads per SM like the single-grid FP32 sweep (24 members of 32..96
// cells a side, two steps: 1.366 ms, against 1.402 at 512)
#ifndef AWFL_ENS_THREADS_PER_SM_ORD5
#define AWFL_ENS_THREADS_PER_SM_ORD5 640
#endif
#include "awfl_ens.cuh"
#include "awfl_fp32.cuh"

namespace awfl {

cudaError_t ens_run_fp32(int ord, int dir, int shape, const EnsList<SweepArgs32> *E, int grid, int *occ,
                         cudaStream_t st) {
  return ens_run<P32>(ord, dir, shape, E, grid, occ, st);
}

cudaError_t upload_tables_ens32(int ord, const double *recon, const double *c2g, const double *s2g,
                                const double *deriv, const double *idl, double sigma, const double *wts) {
  return upload_tables32_here(ord, recon, c2g, s2g, deriv, idl, sigma, wts);
}

}  // namespace awfl
