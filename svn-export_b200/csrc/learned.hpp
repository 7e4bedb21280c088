// Flexible CG, Chebyshev-Jacobi and the training pairs of the plain solver (learned.cu):
// declarations shared with the host runtime.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "device_system.hpp"

namespace mh {

cudaError_t launch_cheb_apply(const DevSystem &sys, const float *r, float *z0, float *z1, float *d, float *z_final,
                              int degree, double lo, double hi, cudaStream_t s, bool follows);
// the rest of a flexible-CG iteration after z = M r (two kernels)
cudaError_t launch_fcg_iteration(const DevSystem &sys, const float *z, cudaStream_t s, bool chained);
cudaError_t launch_spectrum_bound(const DevSystem &sys, unsigned int *out, cudaStream_t s);
cudaError_t launch_pair_make(int64_t n, const double *xs, const double *x, const double *r64, float *e, float *r,
                             double *acc, cudaStream_t s);
cudaError_t launch_pair_scale(int64_t n, float *e, float *r, float scale, cudaStream_t s);

}  // namespace mh
