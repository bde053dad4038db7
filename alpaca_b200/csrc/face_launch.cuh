// Launchers of the run-time selected schemes' kernels (face_flux_ext.cu,
// sweep_ext.cu), called by the dispatchers of the compiled default's units.
#pragma once

#include "kernels.cuh"

namespace alp {

cudaError_t face_flux_ext(Launch const &L, int dir, bool accumulate, dim3 grid, double *F,
                          long long stride, int threads);
cudaError_t face_flux_all_ext(Launch const &L, dim3 grid, int const *nbr26,
                              CaseState const *cases, double *F, long long stride,
                              long long dstride, int threads);
cudaError_t sweep_ext(Launch const &L, int grid, int threads, double const *U0, double *Uout,
                      double const *F, long long stride, long long dstride, int const *nbr26,
                      CaseState const *cases, int stage, int rows, int units);

}  // namespace alp
