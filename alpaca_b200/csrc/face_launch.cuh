// Launchers of the run-time selected schemes' kernels, one set per
// reconstruction stencil (ext_*.cu), and their dispatch.
#pragma once

#include "kernels.cuh"

namespace alp {

// Flux arrays of the directions of a drop-in call.
struct FluxPtrs {
  double *d[3];
};

template <int ST> struct ExtKernels {
  static cudaError_t face(Launch const &L, bool accumulate, dim3 grid, int chunks,
                          FluxPtrs const &F, long long stride, int threads);
  static cudaError_t face_all(Launch const &L, dim3 grid, int chunks, int const *nbr26,
                              CaseState const *cases, double *F, long long stride,
                              long long dstride, int threads);
  static cudaError_t sweep(Launch const &L, int grid, int threads, double const *U0, double *Uout,
                           double const *F, long long stride, long long dstride, int const *nbr26,
                           CaseState const *cases, int stage, int rows, int units);
};

// f(ExtKernels of the launch's stencil)
template <typename Fn> cudaError_t with_stencil(Launch const &L, Fn const &f) {
  switch (L.opt.stencil) {
    case ST_FIRST_ORDER: return f(ExtKernels<ST_FIRST_ORDER>());
    case ST_WENO3: return f(ExtKernels<ST_WENO3>());
    case ST_WENO5: return f(ExtKernels<ST_WENO5>());
    case ST_WENO5Z: return f(ExtKernels<ST_WENO5Z>());
    case ST_TENO5: return f(ExtKernels<ST_TENO5>());
    case ST_WENO7: return f(ExtKernels<ST_WENO7>());
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
