// The last direction's faces fused with the stage update: run-time selected
// schemes.
#include "face_launch.cuh"
#include "sweep.cuh"

namespace alp {
namespace {

template <int DIM, int SCHEME, int W>
__global__ void __launch_bounds__(32 * kSweepWarps)
sweep_update_ext_kernel(double const *Uin, double const *U0, double *Uout,
                        int const *__restrict__ work, BlockMeta const *__restrict__ meta,
                        int const *__restrict__ nbr26, CaseState const *__restrict__ cases,
                        double const *__restrict__ F, long long stride, long long dstride, int stage,
                        int rows,
                        int nunits, ExtPolicy pol, unsigned long long const *__restrict__ glf) {
  __shared__ double high[kSweepWarps][DIM + 2][32];
  sweep_update<DIM, SCHEME, double, ExtPolicy, W>(Uin, U0, Uout, work, meta, nbr26, cases, F,
                                                  stride, dstride, stage, rows, nunits, pol, glf,
                                                  high);
}

template <int DIM, int W>
cudaError_t sweep_w(Launch const &L, int grid, int th, double const *U0, double *Uout, double const *F,
                      long long stride, long long dstride, int const *nbr26,
                      CaseState const *cases, int stage, int rows, int units) {
  ExtPolicy const pol{L.opt};
  switch (L.scheme) {
    case FV_CHAR:
      sweep_update_ext_kernel<DIM, FV_CHAR, W><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, units, pol, L.glf);
      break;
    case FV_PRIM:
      sweep_update_ext_kernel<DIM, FV_PRIM, W><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, units, pol, L.glf);
      break;
    case FS_ROE:
      sweep_update_ext_kernel<DIM, FS_ROE, W><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, units, pol, L.glf);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t sweep_ext(Launch const &L, int grid, int th, double const *U0, double *Uout,
                      double const *F, long long stride, long long dstride, int const *nbr26,
                      CaseState const *cases, int stage, int rows, int units) {
  bool const wide = ext_wide(L.opt);
  switch (L.dim) {
    case 2: return wide ? sweep_w<2, 8>(L, grid, th, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows, units)
                        : sweep_w<2, 6>(L, grid, th, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows, units);
    case 3: return wide ? sweep_w<3, 8>(L, grid, th, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows, units)
                        : sweep_w<3, 6>(L, grid, th, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows, units);
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
