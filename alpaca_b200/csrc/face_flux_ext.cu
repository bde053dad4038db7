// Face-flux kernels of the run-time selected schemes.
#include "face_launch.cuh"
#include "face_kernels.cuh"

namespace alp {
namespace {

// The same two kernels for the run-time selected schemes (ExtPolicy, FP64).
template <int DIM, int DIR, int SCHEME, bool ACCUM, int W>
__global__ void __launch_bounds__(128)
face_flux_ext_kernel(double const *__restrict__ U, int const *__restrict__ work,
                     BlockMeta const *__restrict__ meta, BlockMeta def, double *__restrict__ F,
                     long long stride, ExtPolicy pol, unsigned long long const *__restrict__ glf) {
  int const t = blockIdx.y * blockDim.x + threadIdx.x;
  if (t >= FaceMap<DIM, DIR>::COUNT) return;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  face_flux<DIM, DIR, SCHEME, double, ACCUM, false, ExtPolicy, W>(U, nullptr, slot, item, t, bm, F,
                                                               stride, block_policy(pol, bm, glf));
}

template <int DIM, int SCHEME, int W>
__global__ void __launch_bounds__(128)
face_flux_all_ext_kernel(double const *__restrict__ U, int const *__restrict__ work,
                         BlockMeta const *__restrict__ meta, int const *__restrict__ nbr26,
                         CaseState const *__restrict__ cases, double *__restrict__ F,
                         long long stride, long long dstride, ExtPolicy pol0,
                         unsigned long long const *__restrict__ glf,
                         int const *__restrict__ items) {
  int const t = blockIdx.y * blockDim.x + threadIdx.x;
  int const item = items ? items[blockIdx.x] : (int)blockIdx.x;
  int const slot = work[item];
  BlockMeta const bm = meta[slot];
  if (!(cases[bm.case_id].dt > 0.0)) return;
  ExtPolicy const pol = block_policy(pol0, bm, glf);
  int const dir = blockIdx.z;
  if (dir == 0) {
    if (t < FaceMap<DIM, 0>::COUNT)
      face_flux<DIM, 0, SCHEME, double, false, true, ExtPolicy, W>(U, nbr26, slot, item, t, bm, F,
                                                                stride, pol);
  } else if (DIM > 1 && dir == 1) {
    if (t < FaceMap<DIM, 1>::COUNT)
      face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, double, false, true, ExtPolicy, W>(
          U, nbr26, slot, item, t, bm, F + dstride, stride, pol);
  } else if (DIM > 2) {
    if (t < FaceMap<DIM, 2>::COUNT)
      face_flux<DIM, (DIM > 2 ? 2 : 0), SCHEME, double, false, true, ExtPolicy, W>(
          U, nbr26, slot, item, t, bm, F + 2 * dstride, stride, pol);
  }
}

template <int DIM, int DIR, bool ACC, int W>
cudaError_t ext_dir(Launch const &L, dim3 grid, double *F, long long stride,
                              int threads) {
  ExtPolicy const pol{L.opt};
  switch (L.scheme) {
    case FV_CHAR:
      face_flux_ext_kernel<DIM, DIR, FV_CHAR, ACC, W>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, pol, L.glf);
      break;
    case FV_PRIM:
      face_flux_ext_kernel<DIM, DIR, FV_PRIM, ACC, W>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, pol, L.glf);
      break;
    case FS_ROE:
      face_flux_ext_kernel<DIM, DIR, FS_ROE, ACC, W>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, pol, L.glf);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int DIM, int DIR>
cudaError_t ext_any(Launch const &L, bool acc, dim3 grid, double *F, long long stride, int threads) {
  if (ext_wide(L.opt))
    return acc ? ext_dir<DIM, DIR, true, 8>(L, grid, F, stride, threads)
               : ext_dir<DIM, DIR, false, 8>(L, grid, F, stride, threads);
  return acc ? ext_dir<DIM, DIR, true, 6>(L, grid, F, stride, threads)
             : ext_dir<DIM, DIR, false, 6>(L, grid, F, stride, threads);
}

template <int DIM, int W>
cudaError_t all_ext(Launch const &L, dim3 grid, int const *nbr26, CaseState const *cases,
                              double *F, long long stride, long long dstride, int threads) {
  ExtPolicy const pol{L.opt};
  switch (L.scheme) {
    case FV_CHAR:
      face_flux_all_ext_kernel<DIM, FV_CHAR, W><<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, pol, L.glf, L.items);
      break;
    case FV_PRIM:
      face_flux_all_ext_kernel<DIM, FV_PRIM, W><<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, pol, L.glf, L.items);
      break;
    case FS_ROE:
      face_flux_all_ext_kernel<DIM, FS_ROE, W><<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, pol, L.glf, L.items);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int DIM>
cudaError_t all_any(Launch const &L, dim3 grid, int const *nbr26, CaseState const *cases, double *F,
                    long long stride, long long dstride, int threads) {
  return ext_wide(L.opt) ? all_ext<DIM, 8>(L, grid, nbr26, cases, F, stride, dstride, threads)
                         : all_ext<DIM, 6>(L, grid, nbr26, cases, F, stride, dstride, threads);
}
}  // namespace

cudaError_t face_flux_ext(Launch const &L, int dir, bool acc, dim3 grid, double *F,
                          long long stride, int threads) {
  switch (L.dim * 3 + dir) {
    case 3: return ext_any<1, 0>(L, acc, grid, F, stride, threads);
    case 6: return ext_any<2, 0>(L, acc, grid, F, stride, threads);
    case 7: return ext_any<2, 1>(L, acc, grid, F, stride, threads);
    case 9: return ext_any<3, 0>(L, acc, grid, F, stride, threads);
    case 10: return ext_any<3, 1>(L, acc, grid, F, stride, threads);
    case 11: return ext_any<3, 2>(L, acc, grid, F, stride, threads);
  }
  return cudaErrorInvalidValue;
}

cudaError_t face_flux_all_ext(Launch const &L, dim3 grid, int const *nbr26,
                              CaseState const *cases, double *F, long long stride,
                              long long dstride, int threads) {
  switch (L.dim) {
    case 1: return all_any<1>(L, grid, nbr26, cases, F, stride, dstride, threads);
    case 2: return all_any<2>(L, grid, nbr26, cases, F, stride, dstride, threads);
    case 3: return all_any<3>(L, grid, nbr26, cases, F, stride, dstride, threads);
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
