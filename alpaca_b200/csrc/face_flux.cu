// Face-flux kernels of the compiled default schemes and the dispatch of every
// face-flux launch.
#include "face_launch.cuh"
#include "face_kernels.cuh"

namespace alp {
namespace {

// Every direction of all work items in one launch (drop-in calls: halos from
// the buffer); direction blockIdx.z goes to F.d[blockIdx.z]. A call with one
// block has 34 CTAs per direction: side by side they take 6 us, one launch
// after the other 17 us.
template <int DIM, int SCHEME, typename T, bool ACCUM>
__global__ void __launch_bounds__(128, FaceOccupancy<DIM, SCHEME, T>::min_ctas)
face_flux_kernel(double const *__restrict__ U, int const *__restrict__ work,
                 BlockMeta const *__restrict__ meta, BlockMeta def, FluxPtrs F, long long stride,
                 int chunks) {
  int const item = blockIdx.x / chunks;
  int const t = (int)(blockIdx.x - item * chunks) * blockDim.x + threadIdx.x;
  if (t >= FaceMap<DIM, 0>::COUNT) return;  // as many faces in every direction
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  int const dir = blockIdx.z;
  if (dir == 0)
    face_flux<DIM, 0, SCHEME, T, ACCUM, false>(U, nullptr, slot, item, t, bm, F.d[0], stride);
  else if (DIM > 1 && dir == 1)
    face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, T, ACCUM, false>(U, nullptr, slot, item, t, bm,
                                                                F.d[1], stride);
  else if (DIM > 2)
    face_flux<DIM, (DIM > 2 ? 2 : 0), SCHEME, T, ACCUM, false>(U, nullptr, slot, item, t, bm,
                                                                F.d[2], stride);
}

// Every direction of every work item in one launch (engine): blockIdx.z is the
// direction, stencils gathered from neighbours, direction d written to
// F + d * dstride. Items whose case is inactive (dt == 0) are skipped.
template <int DIM, int SCHEME, typename T>
__global__ void __launch_bounds__(128, FaceOccupancy<DIM, SCHEME, T>::min_ctas)
face_flux_all_kernel(double const *__restrict__ U, int const *__restrict__ work,
                     BlockMeta const *__restrict__ meta, int const *__restrict__ nbr26,
                     CaseState const *__restrict__ cases, double *__restrict__ F,
                     long long stride, long long dstride, int chunks,
                     int const *__restrict__ items) {
  // grid (items x chunks, 1, dir): an item's chunks are consecutive, so the
  // CTAs resident at any time share few blocks' stencils (a few MB of L2
  // instead of one stencil plane of every item in the launch). items (when
  // given): the work-list position of each launch position
  int const chunk = (int)(blockIdx.x % chunks);
  int const pos = (int)(blockIdx.x / chunks);
  int const item = items ? items[pos] : pos;
  int const t = chunk * blockDim.x + threadIdx.x;
  int const slot = work[item];
  BlockMeta const bm = meta[slot];
  if (!(cases[bm.case_id].dt > 0.0)) return;
  int const dir = blockIdx.z;
  if (dir == 0) {
    if (t < FaceMap<DIM, 0>::COUNT)
      face_flux<DIM, 0, SCHEME, T, false, true>(U, nbr26, slot, item, t, bm, F, stride);
  } else if (DIM > 1 && dir == 1) {
    if (t < FaceMap<DIM, 1>::COUNT)
      face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, T, false, true>(U, nbr26, slot, item, t, bm,
                                                                 F + dstride, stride);
  } else if (DIM > 2) {
    if (t < FaceMap<DIM, 2>::COUNT)
      face_flux<DIM, (DIM > 2 ? 2 : 0), SCHEME, T, false, true>(U, nbr26, slot, item, t, bm,
                                                                 F + 2 * dstride, stride);
  }
}

template <int DIM, typename T, bool ACC>
cudaError_t face_flux_dim(Launch const &L, FluxPtrs const &F, long long stride) {
  constexpr int threads = 128;
  int const chunks = (FaceMap<DIM, 0>::COUNT + threads - 1) / threads;
  if ((long long)L.nwork * chunks > 0x7fffffffLL) return cudaErrorInvalidValue;
  dim3 const grid((unsigned)(L.nwork * chunks), 1, DIM);
  if (!L.opt.is_default())
    return with_stencil(L, [&](auto k) {
      return decltype(k)::face(L, ACC, grid, chunks, F, stride, threads);
    });
  switch (L.scheme) {
    case FV_CHAR:
      face_flux_kernel<DIM, FV_CHAR, T, ACC>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, chunks);
      break;
    case FV_PRIM:
      face_flux_kernel<DIM, FV_PRIM, T, ACC>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, chunks);
      break;
    case FS_ROE:
      face_flux_kernel<DIM, FS_ROE, T, ACC>
          <<<grid, threads, 0, L.stream>>>(L.U, L.work, L.meta, L.def, F, stride, chunks);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <typename T, bool ACC>
cudaError_t face_flux_t(Launch const &L, FluxPtrs const &F, long long stride) {
  switch (L.dim) {
    case 1: return face_flux_dim<1, T, ACC>(L, F, stride);
    case 2: return face_flux_dim<2, T, ACC>(L, F, stride);
    case 3: return face_flux_dim<3, T, ACC>(L, F, stride);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_face_flux(Launch const &L, double *const F[3], long long stride,
                             bool accumulate) {
  if (L.nwork <= 0) return cudaSuccess;
  if (!L.opt.is_default() && L.precision != FP64) return cudaErrorInvalidValue;
  FluxPtrs const p{{F[0], F[1], F[2]}};
  if (L.precision == FP32_FLUX)
    return accumulate ? face_flux_t<float, true>(L, p, stride) : face_flux_t<float, false>(L, p, stride);
  return accumulate ? face_flux_t<double, true>(L, p, stride) : face_flux_t<double, false>(L, p, stride);
}

namespace {
template <int DIM, typename T>
cudaError_t face_flux_all_t(Launch const &L, int const *nbr26, CaseState const *cases, double *F,
                            long long stride, long long dstride, int threads, int dirs) {
  int const count = (IC + 1) * (DIM > 1 ? IC : 1) * (DIM > 2 ? IC : 1);
  // items x chunks < 2^31 for up to 2^31 / 68 items (64-thread chunks)
  int const chunks = (count + threads - 1) / threads;
  if ((long long)L.nwork * chunks > 0x7fffffffLL) return cudaErrorInvalidValue;
  dim3 const g2((unsigned)(L.nwork * chunks), 1, dirs);
  if (!L.opt.is_default())
    return with_stencil(L, [&](auto k) {
      return decltype(k)::face_all(L, g2, chunks, nbr26, cases, F, stride, dstride, threads);
    });
  switch (L.scheme) {
    case FV_CHAR:
      face_flux_all_kernel<DIM, FV_CHAR, T><<<g2, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, chunks, L.items);
      break;
    case FV_PRIM:
      face_flux_all_kernel<DIM, FV_PRIM, T><<<g2, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, chunks, L.items);
      break;
    case FS_ROE:
      face_flux_all_kernel<DIM, FS_ROE, T><<<g2, threads, 0, L.stream>>>(L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, chunks, L.items);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_face_flux_all(Launch const &L, int const *nbr26, CaseState const *cases,
                                 double *F, long long stride, long long dstride, int threads,
                                 int dirs) {
  if (L.nwork <= 0) return cudaSuccess;
  if (dirs <= 0) dirs = L.dim;
  if (dirs > L.dim) return cudaErrorInvalidValue;
  if (!L.work || !L.meta || !nbr26 || !cases) return cudaErrorInvalidValue;
  if (threads <= 0) threads = 128;
  if (threads > 128 || (threads & 31)) return cudaErrorInvalidValue;
  if (!L.opt.is_default() && L.precision != FP64) return cudaErrorInvalidValue;
  bool const f32 = L.precision == FP32_FLUX;
  switch (L.dim) {
    case 1: return f32 ? face_flux_all_t<1, float>(L, nbr26, cases, F, stride, dstride, threads, dirs)
                       : face_flux_all_t<1, double>(L, nbr26, cases, F, stride, dstride, threads, dirs);
    case 2: return f32 ? face_flux_all_t<2, float>(L, nbr26, cases, F, stride, dstride, threads, dirs)
                       : face_flux_all_t<2, double>(L, nbr26, cases, F, stride, dstride, threads, dirs);
    case 3: return f32 ? face_flux_all_t<3, float>(L, nbr26, cases, F, stride, dstride, threads, dirs)
                       : face_flux_all_t<3, double>(L, nbr26, cases, F, stride, dstride, threads, dirs);
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
