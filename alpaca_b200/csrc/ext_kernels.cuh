// Kernels of the run-time selected schemes with reconstruction stencil ST
// (ExtPolicy, FP64): the drop-in and engine face fluxes and the last direction
// fused with the stage update. One unit per stencil (ext_*.cu) compiles them.
#pragma once

#include "face_launch.cuh"
#include "sweep.cuh"

namespace alp {
namespace {

// WENO7 reads 8-cell stencils (i-3 .. i+4), the others 6 cells (i-2 .. i+3).
__host__ __device__ constexpr int ext_width(int st) { return st == ST_WENO7 ? 8 : 6; }
// CTAs of 128 threads per SM (168 registers at 3); the 8-cell stencils hold a
// third more state. In 1D the state is three fields: 5 CTAs (96 registers), and 4
// for flux splitting and the 8-cell stencils. Step of 20,000 1D blocks in us, at the
// 2 or 3 CTAs of the other dimensions against 4 or 5: WENO7 FV char 734 / 301, Roe-M
// 745 / 330, WENO5-Z 312 / 217, HLL 259 / 223, LLF 320 / 251; 600 blocks 45 / 35, 49 /
// 41, 33 / 29, 35 / 29, 33 / 33.
__host__ __device__ constexpr int ext_ctas(int dim, int scheme, int st) {
  if (dim == 1) return st == ST_WENO7 || scheme == FS_ROE ? 4 : 5;
  return st == ST_WENO7 ? 2 : 3;
}

template <int DIM, int SCHEME, int ST, bool ACCUM>
__global__ void __launch_bounds__(128, ext_ctas(DIM, SCHEME, ST))
face_flux_ext_kernel(double const *__restrict__ U, int const *__restrict__ work,
                     BlockMeta const *__restrict__ meta, BlockMeta def, FluxPtrs F, long long stride,
                     int chunks, ExtPolicy<ST> pol0, unsigned long long const *__restrict__ glf) {
  constexpr int W = ext_width(ST);
  using P = ExtPolicy<ST>;
  int const item = blockIdx.x / chunks;
  int const t = (int)(blockIdx.x - item * chunks) * blockDim.x + threadIdx.x;
  if (t >= FaceMap<DIM, 0>::COUNT) return;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  P const pol = block_policy(pol0, bm, glf);
  int const dir = blockIdx.z;
  if (dir == 0)
    face_flux<DIM, 0, SCHEME, double, ACCUM, false, P, W>(U, nullptr, slot, item, t, bm, F.d[0],
                                                          stride, pol);
  else if (DIM > 1 && dir == 1)
    face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, double, ACCUM, false, P, W>(
        U, nullptr, slot, item, t, bm, F.d[1], stride, pol);
  else if (DIM > 2)
    face_flux<DIM, (DIM > 2 ? 2 : 0), SCHEME, double, ACCUM, false, P, W>(
        U, nullptr, slot, item, t, bm, F.d[2], stride, pol);
}

template <int DIM, int SCHEME, int ST>
__global__ void __launch_bounds__(128, ext_ctas(DIM, SCHEME, ST))
face_flux_all_ext_kernel(double const *__restrict__ U, int const *__restrict__ work,
                         BlockMeta const *__restrict__ meta, int const *__restrict__ nbr26,
                         CaseState const *__restrict__ cases, double *__restrict__ F,
                         long long stride, long long dstride, int chunks, ExtPolicy<ST> pol0,
                         unsigned long long const *__restrict__ glf,
                         int const *__restrict__ items) {
  constexpr int W = ext_width(ST);
  using P = ExtPolicy<ST>;
  int const pos = blockIdx.x / chunks;
  int const t = (int)(blockIdx.x - pos * chunks) * blockDim.x + threadIdx.x;
  if (t >= FaceMap<DIM, 0>::COUNT) return;
  int const item = items ? items[pos] : pos;
  int const slot = work[item];
  BlockMeta const bm = meta[slot];
  if (!(cases[bm.case_id].dt > 0.0)) return;
  P const pol = block_policy(pol0, bm, glf);
  int const dir = blockIdx.z;
  if (dir == 0)
    face_flux<DIM, 0, SCHEME, double, false, true, P, W>(U, nbr26, slot, item, t, bm, F, stride,
                                                         pol);
  else if (DIM > 1 && dir == 1)
    face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, double, false, true, P, W>(
        U, nbr26, slot, item, t, bm, F + dstride, stride, pol);
  else if (DIM > 2)
    face_flux<DIM, (DIM > 2 ? 2 : 0), SCHEME, double, false, true, P, W>(
        U, nbr26, slot, item, t, bm, F + 2 * dstride, stride, pol);
}

template <int DIM, int SCHEME, int ST>
__global__ void
__launch_bounds__(32 * kSweepWarps, ext_ctas(DIM, SCHEME, ST) * 4 / kSweepWarps)
sweep_update_ext_kernel(double const *Uin, double const *U0, double *Uout,
                        int const *__restrict__ work, BlockMeta const *__restrict__ meta,
                        int const *__restrict__ nbr26, CaseState const *__restrict__ cases,
                        double const *F, long long stride, long long dstride, int stage, int rows,
                        int nunits, ExtPolicy<ST> pol, unsigned long long const *__restrict__ glf) {
  __shared__ double high[kSweepWarps][DIM + 2][32];
  sweep_update<DIM, SCHEME, double, ExtPolicy<ST>, ext_width(ST)>(
      Uin, U0, Uout, work, meta, nbr26, cases, F, stride, dstride, stage, rows, nunits, pol, glf,
      high);
}

// The scheme of a launch as a compile-time value: f(integral constant).
template <int V> struct Const {
  static constexpr int value = V;
};
template <typename Fn> cudaError_t with_scheme(int scheme, Fn const &f) {
  switch (scheme) {
    case FV_CHAR: f(Const<FV_CHAR>()); break;
    case FV_PRIM: f(Const<FV_PRIM>()); break;
    case FS_ROE: f(Const<FS_ROE>()); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
template <typename Fn> cudaError_t with_dim(int dim, Fn const &f) {
  switch (dim) {
    case 1: return f(Const<1>());
    case 2: return f(Const<2>());
    case 3: return f(Const<3>());
  }
  return cudaErrorInvalidValue;
}

}  // namespace

template <int ST>
cudaError_t ExtKernels<ST>::face(Launch const &L, bool acc, dim3 grid, int chunks,
                                 FluxPtrs const &F, long long stride, int threads) {
  ExtPolicy<ST> const pol{L.opt};
  return with_dim(L.dim, [&](auto d) {
    constexpr int D = decltype(d)::value;
    return with_scheme(L.scheme, [&](auto s) {
      constexpr int S = decltype(s)::value;
      if (acc)
        face_flux_ext_kernel<D, S, ST, true><<<grid, threads, 0, L.stream>>>(
            L.U, L.work, L.meta, L.def, F, stride, chunks, pol, L.glf);
      else
        face_flux_ext_kernel<D, S, ST, false><<<grid, threads, 0, L.stream>>>(
            L.U, L.work, L.meta, L.def, F, stride, chunks, pol, L.glf);
    });
  });
}

template <int ST>
cudaError_t ExtKernels<ST>::face_all(Launch const &L, dim3 grid, int chunks, int const *nbr26,
                                     CaseState const *cases, double *F, long long stride,
                                     long long dstride, int threads) {
  ExtPolicy<ST> const pol{L.opt};
  return with_dim(L.dim, [&](auto d) {
    constexpr int D = decltype(d)::value;
    return with_scheme(L.scheme, [&](auto s) {
      face_flux_all_ext_kernel<D, decltype(s)::value, ST><<<grid, threads, 0, L.stream>>>(
          L.U, L.work, L.meta, nbr26, cases, F, stride, dstride, chunks, pol, L.glf, L.items);
    });
  });
}

template <int ST>
cudaError_t ExtKernels<ST>::sweep(Launch const &L, int grid, int threads, double const *U0,
                                  double *Uout, double const *F, long long stride,
                                  long long dstride, int const *nbr26, CaseState const *cases,
                                  int stage, int rows, int units) {
  if (L.dim < 2) return cudaErrorInvalidValue;
  ExtPolicy<ST> const pol{L.opt};
  return with_dim(L.dim, [&](auto d) {
    constexpr int D = decltype(d)::value < 2 ? 2 : decltype(d)::value;
    return with_scheme(L.scheme, [&](auto s) {
      sweep_update_ext_kernel<D, decltype(s)::value, ST><<<grid, threads, 0, L.stream>>>(
          L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, units, pol,
          L.glf);
    });
  });
}

}  // namespace alp
