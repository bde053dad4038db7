// Pencil sweeps (a stepping candidate of the autotuner).
#include "face_kernels.cuh"

namespace alp {
namespace {

// Interior linear index of the cell with index c along DIR at transverse (p1, p2).
template <int DIM, int DIR>
__device__ __forceinline__ int interior_index(int c, int p1, int p2) {
  using M = FaceMap<DIM, DIR>;
  int ci[3] = {0, 0, 0};
  ci[DIR] = c;
  ci[M::O1] = p1;
  ci[M::O2] = p2;
  if constexpr (DIM == 3) return (ci[0] * IC + ci[1]) * IC + ci[2];
  else if constexpr (DIM == 2) return ci[0] * IC + ci[1];
  else return ci[0];
}

// One thread walks a line of 16 cells along DIR: it computes the 17 face
// fluxes in order with a sliding 6-cell stencil window (each cell is loaded
// once per line instead of six times) and forms each cell's flux difference
// F(a-1/2) - F(a+1/2) as soon as both faces are known. The directions run one
// after the other: MODE 0 stores the difference in R, MODE 1 adds to R, MODE 2
// (the last direction) adds, scales by 1/cell size and applies the SSP-RK3
// stage: Uout = (stage ? a0 Uin + a1 U0 : Uin) + c dt rhs. The summation order
// is therefore (dx + dy) + dz instead of the reference's three-order symmetric
// sum (the strict build keeps that one). Stencils are gathered from neighbour
// interiors; cases with dt == 0 are skipped.
template <int DIM, int DIR, int SCHEME, typename T, int MODE>
__global__ void __launch_bounds__(128, FaceOccupancy<DIM, SCHEME>::sweep_ctas)
pencil_kernel(double const *Uin, double const *U0, double *Uout, double *R,
              int const *__restrict__ work, int nwork, BlockMeta const *__restrict__ meta,
              int const *__restrict__ nbr26, CaseState const *__restrict__ cases, int stage) {
  using G = Geo<DIM>;
  using M = FaceMap<DIM, DIR>;
  constexpr int NE = G::NE;
  constexpr int P = M::E1 * M::E2;  // lines per block
  constexpr int step = DIR == 0 ? G::TCY * G::TCZ : (DIR == 1 ? G::TCZ : 1);
  constexpr int lo_slot = DIR == 0 ? 4 : (DIR == 1 ? 10 : 12);
  constexpr int hi_slot = DIR == 0 ? 21 : (DIR == 1 ? 15 : 13);
  int const g = blockIdx.x * blockDim.x + threadIdx.x;
  int const item = g / P;
  if (item >= nwork) return;
  int const p = g - item * P;
  int const p1 = p / M::E2, p2 = p - (p / M::E2) * M::E2;
  int const slot = work[item];
  BlockMeta const bm = meta[slot];
  double const dt = cases[bm.case_id].dt;
  if (!(dt > 0.0)) return;
  Eos const eos{bm.gamma, bm.B, bm.safe};
  double const *blk = Uin + (size_t)slot * G::BLOCK_DOUBLES;
  int const cell0 = line_origin<DIM, DIR>(p1, p2);
  int const nlo = __ldg(nbr26 + (size_t)slot * 26 + lo_slot);
  int const nhi = __ldg(nbr26 + (size_t)slot * 26 + hi_slot);
  double *Rb = R ? R + (size_t)slot * NE * G::INTERIOR : nullptr;

  double w[6][NE];
#pragma unroll
  for (int m = 0; m < 6; ++m)
    stencil_load<DIM, DIR, true>(Uin, blk, HS - 3 + m, cell0, nlo, nhi, w[m]);
  double const ocs = inv(bm.cell_size);
  RkStage const rk = rk_stage(stage, dt);
  double fprev[NE];
#pragma unroll 1
  for (int a = 0; a <= IC; ++a) {
    double f[NE];
    bool const valid = face_compute<DIM, DIR, SCHEME, T>(eos, bm.B, w, f);
#pragma unroll
    for (int n = 0; n < NE; ++n)
      if (!valid) f[n] = 0.0;
    if (a > 0) {
      int const ix = interior_index<DIM, DIR>(a - 1, p1, p2);
      size_t const x = (size_t)slot * G::BLOCK_DOUBLES + cell0 + (HS + a - 1) * step;
#pragma unroll
      for (int n = 0; n < NE; ++n) {
        double const d = fprev[n] - f[n];
        if constexpr (MODE == 0) {
          Rb[n * G::INTERIOR + ix] = d;
        } else if constexpr (MODE == 1) {
          Rb[n * G::INTERIOR + ix] += d;
        } else {
          double const sum = DIM > 1 ? Rb[n * G::INTERIOR + ix] + d : d;
          double const rhs = 0.0 + sum * ocs;
          size_t const xf = x + (size_t)n * G::CELLS;
          Uout[xf] = rk_apply(rk, Uin[xf], rk.first ? 0.0 : U0[xf], rhs);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NE; ++n) fprev[n] = f[n];
    if (a < IC) {
#pragma unroll
      for (int m = 0; m < 5; ++m)
#pragma unroll
        for (int n = 0; n < NE; ++n) w[m][n] = w[m + 1][n];
      stencil_load<DIM, DIR, true>(Uin, blk, HS + a + 3, cell0, nlo, nhi, w[5]);
    }
  }
}

}  // namespace

namespace {
template <int DIM, int DIR, typename T, int MODE>
cudaError_t pencil_t(Launch const &L, double const *U0, double *Uout, double *R, int const *nbr26,
                     CaseState const *cases, int stage) {
  constexpr int P = FaceMap<DIM, DIR>::E1 * FaceMap<DIM, DIR>::E2;
  long long const threads = (long long)L.nwork * P;
  dim3 grid((unsigned)((threads + 127) / 128));
  switch (L.scheme) {
    case FV_CHAR:
      pencil_kernel<DIM, DIR, FV_CHAR, T, MODE><<<grid, 128, 0, L.stream>>>(L.U, U0, Uout, R, L.work, L.nwork, L.meta, nbr26, cases, stage);
      break;
    case FV_PRIM:
      pencil_kernel<DIM, DIR, FV_PRIM, T, MODE><<<grid, 128, 0, L.stream>>>(L.U, U0, Uout, R, L.work, L.nwork, L.meta, nbr26, cases, stage);
      break;
    case FS_ROE:
      pencil_kernel<DIM, DIR, FS_ROE, T, MODE><<<grid, 128, 0, L.stream>>>(L.U, U0, Uout, R, L.work, L.nwork, L.meta, nbr26, cases, stage);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int DIM, typename T>
cudaError_t pencil_dim(Launch const &L, double const *U0, double *Uout, double *R, int const *nbr26,
                       CaseState const *cases, int stage) {
  if (cudaError_t e = pencil_t<DIM, 0, T, DIM == 1 ? 2 : 0>(L, U0, Uout, R, nbr26, cases, stage))
    return e;
  if constexpr (DIM > 1)
    if (cudaError_t e = pencil_t<DIM, (DIM > 1 ? 1 : 0), T, DIM == 2 ? 2 : 1>(L, U0, Uout, R, nbr26, cases, stage))
      return e;
  if constexpr (DIM > 2)
    if (cudaError_t e = pencil_t<DIM, (DIM > 2 ? 2 : 0), T, 2>(L, U0, Uout, R, nbr26, cases, stage))
      return e;
  return cudaSuccess;
}
}  // namespace

cudaError_t launch_pencil_stage(Launch const &L, double const *U0, double *Uout, double *R,
                                int const *nbr26, CaseState const *cases, int stage) {
  if (L.nwork <= 0) return cudaSuccess;
  if (!L.work || !L.meta || !nbr26 || !cases || stage < 0 || stage > 2) return cudaErrorInvalidValue;
  if (L.dim > 1 && !R) return cudaErrorInvalidValue;
  if (!L.opt.is_default()) return cudaErrorInvalidValue;  // pencils: default schemes only
  bool const f32 = L.precision == FP32_FLUX;
  switch (L.dim) {
    case 1: return f32 ? pencil_dim<1, float>(L, U0, Uout, R, nbr26, cases, stage)
                       : pencil_dim<1, double>(L, U0, Uout, R, nbr26, cases, stage);
    case 2: return f32 ? pencil_dim<2, float>(L, U0, Uout, R, nbr26, cases, stage)
                       : pencil_dim<2, double>(L, U0, Uout, R, nbr26, cases, stage);
    case 3: return f32 ? pencil_dim<3, float>(L, U0, Uout, R, nbr26, cases, stage)
                       : pencil_dim<3, double>(L, U0, Uout, R, nbr26, cases, stage);
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
