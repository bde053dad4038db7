// The last direction's faces fused with the stage update, shared by the kernels
// of the compiled default (sweep.cu) and of the run-time selected schemes
// (ext_kernels.cuh).
#pragma once

#include "face_kernels.cuh"

namespace alp {
namespace {

// The policy of one block: for the run-time selected schemes with the
// GlobalLaxFriedrichs wave speeds of its case.
__device__ __forceinline__ DefaultPolicy block_policy(DefaultPolicy const &pol, BlockMeta const &,
                                                      unsigned long long const *) {
  return pol;
}
template <int ST>
__device__ __forceinline__ ExtPolicy<ST> block_policy(ExtPolicy<ST> pol, BlockMeta const &bm,
                                                      unsigned long long const *glf) {
  if (glf && pol.o.splitting == FSP_GLF)
    for (int k = 0; k < 3; ++k) pol.glf[k] = __longlong_as_double(glf[4 * bm.case_id + k]);
  return pol;
}

// The faces of the last direction (z in 3D, y in 2D) and the stage update in one
// launch: a warp sweeps `rows` lines of 16 cells of one work item, two lines at a
// time, lane = cell. A lane computes the flux of its cell's low face; the high
// face's flux is the next lane's, and the faces beyond the last cells of all the
// warp's lines are computed first, one lane per line, and kept in shared memory
// (rows / 2 + 1 passes; none is wasted at 32 rows). With both fluxes of the last
// direction in registers the lane reads the other directions' fluxes and applies
// the stage to its cell, so the last direction's flux array is neither written
// nor read, and the update's loads run beside the other warps' face arithmetic.
// Uin, U0, Uout, F, stage, cases as in stage_update_kernel.
template <int DIM, int SCHEME, typename T, typename P, int W>
__device__ __forceinline__ void sweep_update(double const *Uin, double const *U0, double *Uout,
                                             int const *__restrict__ work,
                                             BlockMeta const *__restrict__ meta,
                                             int const *__restrict__ nbr26,
                                             CaseState const *__restrict__ cases,
                                             double const *__restrict__ F, long long stride,
                                             long long dstride, int stage, int rows, int nunits, P const &pol0,
                                             unsigned long long const *glf,
                                             double (*high)[DIM + 2][32]) {
  using G = Geo<DIM>;
  constexpr int DIR = DIM - 1, NE = G::NE;
  constexpr int LINES = DIM == 3 ? IC * IC : IC;
  int const wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int const unit = blockIdx.x * (blockDim.x >> 5) + wid;
  if (unit >= nunits) return;
  int const per = LINES / rows;
  int const item = unit / per, r0 = (unit - item * per) * rows;
  int const slot = work[item];
  BlockMeta const bm = meta[slot];
  double const dt = cases[bm.case_id].dt;
  if (!(dt > 0.0)) return;
  P const pol = block_policy(pol0, bm, glf);
  double const *Fb = F + (long long)item * stride;
  double const ocs = inv(bm.cell_size);
  RkStage const rk = rk_stage(stage, dt);
#pragma unroll 1
  for (int q = -1; q < rows / 2; ++q) {
    bool const last = q < 0;  // the faces beyond the last cells
    int const line = r0 + (last ? (lane < rows ? lane : 0) : 2 * q + (lane >> 4));
    int const a = last ? IC : lane & 15;
    int const p1 = DIM == 3 ? line >> 4 : line, p2 = DIM == 3 ? line & 15 : 0;
    double f[NE];
    bool const valid = face_value<DIM, DIR, SCHEME, T, true, P, W>(Uin, nbr26, slot, a, p1, p2, bm,
                                                                   f, pol);
#pragma unroll
    for (int n = 0; n < NE; ++n)
      if (!valid) f[n] = 0.0;
    if (last) {
#pragma unroll
      for (int n = 0; n < NE; ++n) high[wid][n][lane] = f[n];
      __syncwarp();
      continue;
    }
    int const i = p1, j = DIM == 3 ? p2 : a, k = DIM == 3 ? a : 0;
    size_t const x = (size_t)slot * G::BLOCK_DOUBLES +
                     G::cell(i + G::fic(0), j + G::fic(1), k + G::fic(2));
    // every load of the cell before its first store (Uout may alias U0, so the
    // compiler would keep the fields' loads behind the previous field's store)
    double u[NE], u0[NE], xl[NE], xh[NE], yl[NE], yh[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      double const *fx = Fb + n * G::FACES;
      xl[n] = fx[G::face(i, j + 1, k + 1)];
      xh[n] = fx[G::face(i + 1, j + 1, k + 1)];
      if constexpr (DIM == 3) {
        yl[n] = fx[dstride + G::face(i + 1, j, k + 1)];
        yh[n] = fx[dstride + G::face(i + 1, j + 1, k + 1)];
      }
      u[n] = Uin[x + (size_t)n * G::CELLS];
      u0[n] = rk.first ? 0.0 : U0[x + (size_t)n * G::CELLS];
    }
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      double hi = __shfl_down_sync(0xffffffffu, f[n], 1);
      if (a == IC - 1) hi = high[wid][n][2 * q + (lane >> 4)];
      double rhs;
      if constexpr (DIM == 3) rhs = flux_divergence<3>(xl[n], xh[n], yl[n], yh[n], f[n], hi, ocs);
      else rhs = flux_divergence<DIM>(xl[n], xh[n], f[n], hi, 0.0, 0.0, ocs);
      Uout[x + (size_t)n * G::CELLS] = rk_apply(rk, u[n], u0[n], 0.0 + rhs);
    }
  }
}

constexpr int kSweepWarps = 2;  // warps (independent of one another) per CTA

}  // namespace
}  // namespace alp
