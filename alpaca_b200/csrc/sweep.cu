// The last direction's faces fused with the stage update: default schemes.
#include "face_launch.cuh"
#include "sweep.cuh"

namespace alp {
namespace {

template <int DIM, int SCHEME, typename T>
__global__ void __launch_bounds__(32 * kSweepWarps, FaceOccupancy<DIM, SCHEME, T>::sweep_ctas * 4 / kSweepWarps)
sweep_update_kernel(double const *Uin, double const *U0, double *Uout,
                    int const *__restrict__ work, BlockMeta const *__restrict__ meta,
                    int const *__restrict__ nbr26, CaseState const *__restrict__ cases,
                    double const *__restrict__ F, long long stride, long long dstride, int stage,
                    int rows, int nunits) {
  __shared__ double high[kSweepWarps][DIM + 2][32];
  sweep_update<DIM, SCHEME, T, DefaultPolicy, 6>(Uin, U0, Uout, work, meta, nbr26, cases, F, stride,
                                                 dstride, stage, rows, nunits, DefaultPolicy(),
                                                 nullptr, high);
}

template <int DIM, typename T>
cudaError_t sweep_t(Launch const &L, double const *U0, double *Uout, double const *F,
                    long long stride, long long dstride, int const *nbr26, CaseState const *cases,
                    int stage, int rows) {
  constexpr int LINES = DIM == 3 ? IC * IC : IC;
  if (rows > LINES) rows = LINES;
  long long const units = (long long)L.nwork * (LINES / rows);
  if (units > 0x7fffffffLL) return cudaErrorInvalidValue;
  int const n = (int)units, grid = (n + kSweepWarps - 1) / kSweepWarps, th = 32 * kSweepWarps;
  if (!L.opt.is_default())
    return with_stencil(L, [&](auto k) {
      return decltype(k)::sweep(L, grid, th, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows,
                                n);
    });
  switch (L.scheme) {
    case FV_CHAR:
      sweep_update_kernel<DIM, FV_CHAR, T><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, n);
      break;
    case FV_PRIM:
      sweep_update_kernel<DIM, FV_PRIM, T><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, n);
      break;
    case FS_ROE:
      sweep_update_kernel<DIM, FS_ROE, T><<<grid, th, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, nbr26, cases, F, stride, dstride, stage, rows, n);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
}  // namespace

// Lines per warp: the longest sweep of 32, 16 or 8 that leaves three times as
// many warps as fit on the chip (148 SMs of a B200, 16 warps of FV char on each).
// Short sweeps repeat the pass of the lines' last faces more often (rows / 2 + 1
// passes for rows / 2 + rows / 32 of work), long ones end in a nearly empty last
// wave: 512 blocks 1.174 ms per step at 16 lines, 8: 1.196, 32: 1.222; 2D 2025 blocks
// 0.235 at 8, 16: 0.241, 4: 0.247.
int sweep_rows(int dim, int nwork) {
  int const lines = dim == 3 ? IC * IC : IC;
  int rows = dim == 3 ? 32 : 16;
  while (rows > 8 && (long long)nwork * (lines / rows) < 3LL * 148 * 16) rows /= 2;
  return rows;
}

// Below these counts the sweeps leave the chip idle (a warp makes five passes
// one after the other where the face launch has five warps). One line for all
// schemes, a little above where most cross. Step in us, face launch + update against
// sweep:
//   3D               100          112          125          144          512 blocks
//   FV char       265 / 264    301 / 293    335 / 316    380 / 357   1352 / 1218
//   FV prim       244 / 255    278 / 278    308 / 302    346 / 334   1230 / 1129
//   FS Roe        296 / 300    339 / 338    373 / 362    421 / 407   1466 / 1354
//   FV char FP32  240 / 252    275 / 275    305 / 297    344 / 333   1210 / 1070
//   FS Roe FP32   283 / 271    321 / 299    356 / 323    403 / 363   1391 / 1218
//   WENO5-Z       305 / 313    350 / 357    389 / 384    447 / 429   1585 / 1413
//   WENO7         554 / 588    623 / 660    693 / 710    787 / 802   2725 / 2614
//   2D              1024         1190         1225         1600        4096 blocks
//   FV char       127 / 129    146 / 149    154 / 155    202 / 193    547 / 436
//   FV prim       123 / 119    140 / 135    145 / 139    195 / 178    529 / 404
//   FS Roe        137 / 145    158 / 164    165 / 170    224 / 209    608 / 502
//   FV char FP32  121 / 113    139 / 129    147 / 136    195 / 178    533 / 405
//   WENO5-Z       164 / 158    188 / 177    198 / 184    265 / 229    729 / 569
//   WENO7         275 / 260    321 / 316    334 / 322    444 / 402   1207 / 1007
// WENO7 crosses near 200 3D blocks and FS Roe near 1300 2D blocks: 2-3 % lost there.
bool sweep_pays(int dim, int nwork) { return dim > 1 && nwork >= (dim == 3 ? 128 : 1200); }

cudaError_t launch_sweep_update(Launch const &L, double const *U0, double *Uout, double const *F,
                                long long stride, long long dstride, int const *nbr26,
                                CaseState const *cases, int stage) {
  if (L.nwork <= 0) return cudaSuccess;
  if (!L.work || !L.meta || !nbr26 || !cases || stage < 0 || stage > 4) return cudaErrorInvalidValue;
  if (!L.opt.is_default() && L.precision != FP64) return cudaErrorInvalidValue;
  bool const f32 = L.precision == FP32_FLUX;
  int const rows = sweep_rows(L.dim, L.nwork);
  switch (L.dim) {
    case 2: return f32 ? sweep_t<2, float>(L, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows)
                       : sweep_t<2, double>(L, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows);
    case 3: return f32 ? sweep_t<3, float>(L, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows)
                       : sweep_t<3, double>(L, U0, Uout, F, stride, dstride, nbr26, cases, stage, rows);
  }
  return cudaErrorInvalidValue;
}

}  // namespace alp
