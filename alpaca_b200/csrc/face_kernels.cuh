// Device code shared by the kernels that compute face fluxes: the face
// numbering, the stencil loads and one face's flux.
#pragma once

#include "face.cuh"
#include "kernels.cuh"
#include "rotate.cuh"
#include "step_common.cuh"

namespace alp {
namespace {

__device__ __forceinline__ int slot_of(int const *work, int item) {
  return work ? work[item] : item;
}

template <int DIM, int DIR> struct FaceMap {
  static constexpr int O1 = DIR == 0 ? 1 : 0;
  static constexpr int O2 = DIR == 2 ? 1 : 2;
  static constexpr int E1 = Geo<DIM>::ic(O1);
  static constexpr int E2 = Geo<DIM>::ic(O2);
  static constexpr int COUNT = (IC + 1) * E1 * E2;
  // Thread t -> face (a along DIR, p1, p2 across). Consecutive threads walk the
  // fastest-varying stored dimension so that stencil loads coalesce.
  __device__ static void decode(int t, int &a, int &p1, int &p2) {
    if constexpr (DIR == DIM - 1) {
      a = t % (IC + 1);
      int const r = t / (IC + 1);
      p1 = r / E2;
      p2 = r % E2;
    } else {
      a = t / (E1 * E2);
      p1 = (t / E2) % E1;
      p2 = t % E2;
    }
  }
};

// Minimum resident 128-thread CTAs per SM of the face kernels, which caps
// their registers (168 / 128 / 96 at 3 / 4 / 5). Measured on the FP64 128^3
// step, ms: FV char 4 CTAs 1.327 vs 3: 1.519, 5 (168 B of spills): 1.319; FV
// prim 5: 1.174 vs 4: 1.267, 6: 1.178; flux splitting 4 (52 B of spills):
// 1.425 vs 3: 1.521, 2: 1.907. In 2D FV char fits 5 without spills: 2025
// blocks 0.262 against 0.289 at 4. The sweeps (sweep.cuh) hold the stage
// update's state as well: flux splitting runs them at 3. FP32-flux
// instantiations hold fewer live doubles: FS 4 (2.05 ms vs 3: 2.23, when
// measured; 1D 6, 20,000 blocks 0.211 vs 4: 0.266, 600: 26.8 us vs 30.9), FV char 5
// (1.56 vs 4: 1.64), FV prim 5 (1.455 vs 6: 1.48).
template <int DIM, int SCHEME, typename T = double> struct FaceOccupancy {
  static constexpr bool f32 = sizeof(T) == 4;
  static constexpr int min_ctas = SCHEME == FV_CHAR ? (f32 || DIM == 2 ? 5 : 4)
                                  : SCHEME == FV_PRIM ? 5
                                                      : (f32 && DIM == 1 ? 6 : 4);
  static constexpr int sweep_ctas = SCHEME == FS_ROE && !f32 ? 3 : min_ctas;
};

// Stores one face's fluxes in the reference flux-array layout: = (zero for a
// skipped face) or, for the drop-in contract, += (skipped faces untouched).
template <int DIM, int DIR, bool ACCUM>
__device__ __forceinline__ void write_flux(double *__restrict__ F, int item, long long stride,
                                           int a, int p1, int p2, bool valid,
                                           double const (&flux)[DIM + 2]) {
  using G = Geo<DIM>;
  using M = FaceMap<DIM, DIR>;
  int fi[3];
  fi[DIR] = a;
  fi[M::O1] = p1 + 1;
  fi[M::O2] = p2 + 1;
  double *fo = F + (long long)item * stride + G::face(fi[0], fi[1], fi[2]);
#pragma unroll
  for (int f = 0; f < DIM + 2; ++f) {
    double const v = valid ? flux[f] : 0.0;
    if (ACCUM) {
      if (valid) fo[f * G::FACES] += v;
    } else {
      fo[f * G::FACES] = v;
    }
  }
}

// Stencil of the face a (between cells a-1 and a along DIR) at transverse
// position (p1, p2): cells a-3 .. a+2 in interior numbering, all fields.
// GATHER: cells outside the interior along DIR come from the neighbour blocks'
// interiors (nbr26; zero gradient at domain faces) instead of the block's own
// halo cells, so no halo copy is needed between stages.
template <int DIM, int DIR, int GATHER>
__device__ __forceinline__ double const *stencil_cell(double const *__restrict__ U,
                                                      double const *blk, int c, int cell0,
                                                      int nlo, int nhi) {
  using G = Geo<DIM>;
  constexpr int step = DIR == 0 ? G::TCY * G::TCZ : (DIR == 1 ? G::TCZ : 1);
  // cell0: offset of (transverse position, DIR index 0) in the block
  if (GATHER && c < HS)
    return nlo >= 0 ? U + (size_t)nlo * G::BLOCK_DOUBLES + cell0 + (c + IC) * step
                    : blk + cell0 + HS * step;
  if (GATHER && c >= HS + IC)
    return nhi >= 0 ? U + (size_t)nhi * G::BLOCK_DOUBLES + cell0 + (c - IC) * step
                    : blk + cell0 + (HS + IC - 1) * step;
  return blk + cell0 + c * step;
}

template <int DIM, int DIR>
__device__ __forceinline__ int line_origin(int p1, int p2) {
  using G = Geo<DIM>;
  using M = FaceMap<DIM, DIR>;
  int c[3];
  c[DIR] = 0;
  c[M::O1] = G::fic(M::O1) + p1;
  c[M::O2] = G::fic(M::O2) + p2;
  return G::cell(c[0], c[1], c[2]);
}

// GATHER of the loads below: 0 the block's own halo cells, 1 the neighbours'
// interiors, 2 the same through L2 (cells written earlier in the same launch).
template <int DIM, int GATHER>
__device__ __forceinline__ void load_cell(double const *src, double (&dst)[DIM + 2]) {
#pragma unroll
  for (int f = 0; f < DIM + 2; ++f)
    dst[f] = GATHER == 2 ? __ldcg(src + f * Geo<DIM>::CELLS) : __ldg(src + f * Geo<DIM>::CELLS);
}

// Cell c of a stencil line (stencil_cell), with symmetry walls: a neighbour
// entry of -2 across the block face mirrors the line about the wall and negates
// the momentum normal to it (symmetry_boundary_condition.h:60-113, 148-217;
// boundary_constants.h:35-46, 167-209); -1 is zero gradient.
template <int DIM, int DIR, int GATHER>
__device__ __forceinline__ void stencil_load(double const *__restrict__ U, double const *blk,
                                             int c, int cell0, int nlo, int nhi,
                                             double (&dst)[DIM + 2]) {
  constexpr int step = DIR == 0 ? Geo<DIM>::TCY * Geo<DIM>::TCZ : (DIR == 1 ? Geo<DIM>::TCZ : 1);
  if (GATHER && ((c < HS && nlo == -2) || (c >= HS + IC && nhi == -2))) {
    int const m = c < HS ? 2 * HS - 1 - c : 2 * (HS + IC) - 1 - c;
    load_cell<DIM, GATHER>(blk + cell0 + m * step, dst);
    dst[MOMX + DIR] = -1.0 * dst[MOMX + DIR];
    return;
  }
  load_cell<DIM, GATHER>(stencil_cell<DIM, DIR, GATHER>(U, blk, c, cell0, nlo, nhi), dst);
}

// Flux of the face (a; p1, p2) of direction DIR of the block in `slot`; false
// for a face the reference skips.
template <int DIM, int DIR, int SCHEME, typename T, int GATHER, typename P = DefaultPolicy,
          int W = 6>
__device__ __forceinline__ bool face_value(double const *__restrict__ U,
                                           int const *__restrict__ nbr26, int slot, int a, int p1,
                                           int p2, BlockMeta const &bm, double (&fd)[DIM + 2],
                                           P const &pol = P()) {
  using G = Geo<DIM>;
  constexpr int NE = G::NE;
  Eos const eos{bm.gamma, bm.B, bm.safe};
  double const *blk = U + (size_t)slot * G::BLOCK_DOUBLES;
  int const cell0 = line_origin<DIM, DIR>(p1, p2);
  // low / high neighbour along DIR (26-table slots of W,E / S,N / B,T)
  constexpr int lo_slot = DIR == 0 ? 4 : (DIR == 1 ? 10 : 12);
  constexpr int hi_slot = DIR == 0 ? 21 : (DIR == 1 ? 15 : 13);
  int const nlo = GATHER && a < W / 2 ? __ldg(nbr26 + (size_t)slot * 26 + lo_slot) : 0;
  int const nhi = GATHER && a > IC - W / 2 ? __ldg(nbr26 + (size_t)slot * 26 + hi_slot) : 0;
  double cons[W][NE];
#pragma unroll
  for (int m = 0; m < W; ++m)
    stencil_load<DIM, DIR, GATHER>(U, blk, HS + a - W / 2 + m, cell0, nlo, nhi, cons[m]);
  bool valid;
  if constexpr (DIM == 3 && DIR != 0) {
    // 3D y and z faces: the x-face computation of the rotated stencil
    // (canon_field), the same code as the fused tile kernel
    double rc[W][NE];
#pragma unroll
    for (int m = 0; m < W; ++m)
#pragma unroll
      for (int c = 0; c < NE; ++c) rc[m][c] = cons[m][canon_field(DIR, c)];
    double rf[NE];
    valid = face_compute<3, 0, SCHEME, T, P, W>(eos, bm.B, rc, rf, pol);
#pragma unroll
    for (int c = 0; c < NE; ++c) fd[canon_field(DIR, c)] = rf[c];
  } else {
    valid = face_compute<DIM, DIR, SCHEME, T, P, W>(eos, bm.B, cons, fd, pol);
  }
  return valid;
}

// Flux of the face with thread index t of direction DIR of the block in `slot`.
template <int DIM, int DIR, int SCHEME, typename T, bool ACCUM, int GATHER,
          typename P = DefaultPolicy, int W = 6>
__device__ __forceinline__ void face_flux(double const *__restrict__ U,
                                          int const *__restrict__ nbr26, int slot, int item,
                                          int t, BlockMeta const &bm, double *__restrict__ F,
                                          long long stride, P const &pol = P()) {
  int a, p1, p2;
  FaceMap<DIM, DIR>::decode(t, a, p1, p2);
  double fd[DIM + 2];
  bool const valid =
      face_value<DIM, DIR, SCHEME, T, GATHER, P, W>(U, nbr26, slot, a, p1, p2, bm, fd, pol);
  write_flux<DIM, DIR, ACCUM>(F, item, stride, a, p1, p2, valid, fd);
}

}  // namespace
}  // namespace alp
