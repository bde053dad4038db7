// Per-face flux of the block right-hand side, shared by the face-flux kernels
// (face_flux.cu, sweep.cuh, small.cu, ext_kernels.cuh, pencil.cu) and the fused
// tile-stage kernel (tile_step.cuh): all evaluate every face through face_compute,
// so they produce the same bits.
#pragma once

#include <cfloat>

#include "kernels.cuh"

// The default policy's Riemann solver is known at compile time, which leaves the
// code for the others unreachable in prim_flux's default instantiations.
#pragma nv_diag_suppress 128
#include "numerics.cuh"
#include "schemes_ext.cuh"

namespace alp {

// Structural nonzeros of the left eigenvector matrix row n, column l
// (eigendecomposition.h:316-359).
template <int DIM, int DIR>
__host__ __device__ constexpr bool left_nonzero(int n, int l) {
  // the rows of the two acoustic waves and of the principal-momentum wave are full
  if (n == 0 || n == DIM + 1 || n == DIM) return true;
  // minor-momentum waves: mass and their own momentum only
  return l == MASS || l == MOMX + (n == 1 ? Minor<DIR>::m1 : Minor<DIR>::m2);
}

// Fast-build FP64 forms of the per-state quantities, with the kinetic energy
// as a plain chain of products.

// A reconstructed state's 1/rho, principal velocity and pressure.
struct ReconState {
  double one, v, p;
};
template <int DIM, int DIR>
__device__ __forceinline__ ReconState recon_state(Eos const &e, double const (&c)[DIM + 2]) {
  double q = c[MOMX] * c[MOMX];
  if constexpr (DIM > 1) q = fma(c[MOMX + 1], c[MOMX + 1], q);
  if constexpr (DIM > 2) q = fma(c[MOMX + 2], c[MOMX + 2], q);
  ReconState s;
  s.one = inv(c[MASS]);
  s.v = c[MOMX + DIR] * s.one;
  double const one = e.safe && !(c[MASS] > DBL_EPSILON) ? 1.0 / DBL_EPSILON : s.one;
  s.p = fma(e.gamma - 1.0, fma(-0.5 * one, q, c[ENERGY]), -(e.gamma * e.B));
  if (e.safe) s.p = dmax(s.p, -e.B + DBL_EPSILON);
  return s;
}

// Physical flux of a cell along DIR.
template <int DIM, int DIR>
__device__ __forceinline__ void phys_flux(Eos const &e, double const (&c)[DIM + 2],
                                          double (&f)[DIM + 2]) {
  ReconState const s = recon_state<DIM, DIR>(e, c);
  f[MASS] = c[MOMX + DIR];
  f[ENERGY] = (c[ENERGY] + s.p) * s.v;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    f[MOMX + d] = d == DIR ? fma(c[MOMX + d], s.v, s.p) : c[MOMX + d] * s.v;
}

// The forms of a face's flux that face_compute chooses from; arguments and result
// as there.

// Characteristic finite-volume reconstruction or Roe flux splitting in the fast
// build's FP64, six cells.
template <int DIM, int DIR, int SCHEME, typename P>
__device__ __forceinline__ bool frame_flux(Eos const &eos, double B,
                                           double const (&cons)[6][DIM + 2],
                                           double (&fd)[DIM + 2], P const &pol) {
  constexpr int NE = DIM + 2, C = 2;
  bool valid = true;
  // the factored characteristic frame on the five differences of the six
  // cells (each side's reconstruction is its own cell plus an increment)
  auto const ct = char_cell<DIM, DIR>(eos, cons[C]);
  auto const cn = char_cell<DIM, DIR>(eos, cons[C + 1]);
  if (!(cons[C][MASS] > 0.0) || !(cons[C + 1][MASS] > 0.0)) valid = false;
  auto const r = char_frame<DIM, DIR>(eos, ct, cn, cons[C][MASS], cons[C + 1][MASS]);
  if constexpr (SCHEME == FV_CHAR) {
    double G[NE][5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double x[NE], ch[NE];
#pragma unroll
      for (int l = 0; l < NE; ++l) x[l] = cons[m + 1][l] - cons[m][l];
      char_project<DIM, DIR>(r, x, ch);
#pragma unroll
      for (int n = 0; n < NE; ++n) G[n][m] = ch[n];
    }
    double il[NE], ir[NE];
    double const minor = dmax(r.rho2, kMinorRho2);
#pragma unroll
    for (int n = 0; n < NE; ++n)
      pol.increments(G[n], char_scale<DIM>(minor, n), il[n], ir[n], minor_wave<DIM>(n));
    double cm[NE], cp[NE];
    char_restore<DIM, DIR>(r, cons[C], il, 1.0, cm);
    char_restore<DIM, DIR>(r, cons[C + 1], ir, -1.0, cp);
    if (!(cm[MASS] > DBL_EPSILON) || !(cp[MASS] > DBL_EPSILON)) valid = false;
    auto const sm = recon_state<DIM, DIR>(eos, cm);
    auto const sp = recon_state<DIM, DIR>(eos, cp);
    if (!(sm.p > -B) || !(sp.p > -B)) valid = false;
    pol.template riemann<DIM, DIR, double>(eos, cm, cp, sm.p, sp.p, sm.v, sp.v, sm.one, sp.one,
                                           fd);
  } else {
    // Roe flux-vector splitting: the split fluxes f +/- alpha u of each
    // wave from the projected differences of f and u. The mean of the two
    // reconstructions is (f_i + f_i+1) / 2 plus R times half of
    // (left increment - right increment - alpha L (u_i+1 - u_i)).
    double al[3];
    pol.frame_eigenvalues(eos, r, ct, cn, cons[C][MASS], cons[C + 1][MASS], al);
    double A[NE][5], N[NE][5], w[NE];
    double fa[NE], fb[NE], fi[NE];
    phys_flux<DIM, DIR>(eos, cons[0], fa);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double x[NE], y[NE], cu[NE], cf[NE];
      if (m == 2) {
#pragma unroll
        for (int l = 0; l < NE; ++l) fi[l] = fa[l];
      }
      phys_flux<DIM, DIR>(eos, cons[m + 1], fb);
#pragma unroll
      for (int l = 0; l < NE; ++l) {
        x[l] = cons[m + 1][l] - cons[m][l];
        y[l] = fb[l] - fa[l];
      }
      if (m == 2) {
#pragma unroll
        for (int l = 0; l < NE; ++l) fi[l] = 0.5 * (fi[l] + fb[l]);
      }
      char_project<DIM, DIR>(r, x, cu);
      char_project<DIM, DIR>(r, y, cf);
#pragma unroll
      for (int n = 0; n < NE; ++n) {
        double const a = n == 0 ? al[0] : (n == NE - 1 ? al[2] : al[1]);
        if (m < 4) A[n][m] = fma(a, cu[n], cf[n]);
        if (m > 0) N[n][m] = fma(-a, cu[n], cf[n]);
        if (m == 2) w[n] = a * cu[n];
      }
#pragma unroll
      for (int l = 0; l < NE; ++l) fa[l] = fb[l];
    }
    MinorUnits const mu = minor_units(r.rho2);
    if (DIM > 1 && __builtin_expect(mu.tiny, 0)) {
#pragma unroll
      for (int n = 1; n < DIM; ++n) {
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          if (m < 4) A[n][m] *= mu.unit;
          if (m > 0) N[n][m] *= mu.unit;
        }
        w[n] *= mu.unit;
      }
    }
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      double l, q;
      A[n][4] = 0.0;
      N[n][0] = 0.0;
      pol.increments_two(A[n], N[n], char_scale<DIM>(mu.scale, n), l, q, minor_wave<DIM>(n));
      w[n] = 0.5 * ((l - q) - w[n]);
    }
    if (DIM > 1 && __builtin_expect(mu.tiny, 0)) {
#pragma unroll
      for (int n = 1; n < DIM; ++n) w[n] *= mu.back;
    }
    char_restore<DIM, DIR>(r, fi, w, 1.0, fd);
  }
  return valid;
}

// The same in the FP32-flux form: projection, reconstruction and wave speeds in
// float on variations formed in double, the cells' states and fluxes added in
// double.
template <int DIM, int DIR, int SCHEME, typename P>
__device__ __forceinline__ bool packed_flux(Eos const &eos, double B,
                                            double const (&cons)[6][DIM + 2],
                                            double (&fd)[DIM + 2], P const &pol) {
  using T = float;
  constexpr int NE = DIM + 2, C = 2;
  bool valid = true;
  auto const pt = cell_prims<DIM, DIR>(eos, cons[C]);
  auto const pn = cell_prims<DIM, DIR>(eos, cons[C + 1]);
  if (!(pt.rho > 0.0) || !(pn.rho > 0.0)) valid = false;
  Roe<T> const r = roe_average<DIM, DIR, T>(eos, pt, pn);
  if constexpr (SCHEME == FV_CHAR) {
    // WENO5 is translation invariant and R L = I: the variations alone are
    // projected and reconstructed, the face's left cell is added back
    T dm[NE], dp[NE];
    // the first differences of the six cells, projected and reconstructed
    // with both sides of the face as the lanes of packed f32x2 arithmetic:
    // differences 0 and 4, 1 and 3 as pairs, 2 alone
    float2 x0[NE], x1[NE], chp[NE], out[NE];
    float x2[NE];
#pragma unroll
    for (int l = 0; l < NE; ++l) {
      x0[l] = make_float2(float(cons[1][l] - cons[0][l]), float(cons[5][l] - cons[4][l]));
      x1[l] = make_float2(float(cons[2][l] - cons[1][l]), float(cons[4][l] - cons[3][l]));
      x2[l] = float(cons[3][l] - cons[2][l]);
    }
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T L[NE];
      left_row<DIM, DIR, T>(n, r, L);
      float2 g0 = make_float2(0.0f, 0.0f), g1 = g0;
      float g2 = 0.0f;
      bool first = true;
#pragma unroll
      for (int q = 0; q < NE; ++q) {
        int const l = sum_seq<DIM, DIR>(q);
        if (!left_nonzero<DIM, DIR>(n, l)) continue;
        float2 const Ld = dup2(L[l]);
        g0 = first ? mul2(Ld, x0[l]) : fma2(Ld, x0[l], g0);
        g1 = first ? mul2(Ld, x1[l]) : fma2(Ld, x1[l], g1);
        g2 = first ? L[l] * x2[l] : fmaf(L[l], x2[l], g2);
        first = false;
      }
      float2 const i = weno5_packed(g0, g1, dup2(g2), make_float2(g1.y, g1.x), 1.0e-6f);
      chp[n] = make_float2(i.x, g2 - i.y);  // the right cell is g2 beyond the left one
    }
    to_physical_packed<DIM, DIR>(r, chp, out);
#pragma unroll
    for (int f = 0; f < NE; ++f) {
      dm[f] = out[f].x;
      dp[f] = out[f].y;
    }
    double cm[NE], cp[NE];
#pragma unroll
    for (int f = 0; f < NE; ++f) {
      cm[f] = cons[C][f] + double(dm[f]);
      cp[f] = cons[C][f] + double(dp[f]);
    }
    if (!(cm[MASS] > DBL_EPSILON) || !(cp[MASS] > DBL_EPSILON)) valid = false;
    auto const sm = recon_state<DIM, DIR>(eos, cm);
    auto const sp = recon_state<DIM, DIR>(eos, cp);
    if (!(sm.p > -B) || !(sp.p > -B)) valid = false;
    hllc_flux<DIM, DIR>(hllc_upwind_mixed(eos, cm[MASS], cp[MASS], sm.p, sp.p, sm.v, sp.v,
                                          sm.one, sp.one),
                        cm, cp, fd);
  } else {
    // the variations of the state and the physical flux projected
    // as the two lanes of packed f32x2 arithmetic, the split fluxes'
    // differences reconstructed with both sides as lanes; the left cell's
    // flux (its characteristic values restored by R) added back in double
    float2 x[5][NE];
    double f0[NE], fa[NE], fb[NE];
    phys_flux<DIM, DIR>(eos, cons[0], fa);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      phys_flux<DIM, DIR>(eos, cons[m + 1], fb);
#pragma unroll
      for (int l = 0; l < NE; ++l) {
        x[m][l] = make_float2(float(cons[m + 1][l] - cons[m][l]), float(fb[l] - fa[l]));
        fa[l] = fb[l];
        if (m == C - 1) f0[l] = fb[l];
      }
    }
    T ch[NE], flux[NE], ev_nl0, ev_lin, ev_nl1;
    pol.template fs_eigenvalues<DIM, DIR, T>(eos, r, pt, pn, ev_nl0, ev_lin, ev_nl1);
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T L[NE];
      left_row<DIM, DIR, T>(n, r, L);
      float const alpha = n == 0 ? ev_nl0 : (n == NE - 1 ? ev_nl1 : ev_lin);
      float A[5], N[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float2 acc = make_float2(0.0f, 0.0f);
        bool first = true;
#pragma unroll
        for (int q = 0; q < NE; ++q) {
          int const l = sum_seq<DIM, DIR>(q);
          if (!left_nonzero<DIM, DIR>(n, l)) continue;
          acc = first ? mul2(x[m][l], dup2(L[l])) : fma2(x[m][l], dup2(L[l]), acc);
          first = false;
        }
        A[m] = fmaf(alpha, acc.x, acc.y);
        N[m] = fmaf(-alpha, acc.x, acc.y);
      }
      float2 const i = weno5_packed(make_float2(A[0], N[4]), make_float2(A[1], N[3]),
                                    make_float2(A[2], N[2]), make_float2(A[3], N[1]), 1.0e-6f);
      ch[n] = 0.5f * (i.x + (N[2] - i.y));
    }
    to_physical<DIM, DIR, T>(r, ch, flux);
#pragma unroll
    for (int f = 0; f < NE; ++f) fd[f] = f0[f] + double(flux[f]);
  }
  return valid;
}

// Characteristic finite-volume reconstruction or flux splitting in the reference's
// order of operations: the strict build, and the fast build's eight-cell stencils
// (FP64).
template <int DIM, int DIR, int SCHEME, typename T, typename P, int W>
__device__ __forceinline__ bool ordered_flux(Eos const &eos, double B,
                                             double const (&cons)[W][DIM + 2],
                                             double (&fd)[DIM + 2], P const &pol) {
  constexpr int NE = DIM + 2, C = W / 2 - 1, mP = MOMX + DIR;
  bool valid = true;
  auto const pt = cell_prims<DIM, DIR>(eos, cons[C]);
  auto const pn = cell_prims<DIM, DIR>(eos, cons[C + 1]);
  if (!(pt.rho > 0.0) || !(pn.rho > 0.0)) valid = false;
  Roe<T> const r = roe_average<DIM, DIR, T>(eos, pt, pn);
  T ch[2][NE], flux[NE];
  if constexpr (SCHEME == FV_CHAR && sizeof(T) == 4) {
    // FP32 form: characteristic projection and WENO5 of the state's variation
    // (WENO5 is translation invariant and R L = I), the face's left cell added
    // back in double. The variation is formed in double and converted once.
    T dm[NE], dp[NE];
    float du[W][NE];
#pragma unroll
    for (int m = 0; m < W; ++m)
#pragma unroll
      for (int l = 0; l < NE; ++l) du[m][l] = m == C ? 0.0f : float(cons[m][l] - cons[C][l]);
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T L[NE];
      left_row<DIM, DIR, T>(n, r, L);
      T uc[W];
#pragma unroll
      for (int m = 0; m < W; ++m) {
        T s = T(0);
#pragma unroll
        for (int q = 0; q < NE; ++q) {
          int const l = sum_seq<DIM, DIR>(q);
          if (!left_nonzero<DIM, DIR>(n, l)) continue;
          s = fmaf(L[l], du[m][l], s);
        }
        uc[m] = s;
      }
      pol.pair(uc, ch[0][n], ch[1][n]);
    }
    to_physical<DIM, DIR, T>(r, ch[0], dm);
    to_physical<DIM, DIR, T>(r, ch[1], dp);
    double cm[NE], cp[NE];
#pragma unroll
    for (int f = 0; f < NE; ++f) {
      cm[f] = cons[C][f] + double(dm[f]);
      cp[f] = cons[C][f] + double(dp[f]);
    }
    if (!(cm[MASS] > DBL_EPSILON) || !(cp[MASS] > DBL_EPSILON)) valid = false;
    double const one_l = inv(cm[MASS]), one_r = inv(cp[MASS]);
    double const pm = eos_pressure<DIM, false>(eos, cm[MASS], cm[MOMX], DIM > 1 ? cm[MOMX + (DIM > 1)] : 0.0,
                                        DIM > 2 ? cm[MOMX + 2 * (DIM > 2)] : 0.0, cm[ENERGY], one_l);
    double const pp = eos_pressure<DIM, false>(eos, cp[MASS], cp[MOMX], DIM > 1 ? cp[MOMX + (DIM > 1)] : 0.0,
                                        DIM > 2 ? cp[MOMX + 2 * (DIM > 2)] : 0.0, cp[ENERGY], one_r);
    if (!(pm > -B) || !(pp > -B)) valid = false;
    hllc_mixed<DIM, DIR>(eos, cm, cp, pm, pp, cm[mP] * one_l, cp[mP] * one_r, one_l, one_r, fd);
    return valid;
  } else if constexpr (SCHEME == FV_CHAR) {
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T L[NE];
      left_row<DIM, DIR, T>(n, r, L);
      T uc[W];
#pragma unroll
      for (int m = 0; m < W; ++m) {
        T s = T(0);
        bool first = true;
#pragma unroll
        for (int q = 0; q < NE; ++q) {
          int const l = sum_seq<DIM, DIR>(q);
          if (!left_nonzero<DIM, DIR>(n, l)) continue;
          T const prod = L[l] * T(cons[m][l]);
          s = first ? prod : s + prod;
          first = false;
        }
        uc[m] = s;
      }
      pol.pair(uc, ch[0][n], ch[1][n]);
    }
    T cm[NE], cp[NE];
    to_physical<DIM, DIR, T>(r, ch[0], cm);
    to_physical<DIM, DIR, T>(r, ch[1], cp);
    if (!(cm[MASS] > eps_of<T>()) || !(cp[MASS] > eps_of<T>())) valid = false;
    // prime states of the reconstructed states (prime_state_handler.h:277-371),
    // pressure recovered in double
    T const one_l = inv(cm[MASS]), one_r = inv(cp[MASS]);
    double const pm = eos_pressure<DIM, false>(eos, double(cm[MASS]), double(cm[MOMX]),
                                        DIM > 1 ? double(cm[MOMX + (DIM > 1)]) : 0.0,
                                        DIM > 2 ? double(cm[MOMX + 2 * (DIM > 2)]) : 0.0,
                                        double(cm[ENERGY]), double(one_l));
    double const pp = eos_pressure<DIM, false>(eos, double(cp[MASS]), double(cp[MOMX]),
                                        DIM > 1 ? double(cp[MOMX + (DIM > 1)]) : 0.0,
                                        DIM > 2 ? double(cp[MOMX + 2 * (DIM > 2)]) : 0.0,
                                        double(cp[ENERGY]), double(one_r));
    if (!(pm > -B) || !(pp > -B)) valid = false;
    T const vl = cm[mP] * one_l;
    T const vr = cp[mP] * one_r;
    pol.template riemann<DIM, DIR, T>(eos, cm, cp, T(pm), T(pp), vl, vr, one_l, one_r, flux);
  } else {
    // Roe flux-vector splitting (flux_splitting_scheme.cpp:42-76, 185-315)
    double advd[W][NE];
#pragma unroll
    for (int m = 0; m < W; ++m) {
      double const one_rho = inv(cons[m][MASS]);
      double const p = eos_pressure<DIM, false>(
          eos, cons[m][MASS], cons[m][MOMX], DIM > 1 ? cons[m][MOMX + (DIM > 1)] : 0.0,
          DIM > 2 ? cons[m][MOMX + 2 * (DIM > 2)] : 0.0, cons[m][ENERGY], one_rho);
      double const vel = cons[m][mP] * one_rho;
      double const rho = cons[m][MASS];
      // the fast build uses rho u = m for the mass and momentum fluxes
      advd[m][MASS] = ALP_FAST ? cons[m][mP] : rho * vel;
      advd[m][ENERGY] = (cons[m][ENERGY] + p) * vel;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        double const vd = cons[m][MOMX + d] * one_rho;
        double v = ALP_FAST ? cons[m][mP] * vd : rho * (vel * vd);
        if (d == DIR) v += p;
        advd[m][MOMX + d] = v;
      }
    }
    T ev_nl0, ev_lin, ev_nl1;
    pol.template fs_eigenvalues<DIM, DIR, T>(eos, r, pt, pn, ev_nl0, ev_lin, ev_nl1);
    // FP32 form: increments against the face's left cell; the characteristic
    // flux of that cell, L f_i, is restored by R as f_i in double
    constexpr bool DELTA = sizeof(T) == 4;
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T L[NE];
      left_row<DIM, DIR, T>(n, r, L);
      T const alpha = n == 0 ? ev_nl0 : (n == NE - 1 ? ev_nl1 : ev_lin);
      T pos[W], neg[W];
#pragma unroll
      for (int m = 0; m < W; ++m) {
        T sp = T(0), sn = T(0);
        bool first = true;
#pragma unroll
        for (int q = 0; q < NE; ++q) {
          int const l = sum_seq<DIM, DIR>(q);
          if (!left_nonzero<DIM, DIR>(n, l)) continue;
          T const uct = (DELTA ? T(cons[m][l] - cons[C][l]) : T(cons[m][l])) * L[l];
          T const act = (DELTA ? T(advd[m][l] - advd[C][l]) : T(advd[m][l])) * L[l];
          if constexpr (ALP_FAST) {
            // project state (into sp) and flux (into sn), split afterwards:
            // L (f +/- alpha u) = L f +/- alpha L u
            sp = first ? uct : sp + uct;
            sn = first ? act : sn + act;
          } else {
            T const tp = act + alpha * uct;
            T const tn = act - alpha * uct;
            sp = first ? tp : sp + tp;
            sn = first ? tn : sn + tn;
          }
          first = false;
        }
        if constexpr (ALP_FAST) {
          pos[m] = sn + alpha * sp;
          neg[m] = sn - alpha * sp;
        } else {
          pos[m] = sp;
          neg[m] = sn;
        }
      }
      T wl, wr;
      pol.two(pos, neg, wl, wr);
      ch[0][n] = T(0.5) * (wl + wr);
    }
    to_physical<DIM, DIR, T>(r, ch[0], flux);
    if constexpr (DELTA) {
#pragma unroll
      for (int f = 0; f < NE; ++f) fd[f] = advd[C][f] + double(flux[f]);
      return valid;
    }
  }
#pragma unroll
  for (int f = 0; f < NE; ++f) fd[f] = double(flux[f]);
  return valid;
}

// Primitive finite-volume reconstruction (primitive_state_reconstruction.h:56-107).
template <int DIM, int DIR, typename T, typename P, int W>
__device__ __forceinline__ bool prim_flux(Eos const &eos, double B,
                                          double const (&cons)[W][DIM + 2],
                                          double (&fd)[DIM + 2], P const &pol) {
  constexpr int NE = DIM + 2, C = W / 2 - 1;
  bool valid = true;
  double prim[W][NE];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    if constexpr (ALP_FAST) {
      // velocities, then the pressure with the kinetic energy u . m / 2
      prim[m][RHO] = cons[m][MASS];
      double const one = inv(cons[m][MASS]);
      double v[DIM], mom[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        mom[d] = cons[m][MOMX + d];
        prim[m][VELX + d] = v[d] = mom[d] * one;
      }
      double um = axis_dot<DIM, DIR>(v, mom);
      if (eos.safe && !(cons[m][MASS] > DBL_EPSILON)) um *= cons[m][MASS] * (1.0 / DBL_EPSILON);
      double p = fma(eos.gamma - 1.0, fma(-0.5, um, cons[m][ENERGY]), -(eos.gamma * eos.B));
      if (eos.safe) p = dmax(p, -eos.B + DBL_EPSILON);
      prim[m][PRES] = p;
    } else {
      prim[m][RHO] = cons[m][MASS];
      double const one_rho = inv(cons[m][MASS]);
#pragma unroll
      for (int d = 0; d < DIM; ++d) prim[m][VELX + d] = cons[m][MOMX + d] * one_rho;
      prim[m][PRES] = eos_pressure<DIM>(
          eos, cons[m][MASS], cons[m][MOMX], DIM > 1 ? cons[m][MOMX + (DIM > 1)] : 0.0,
          DIM > 2 ? cons[m][MOMX + 2 * (DIM > 2)] : 0.0, cons[m][ENERGY], one_rho);
    }
  }
  if constexpr (ALP_FAST && sizeof(T) == 4) {
    // FP32 form: WENO5 of the primes' differences, added to the side's own cell
    double pm[NE], pp[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      float G[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) G[m] = float(prim[m + 1][n] - prim[m][n]);
      float2 const i = weno5_packed(make_float2(G[0], G[4]), make_float2(G[1], G[3]),
                                    dup2(G[2]), make_float2(G[3], G[1]), 1.0e-6f);
      pm[n] = prim[C][n] + double(i.x);
      pp[n] = prim[C + 1][n] - double(i.y);
    }
    if (!(pm[RHO] > DBL_EPSILON) || !(pp[RHO] > DBL_EPSILON)) valid = false;
    if (!(pm[PRES] > -B) || !(pp[PRES] > -B)) valid = false;
    hllc_flux_primes<DIM, DIR>(eos,
                               hllc_upwind_mixed(eos, pm[RHO], pp[RHO], pm[PRES], pp[PRES],
                                                 pm[VELX + DIR], pp[VELX + DIR], inv(pm[RHO]),
                                                 inv(pp[RHO])),
                               pm, pp, fd);
  } else if constexpr (sizeof(T) == 4) {
    // FP32 form: WENO5 of the increments against the left cell's primes
    double pmd[NE], ppd[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      T arr[W];
#pragma unroll
      for (int m = 0; m < W; ++m) arr[m] = T(prim[m][n] - prim[C][n]);
      T wl, wr;
      pol.pair(arr, wl, wr);
      pmd[n] = prim[C][n] + double(wl);
      ppd[n] = prim[C][n] + double(wr);
    }
    double cm[NE], cp[NE];
    cm[MASS] = pmd[RHO];
    cp[MASS] = ppd[RHO];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      cm[MOMX + d] = pmd[VELX + d] * pmd[RHO];
      cp[MOMX + d] = ppd[VELX + d] * ppd[RHO];
    }
    cm[ENERGY] = eos_energy<DIM, double>(eos, pmd[RHO], pmd[VELX], DIM > 1 ? pmd[VELX + (DIM > 1)] : 0.0,
                                         DIM > 2 ? pmd[VELX + 2 * (DIM > 2)] : 0.0, pmd[PRES]);
    cp[ENERGY] = eos_energy<DIM, double>(eos, ppd[RHO], ppd[VELX], DIM > 1 ? ppd[VELX + (DIM > 1)] : 0.0,
                                         DIM > 2 ? ppd[VELX + 2 * (DIM > 2)] : 0.0, ppd[PRES]);
    if (!(cm[MASS] > DBL_EPSILON) || !(cp[MASS] > DBL_EPSILON)) valid = false;
    if (!(pmd[PRES] > -B) || !(ppd[PRES] > -B)) valid = false;
    hllc_mixed<DIM, DIR>(eos, cm, cp, pmd[PRES], ppd[PRES], pmd[VELX + DIR], ppd[VELX + DIR],
                         inv(cm[MASS]), inv(cp[MASS]), fd);
  } else {
    T pm[NE], pp[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      if constexpr (ALP_FAST && P::FAST_FRAME) {
        double G[5], l, r;
#pragma unroll
        for (int m = 0; m < 5; ++m) G[m] = prim[m + 1][n] - prim[m][n];
        pol.increments(G, 1.0, l, r, false);
        pm[n] = prim[C][n] + l;
        pp[n] = prim[C + 1][n] - r;
      } else {
        T arr[W];
#pragma unroll
        for (int m = 0; m < W; ++m) arr[m] = T(prim[m][n]);
        pol.pair(arr, pm[n], pp[n]);
      }
    }
    if (ALP_FAST && pol.default_riemann()) {
      // the upwind side's conservatives alone (hllc_upwind)
      if (!(pm[RHO] > DBL_EPSILON) || !(pp[RHO] > DBL_EPSILON)) valid = false;
      if (!(pm[PRES] > -B) || !(pp[PRES] > -B)) valid = false;
      hllc_flux_primes<DIM, DIR>(eos,
                                 hllc_upwind(eos, pm[RHO], pp[RHO], pm[PRES], pp[PRES],
                                             pm[VELX + DIR], pp[VELX + DIR], inv(pm[RHO]),
                                             inv(pp[RHO])),
                                 pm, pp, fd);
      return valid;
    }
    // PrimeStatesToConservatives (prime_state_handler.h:195-275)
    T cm[NE], cp[NE];
    cm[MASS] = pm[RHO];
    cp[MASS] = pp[RHO];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      cm[MOMX + d] = pm[VELX + d] * pm[RHO];
      cp[MOMX + d] = pp[VELX + d] * pp[RHO];
    }
    cm[ENERGY] = eos_energy<DIM, T>(eos, pm[RHO], pm[VELX], DIM > 1 ? pm[VELX + (DIM > 1)] : T(0),
                                    DIM > 2 ? pm[VELX + 2 * (DIM > 2)] : T(0), pm[PRES]);
    cp[ENERGY] = eos_energy<DIM, T>(eos, pp[RHO], pp[VELX], DIM > 1 ? pp[VELX + (DIM > 1)] : T(0),
                                    DIM > 2 ? pp[VELX + 2 * (DIM > 2)] : T(0), pp[PRES]);
    if (!(cm[MASS] > eps_of<T>()) || !(cp[MASS] > eps_of<T>())) valid = false;
    if (!(double(pm[PRES]) > -B) || !(double(pp[PRES]) > -B)) valid = false;
    // HLLC's own 1/density (hllc_riemann_solver.h:75-78)
    pol.template riemann<DIM, DIR, T>(eos, cm, cp, pm[PRES], pp[PRES], pm[VELX + DIR],
                                      pp[VELX + DIR], inv(cm[MASS]), inv(cp[MASS]), fd);
  }
  return valid;
}

// Flux of one face from its stencil of W cells, the face between the middle two
// (the reference's per-face work: FiniteVolumeScheme::ComputeFluxes<DIR> with the
// selected reconstruction and HLLC, or FluxSplittingScheme::ComputeFluxes<DIR>).
// Writes the flux in double to fd and returns false for a face the reference skips
// (invalid reconstructed state, finite_volume_scheme.cpp:218-225) or whose Roe
// average has a non-positive density (eigendecomposition.h:244).
// P selects reconstruction stencil, Riemann solver and splitting eigenvalues
// (DefaultPolicy: WENO5, HLLC/Einfeldt, Roe; ExtPolicy: run-time choice, FP64).
template <int DIM, int DIR, int SCHEME, typename T, typename P = DefaultPolicy, int W = 6>
__device__ __forceinline__ bool face_compute(Eos const &eos, double B,
                                             double const (&cons)[W][DIM + 2],
                                             double (&fd)[DIM + 2], P const &pol = P()) {
  if constexpr (SCHEME == FV_PRIM)
    return prim_flux<DIM, DIR, T, P, W>(eos, B, cons, fd, pol);
  else if constexpr (ALP_FAST && sizeof(T) == 4)
    return packed_flux<DIM, DIR, SCHEME, P>(eos, B, cons, fd, pol);
  else if constexpr (ALP_FAST && P::FAST_FRAME)
    return frame_flux<DIM, DIR, SCHEME, P>(eos, B, cons, fd, pol);
  else
    return ordered_flux<DIM, DIR, SCHEME, T, P, W>(eos, B, cons, fd, pol);
}

}  // namespace alp
