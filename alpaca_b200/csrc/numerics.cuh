// Device numerics of the ALPACA face flux: stiffened-gas EOS, WENO5-JS, the
// Roe eigensystem, HLLC with Einfeldt speeds and Roe flux-vector splitting.
// Each function states the reference lines (ALPACA src/) whose arithmetic it
// follows; the association order of every sum is kept so that results agree
// with the CPU reference to rounding (FMA contraction is the only difference).
// T is the compute type of reconstruction and flux (double, or float in the
// FP32-flux form); pressure recovery from total energy always runs in double.
//
// Two builds share this file. The strict build (ALP_STRICT, compiled with
// -fmad=false) evaluates every expression exactly as the reference writes it,
// IEEE division included, and reproduces the reference bit for bit. The fast
// build replaces divisions and square roots by refined reciprocals (one
// third-order step each, reused where the same divisor recurs), projects and
// reconstructs the differences of the stencil, evaluates the WENO5 weights of a
// face's two reconstructions with shared second differences, and takes float
// square roots from the hardware approximation; all change results only at the
// rounding level.
#pragma once

#include <cfloat>

#include "layout.cuh"

#ifdef ALP_STRICT
#define ALP_FAST 0
#else
#define ALP_FAST 1
#endif

namespace alp {

// Reciprocal by one third-order Householder iteration on f(y) = 1/y - b
// (Householder 1970: y <- y (1 + e + e^2), e = 1 - b y), seeded with the PTX
// approximate reciprocal: the seed's ~2^-20 relative error becomes its cube,
// 2^-60, in three operations (two Newton steps: four), so that the rounding of
// the last operation is all that is left. For 2^-1022 <= |b| <= 2^1022.
__device__ __forceinline__ double rcp_nr(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double const e = fma(-b, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1/sqrt(x) by one third-order Householder iteration on f(y) = 1/y^2 - x
// (y <- y (1 + e/2 + 3 e^2/8), e = 1 - x y^2), seeded with the PTX approximate
// reciprocal square root (fast build only). The iteration leaves 5/16 e^3, below
// 2^-58; the rounding of x y in e, half of which reaches y, and that of the last
// operation are larger. For normal x.
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double const e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/x: IEEE division in the strict build, rcp_nr (double) or the PTX
// approximate reciprocal (float, one instruction, about 1 ulp) in the fast
// build.
__device__ __forceinline__ double inv(double x) {
  if constexpr (ALP_FAST) return rcp_nr(x);
  else return 1.0 / x;
}
__device__ __forceinline__ float inv(float x) {
  if constexpr (ALP_FAST) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  } else {
    return 1.0f / x;
  }
}
// a / b, where ib is 1/b as returned by inv(b): the strict build divides.
template <typename T> __device__ __forceinline__ T quot(T a, T b, T ib) {
  if constexpr (ALP_FAST) return a * ib;
  else return a / b;
}
template <typename T> __device__ __forceinline__ T quot(T a, T b) {
  if constexpr (ALP_FAST) return a * inv(b);
  else return a / b;
}

// Square root: IEEE in double and in the strict build; in the fast build's
// float arithmetic (the FP32-flux form) the PTX approximate square root, one
// instruction with a few ulp of error against the IEEE sequence.
__device__ __forceinline__ double tsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float tsqrt(float x) {
  if constexpr (ALP_FAST) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  } else {
    return sqrtf(x);
  }
}

// A product rounded on its own (never fused into a following addition).
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }

template <typename T> __device__ __forceinline__ T dmin(T a, T b) { return (b < a) ? b : a; }
template <typename T> __device__ __forceinline__ T dmax(T a, T b) { return (a < b) ? b : a; }
template <typename T> __device__ __forceinline__ T eps_of();
template <> __device__ __forceinline__ double eps_of<double>() { return DBL_EPSILON; }
template <> __device__ __forceinline__ float eps_of<float>() { return FLT_EPSILON; }

// ConsistencyManagedSum with FUSY on (utilities/mathematical_functions.h:79-89)
template <typename T> __device__ __forceinline__ T cms3(T a, T b, T c) {
  T const s1 = (a + b) + c;
  T const s2 = (a + c) + b;
  T const s3 = (b + c) + a;
  T mn = s1, mx = s1;
  if (s2 < mn) mn = s2;
  if (s3 < mn) mn = s3;
  if (mx < s2) mx = s2;
  if (mx < s3) mx = s3;
  return T(0.5) * (mn + mx);
}

// DimensionAwareConsistencyManagedSum (mathematical_functions.h:98-108)
template <int DIM, typename T> __device__ __forceinline__ T dacms(T a, T b, T c) {
  if constexpr (DIM == 1) return a;
  else if constexpr (DIM == 2) return a + b;
  else return cms3(a, b, c);
}

// Sum of three squares: DimensionAwareConsistencyManagedSum in the strict build
// and in 1D / 2D. The fast build's 3D sum is independent of the order of its
// terms as well: it sorts them (the bit patterns of non-negative floating-point
// values order like the values) and adds the two smaller first, two additions and
// integer compares against seven additions and four floating-point compares, so
// that prime states, energies, signal speeds (dt) and the primitive form do not
// change when the axes are exchanged. ORDERED = false adds them as they come, for
// the characteristic forms, whose projections follow an order anyway.
template <int DIM, bool ORDERED = true, typename T>
__device__ __forceinline__ T sum_sq(T a, T b, T c) {
  if constexpr (!ALP_FAST || DIM < 3) {
    return dacms<DIM>(a, b, c);
  } else if constexpr (!ORDERED) {
    return (a + b) + c;
  } else {
    static_assert(sizeof(T) == 8, "the FP32-flux form sums floats unordered");
    long long const ia = __double_as_longlong(a), ib = __double_as_longlong(b);
    long long const ic = __double_as_longlong(c);
    long long const lo = min(ia, ib), hi = max(ia, ib);
    long long const x0 = min(lo, ic), t = max(lo, ic);
    long long const x1 = min(t, hi), x2 = max(t, hi);
    return (__longlong_as_double(x0) + __longlong_as_double(x1)) + __longlong_as_double(x2);
  }
}

// ---- stiffened gas (generic_stiffened_gas.h:40-102, stiffened_gas.cpp:62-149,
//      stiffened_gas_safe.cpp:61-146) --------------------------------------

struct Eos {
  double gamma, B;
  int safe;
};

// one_mass = inv(mass) (unused by the strict build, which divides); ORDERED as in
// sum_sq
template <int DIM, bool ORDERED = true>
__device__ __forceinline__ double eos_pressure(Eos const &e, double mass, double mx, double my,
                                               double mz, double energy, double one_mass) {
  if (e.safe) {
    double const m = dmax(mass, DBL_EPSILON);
    double const p =
        -e.gamma * e.B +
        (e.gamma - 1.0) * (energy - quot(0.5 * sum_sq<DIM, ORDERED>(mx * mx, my * my, mz * mz), m,
                                         mass > DBL_EPSILON ? one_mass : inv(m)));
    return dmax(p, -e.B + DBL_EPSILON);
  }
  double const q = 0.5 * sum_sq<DIM, ORDERED>(mx * mx, my * my, mz * mz);
  return -e.gamma * e.B + (e.gamma - 1.0) * (energy - quot(q, mass, one_mass));
}
template <int DIM>
__device__ __forceinline__ double eos_pressure(Eos const &e, double mass, double mx, double my,
                                               double mz, double energy) {
  return eos_pressure<DIM>(e, mass, mx, my, mz, energy, ALP_FAST ? inv(mass) : 0.0);
}

template <int DIM, typename T>
__device__ __forceinline__ T eos_energy(Eos const &e, T rho, T u, T v, T w, T p) {
  T const g = T(e.gamma), B = T(e.B);
  return quot(p + g * B, g - T(1)) + (T(0.5) * sum_sq<DIM>(u * u, v * v, w * w) * rho);
}

// one_rho = inv(rho) (unused by the strict build)
template <typename T>
__device__ __forceinline__ T eos_speed_of_sound(Eos const &e, T rho, T p, T one_rho) {
  T const g = T(e.gamma), B = T(e.B);
  if (e.safe) {
    T const r = dmax(rho, eps_of<T>());
    T const c2 = quot(g * (p + B), r, rho > eps_of<T>() ? one_rho : inv(r));
    return tsqrt(dmax(c2, eps_of<T>()));
  }
  return tsqrt(quot(g * (p + B), rho, one_rho));
}
template <typename T> __device__ __forceinline__ T eos_speed_of_sound(Eos const &e, T rho, T p) {
  return eos_speed_of_sound<T>(e, rho, p, ALP_FAST ? inv(rho) : T(0));
}

// ---- WENO5-JS (stencils/spatial_reconstruction_stencils/weno5.h:88-158) --
// As the reference writes it: the strict build's form.
// a[0..5] are cells i-2..i+3 around face i+1/2; UpwindLeft uses {offset 0,
// sign +1}, UpwindRight {1, -1} (stencils/apply_wrapper.h:47-57).
template <typename T>
__device__ __forceinline__ T weno5_core(T v1, T v2, T v3, T v4, T v5) {
  T const c1 = T(13.0 / 12.0), c2 = T(0.25);
  T const s11 = v1 + T(-2.0) * v2 + v3;
  T const s12 = v1 + T(-4.0) * v2 + T(3.0) * v3;
  T const s1 = c1 * s11 * s11 + c2 * s12 * s12;
  T const s21 = v2 + T(-2.0) * v3 + v4;
  T const s22 = v2 + T(-1.0) * v4;
  T const s2 = c1 * s21 * s21 + c2 * s22 * s22;
  T const s31 = v3 + T(-2.0) * v4 + v5;
  T const s32 = T(3.0) * v3 + T(-4.0) * v4 + v5;
  T const s3 = c1 * s31 * s31 + c2 * s32 * s32;
  T const eps = T(1.0e-6);
  T const q1 = T(2.0 / 6.0) * v1 + T(-7.0 / 6.0) * v2 + T(11.0 / 6.0) * v3;
  T const q2 = T(-1.0 / 6.0) * v2 + T(5.0 / 6.0) * v3 + T(2.0 / 6.0) * v4;
  T const q3 = T(2.0 / 6.0) * v3 + T(5.0 / 6.0) * v4 + T(-1.0 / 6.0) * v5;
  T const t1 = (s1 + eps) * (s1 + eps);
  T const t2 = (s2 + eps) * (s2 + eps);
  T const t3 = (s3 + eps) * (s3 + eps);
  T const a1 = quot(T(0.1), t1);
  T const a2 = quot(T(0.6), t2);
  T const a3 = quot(T(0.3), t3);
  T const one_a_sum = quot(T(1.0), a1 + a2 + a3);
  T const w1 = a1 * one_a_sum;
  T const w2 = a2 * one_a_sum;
  T const w3 = a3 * one_a_sum;
  return w1 * q1 + w2 * q2 + w3 * q3;
}
template <typename T> __device__ __forceinline__ T weno5_left(T const (&a)[6]) {
  return weno5_core(a[0], a[1], a[2], a[3], a[4]);
}
template <typename T> __device__ __forceinline__ T weno5_right(T const (&a)[6]) {
  return weno5_core(a[5], a[4], a[3], a[2], a[1]);
}

// Fast-build WENO5-JS from first differences. For a stencil v1..v5 around
// the face of v3, with g1..g4 = v2-v1, v3-v2, v4-v3, v5-v4, the second
// differences d1..d3 = g2-g1, g3-g2, g4-g3, a = g2 + d1 and b = g3 - d3, the
// three candidate values are
//   q1 = v3 + (2 a + g2) / 6, q2 = v3 + (2 g3 + g2) / 6, q3 = v3 + (2 g3 + b) / 6
// and the reference's smoothness indicators 13/12 (..)^2 + 1/4 (..)^2 become
//   4/3 d1^2 + g2 a, 4/3 d2^2 + g2 g3, 4/3 d3^2 + g3 b
// (in each the terms' absolute sum stays below twice the indicator, so no
// digits are lost to cancellation). q_k = 4/3 d_k^2 + eps is passed in: the two
// sides of a face share two of them. With t_k the squared indicators (eps
// added) and the ideal weights 0.1, 0.6, 0.3 as 1, 6, 3, scaled by t1 t2 t3,
// the result is v3 + num / (6 den). The differences of the mirrored stencil,
// reversed without their sign change, negate num and leave den unchanged.
// 20 operations a side; with the indicators as two squares each it took 26.
struct Weno5Frac { double num, den; };

__device__ __forceinline__ double weno5_q(double d, double eps) {
  return fma((4.0 / 3.0) * d, d, eps);
}
__device__ __forceinline__ Weno5Frac weno5_frac(double g2, double g3, double d1, double d3,
                                                double q1, double q2, double q3) {
  double const a = g2 + d1, b = g3 - d3;
  double const s1 = fma(g2, a, q1), s2 = fma(g2, g3, q2), s3 = fma(g3, b, q3);
  double const r1 = fma(2.0, a, g2), r2 = fma(2.0, g3, g2), r3 = fma(2.0, g3, b);
  double const t1 = s1 * s1, t2 = s2 * s2, t3 = s3 * s3;
  // num = t2 t3 r1 + 3 t1 (2 t3 r2 + t2 r3), den the same with r = 1
  double const y = 3.0 * t1, z = t3 + t3, p = t2 * t3;
  return {fma(y, fma(z, r2, t2 * r3), p * r1), fma(y, z + t2, p)};
}

// num_l / (6 den_l) and num_r / (6 den_r). One reciprocal serves both while the
// product of the denominators, each between ~1e-23 (eps^4) and ~1e2 |g|^8, stays
// in range: for differences up to ~1e17 and the reference's eps. `apart` takes a
// reciprocal per side, for differences up to ~1e38 and eps down to ~1e-77 (one
// operation more).
__device__ __forceinline__ void weno5_finish(Weno5Frac const &l, Weno5Frac const &r,
                                             double &left, double &right, bool apart) {
  if (apart) {
    left = l.num * inv(6.0 * l.den);
    right = r.num * inv(6.0 * r.den);
    return;
  }
  double const rr = inv((6.0 * l.den) * r.den);
  left = l.num * (r.den * rr);
  right = r.num * (l.den * rr);
}

// Both reconstructions of a face from the five first differences of its six
// cells: the UpwindLeft value is (left cell) + left, the UpwindRight value
// (right cell) - right. eps is the reference's 1e-6, times the square of the
// factor by which the caller scaled the differences (WENO5 of scaled data with
// eps scaled alike is the scaled WENO5).
__device__ __forceinline__ void weno5_increments(double const (&G)[5], double eps, double &left,
                                                 double &right, bool apart) {
  double const D1 = G[1] - G[0], D2 = G[2] - G[1], D3 = G[3] - G[2], D4 = G[4] - G[3];
  double const q2 = weno5_q(D2, eps), q3 = weno5_q(D3, eps);
  weno5_finish(weno5_frac(G[1], G[2], D1, D3, weno5_q(D1, eps), q2, q3),
               weno5_frac(G[3], G[2], -D4, -D2, weno5_q(D4, eps), q3, q2), left, right, apart);
}
// The same for two arrays (flux splitting): UpwindLeft from the differences
// A[0..3], UpwindRight from B[1..4].
__device__ __forceinline__ void weno5_increments_two(double const (&A)[5], double const (&B)[5],
                                                     double eps, double &left, double &right,
                                                     bool apart) {
  double const A1 = A[1] - A[0], A2 = A[2] - A[1], A3 = A[3] - A[2];
  double const B2 = B[2] - B[1], B3 = B[3] - B[2], B4 = B[4] - B[3];
  weno5_finish(weno5_frac(A[1], A[2], A1, A3, weno5_q(A1, eps), weno5_q(A2, eps), weno5_q(A3, eps)),
               weno5_frac(B[3], B[2], -B4, -B2, weno5_q(B4, eps), weno5_q(B3, eps), weno5_q(B2, eps)),
               left, right, apart);
}

// ---- packed FP32 pairs (Blackwell f32x2: one instruction for two lanes) ----
// Used by the fast build's FP32-flux form, where both sides of a face run the
// same arithmetic: lane x the left (UpwindLeft) side, lane y the right one.
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// a - b, rounded once (a + (-1) b)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, dup2(-1.0f), a); }

// weno5_frac of both sides of a face as the lanes of packed arithmetic: lane x
// from the first differences g1..g4 of the UpwindLeft stencil, lane y from those
// of the mirrored UpwindRight stencil (reversed, sign kept). Returns the
// increments num / (6 den). The t_k are first multiplied by the power of two
// that brings the largest into [1, 2) (exact: the scale is built from the
// exponent bits), so the products stay inside the float range; a product that
// underflows belongs to a weight below 2^-126 of the largest. One reciprocal per
// side (a scaled denominator can be as small as the ratio of two smoothness
// terms, so the product of two could underflow).
__device__ __forceinline__ float2 weno5_packed(float2 g1, float2 g2, float2 g3, float2 g4,
                                               float eps) {
  float2 const two = dup2(2.0f), c = dup2(4.0f / 3.0f), e = dup2(eps);
  float2 const d1 = sub2(g2, g1), d2 = sub2(g3, g2), d3 = sub2(g4, g3);
  float2 const a = add2(g2, d1), b = sub2(g3, d3);
  float2 const s1 = fma2(g2, a, fma2(mul2(c, d1), d1, e));
  float2 const s2 = fma2(g2, g3, fma2(mul2(c, d2), d2, e));
  float2 const s3 = fma2(g3, b, fma2(mul2(c, d3), d3, e));
  float2 const r1 = fma2(two, a, g2), r2 = fma2(two, g3, g2), r3 = fma2(two, g3, b);
  float2 const t1 = mul2(s1, s1), t2 = mul2(s2, s2), t3 = mul2(s3, s3);
  // per lane: the power of two that brings the largest t_k into [1, 2)
  unsigned const ex = min((__float_as_uint(fmaxf(t1.x, fmaxf(t2.x, t3.x))) >> 23) & 0xffu, 253u);
  unsigned const ey = min((__float_as_uint(fmaxf(t1.y, fmaxf(t2.y, t3.y))) >> 23) & 0xffu, 253u);
  float2 const sc = make_float2(__uint_as_float((254u - ex) << 23), __uint_as_float((254u - ey) << 23));
  float2 const u1 = mul2(t1, sc), u2 = mul2(t2, sc), u3 = mul2(t3, sc);
  float2 const y = mul2(dup2(3.0f), u1), z = add2(u3, u3), p = mul2(u2, u3);
  float2 const num = fma2(y, fma2(z, r2, mul2(u2, r3)), mul2(p, r1));
  float2 const q = mul2(dup2(6.0f), fma2(y, add2(z, u2), p));
  return mul2(num, make_float2(inv(q.x), inv(q.y)));
}

// ---- Roe eigensystem (solvers/eigendecomposition.h:181-467) --------------
// The left/right eigenvector matrices are never stored: their entries are
// generated from the Roe-averaged scalars below when applied.
template <typename T> struct Roe {
  T up, u1, u2;     // principal, first and second minor velocity
  T H;              // enthalpy
  T c, cc, one_cc;  // speed of sound, c^2, 1/c^2
  T half_cc;        // 0.5 * one_cc
  T gru;            // Gruneisen coefficient gamma - 1
  T rho, one_rho;   // Roe density and its inverse
  T q2;             // |u|^2 (dimension-aware sum)
};

// minor directions (eigendecomposition.h:84-125)
template <int DIR> struct Minor;
template <> struct Minor<0> { static constexpr int m1 = 1, m2 = 2; };
template <> struct Minor<1> { static constexpr int m1 = 0, m2 = 2; };
template <> struct Minor<2> { static constexpr int m1 = 0, m2 = 1; };

// symmetry-preserving summation order of the characteristic projection
// (solvers/state_reconstruction/state_reconstruction.h:35-58): position q of
// the sequence for direction DIR.
template <int DIM, int DIR> __host__ __device__ constexpr int sum_seq(int q) {
  if (DIM == 1) return q == 0 ? MOMX : (q == 1 ? MASS : ENERGY);
  if (DIM == 2) return q < 2 ? MOMX + q : (q == 2 ? MASS : ENERGY);
  if (q >= 3) return q == 3 ? MASS : ENERGY;
  // 3D: X -> (MomY, MomZ, MomX), Y -> (MomZ, MomX, MomY), Z -> (MomX, MomY, MomZ)
  return MOMX + (DIR + 1 + q) % 3;
}

// Cell quantities the Roe average needs; conservatives are double.
template <int DIM, int DIR> struct CellPrims {
  double rho, one_rho, p, up, u1, u2, H;
};

template <int DIM, int DIR>
__device__ __forceinline__ CellPrims<DIM, DIR> cell_prims(Eos const &e, double const (&c)[DIM + 2]) {
  CellPrims<DIM, DIR> r;
  r.rho = c[MASS];
  r.one_rho = inv(c[MASS]);
  double const mx = c[MOMX];
  double const my = DIM > 1 ? c[MOMX + (DIM > 1 ? 1 : 0)] : 0.0;
  double const mz = DIM > 2 ? c[MOMX + (DIM > 2 ? 2 : 0)] : 0.0;
  // velocities from the prime-state buffer: momentum * (1/rho)
  // (prime_state_handler.h:293-311)
  r.up = c[MOMX + DIR] * r.one_rho;
  r.u1 = DIM > 1 ? c[MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0)] * r.one_rho : 0.0;
  r.u2 = DIM > 2 ? c[MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0)] * r.one_rho : 0.0;
  r.p = eos_pressure<DIM, false>(e, c[MASS], mx, my, mz, c[ENERGY], r.one_rho);
  // Enthalpy (stiffened_gas.cpp:88-96 / stiffened_gas_safe.cpp:77-84)
  r.H = e.safe ? quot(c[ENERGY] + r.p, dmax(c[MASS], DBL_EPSILON))
               : quot(c[ENERGY] + r.p, c[MASS], r.one_rho);
  return r;
}

// Roe averages of one face (eigendecomposition.h:252-310)
template <int DIM, int DIR, typename T>
__device__ __forceinline__ Roe<T> roe_average(Eos const &e, CellPrims<DIM, DIR> const &t,
                                              CellPrims<DIM, DIR> const &n) {
  Roe<T> r;
  T const gB = T(e.gamma * e.B);
  T const psi_t = (T(t.p) + gB) * T(t.one_rho);
  T const psi_n = (T(n.p) + gB) * T(n.one_rho);
  // sr_k * rho_div are the Roe weights sqrt(rho_k) / (sqrt(rho_t) + sqrt(rho_n))
  constexpr bool WEIGHTS = ALP_FAST && sizeof(T) == 8;
  T sr_t, sr_n, rho_div;
  if constexpr (WEIGHTS) {
    // the weights themselves (rho_div = 1) from one reciprocal square root:
    // mu = sqrt(rho_t / rho_n), lambda = 1 / mu, w_t = 1 / (1 + lambda),
    // w_n = lambda w_t, Roe density rho_t lambda and its inverse mu / rho_t
    T const ratio = n.rho * t.one_rho;
    T const mu = rsqrt_nr(ratio);
    T const lambda = ratio * mu;
    sr_t = inv(T(1) + lambda);
    sr_n = lambda * sr_t;
    rho_div = T(1);
    r.rho = t.rho * lambda;
    r.one_rho = t.one_rho * mu;
  } else {
    sr_t = tsqrt(T(t.rho));
    sr_n = tsqrt(T(n.rho));
    rho_div = quot(T(1), sr_t + sr_n);
    r.rho = sr_t * sr_n;
    r.one_rho = quot(T(1), r.rho);
  }
  r.up = ((T(t.up) * sr_t) + (T(n.up) * sr_n)) * rho_div;
  r.u1 = ((T(t.u1) * sr_t) + (T(n.u1) * sr_n)) * rho_div;
  r.u2 = ((T(t.u2) * sr_t) + (T(n.u2) * sr_n)) * rho_div;
  T const psi = ((psi_t * sr_t) + (psi_n * sr_n)) * rho_div;
  r.H = (T(t.H) * sr_t + T(n.H) * sr_n) * rho_div;
  r.gru = T(e.gamma - 1.0);
  r.q2 = sum_sq<DIM, false>(r.up * r.up, r.u1 * r.u1, r.u2 * r.u2);
  T const dup = T(t.up) - T(n.up), du1 = T(t.u1) - T(n.u1), du2 = T(t.u2) - T(n.u2);
  T const tmp = sum_sq<DIM, false>(dup * dup, du1 * du1, du2 * du2);
  // 0.5 rho_roe rho_div^2 = 0.5 w_t w_n
  T const jump = WEIGHTS ? T(0.5) * (sr_t * sr_n) * tmp
                         : T(0.5) * r.rho * (rho_div * rho_div) * tmp;
  T const p_over_rho =
      ((T(t.p) * T(t.one_rho)) * sr_t + (T(n.p) * T(n.one_rho)) * sr_n) * rho_div + jump;
  r.cc = psi + r.gru * p_over_rho;
  r.one_cc = quot(T(1), r.cc);
  r.c = tsqrt(r.cc);
  r.half_cc = T(0.5) * r.one_cc;
  return r;
}

// Row n of the left eigenvector matrix, indexed by conservative equation
// (eigendecomposition.h:316-359). Entries that are structurally zero are
// returned as 0 and skipped by the projection (adding 0*u leaves a sum unchanged).
template <int DIM, int DIR, typename T>
__device__ __forceinline__ void left_row(int n, Roe<T> const &r, T (&L)[DIM + 2]) {
  constexpr int NE = DIM + 2;
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
#pragma unroll
  for (int l = 0; l < NE; ++l) L[l] = T(0);
  if (n == 0 || n == NE - 1) {
    T const sgn = n == 0 ? T(1) : T(-1);
    // 0.5/cc * (gru q^2 - gru H +/- (u +/- c) c)
    if (n == 0)
      L[MASS] = r.half_cc * (r.gru * r.q2 - r.gru * r.H + (r.up + r.c) * r.c);
    else
      L[MASS] = r.half_cc * (r.gru * r.q2 - r.gru * r.H - (r.up - r.c) * r.c);
    L[mP] = r.half_cc * (-r.up * r.gru - sgn * r.c);
    if (DIM > 1) L[m1] = r.half_cc * (-r.u1 * r.gru);
    if (DIM > 2) L[m2] = r.half_cc * (-r.u2 * r.gru);
    L[ENERGY] = r.half_cc * r.gru;
  } else if (n == DIM) {  // principal-momentum wave
    L[MASS] = r.one_cc * (r.H - r.q2);
    L[mP] = r.one_cc * r.up;
    if (DIM > 1) L[m1] = r.one_cc * r.u1;
    if (DIM > 2) L[m2] = r.one_cc * r.u2;
    L[ENERGY] = -r.one_cc;
  } else if (n == 1) {  // first minor momentum (DIM >= 2)
    L[MASS] = r.u1 * r.one_rho;
    L[m1] = -r.one_rho;
  } else {  // n == 2, second minor momentum (DIM == 3)
    L[MASS] = -r.u2 * r.one_rho;
    L[m2] = r.one_rho;
  }
}

// TransformToPhysicalSpace with generated right eigenvectors
// (eigendecomposition.h:144-165 and 366-409): linear waves summed first, then
// the nonlinear pair (u-c, u+c) added together.
template <int DIM, int DIR, typename T>
__device__ __forceinline__ void to_physical(Roe<T> const &r, T const (&ch)[DIM + 2],
                                            T (&out)[DIM + 2]) {
  constexpr int NE = DIM + 2;
  constexpr int EV = DIM;
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
  // R[MASS][*] = (1, 0, 0, gru, 1)
  {
    T s = ch[EV] * r.gru;  // minor columns are zero
    out[MASS] = s + (ch[0] * T(1) + ch[NE - 1] * T(1));
  }
  // R[mP][*] = (u-c, 0, 0, gru*u, u+c)
  {
    T s = ch[EV] * (r.gru * r.up);
    out[mP] = s + (ch[0] * (r.up - r.c) + ch[NE - 1] * (r.up + r.c));
  }
  if constexpr (DIM > 1) {
    // R[m1][*] = (u1, -rho, 0, gru*u1, u1)
    T s = ch[1] * (-r.rho);
    s = s + ch[EV] * (r.gru * r.u1);
    out[m1] = s + (ch[0] * r.u1 + ch[NE - 1] * r.u1);
  }
  if constexpr (DIM > 2) {
    // R[m2][*] = (u2, 0, rho, gru*u2, u2)
    T s = ch[2] * r.rho;
    s = s + ch[EV] * (r.gru * r.u2);
    out[m2] = s + (ch[0] * r.u2 + ch[NE - 1] * r.u2);
  }
  // R[ENERGY][*] = (H - u c, -u1 rho, rho u2, gru H - c c, H + u c)
  {
    T s = T(0);
    if constexpr (DIM == 2) s = ch[1] * (-r.u1 * r.rho);
    if constexpr (DIM > 2) {
      // The two minor-wave terms are rounded as products before they are
      // added, so that this sum does not depend on which minor momentum is
      // numbered first (rotate.cuh numbers those of y faces the other way
      // round). The strict build rounds every product anyway; the fast build's
      // projection adds its terms in an order, so its characteristic fluxes
      // still change at rounding level when the minor momenta are exchanged.
      T const t1 = rmul(ch[1], -r.u1 * r.rho);
      T const t2 = rmul(ch[2], r.rho * r.u2);
      s = t1 + t2;
    }
    s = s + ch[EV] * (r.gru * r.H - r.c * r.c);
    out[ENERGY] = s + (ch[0] * (r.H - r.up * r.c) + ch[NE - 1] * (r.H + r.up * r.c));
  }
}

// to_physical of both sides at once: ch[n] = (left, right) characteristic
// values; the same right-eigenvector entries, packed.
template <int DIM, int DIR>
__device__ __forceinline__ void to_physical_packed(Roe<float> const &r, float2 const (&ch)[DIM + 2],
                                                   float2 (&out)[DIM + 2]) {
  constexpr int NE = DIM + 2;
  constexpr int EV = DIM;
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
  float2 const a = ch[0], z = ch[NE - 1], w = ch[EV];
  out[MASS] = fma2(w, dup2(r.gru), add2(a, z));
  out[mP] = fma2(w, dup2(r.gru * r.up), fma2(a, dup2(r.up - r.c), mul2(z, dup2(r.up + r.c))));
  if constexpr (DIM > 1)
    out[m1] = fma2(ch[1], dup2(-r.rho),
                   fma2(w, dup2(r.gru * r.u1), mul2(add2(a, z), dup2(r.u1))));
  if constexpr (DIM > 2)
    out[m2] = fma2(ch[2], dup2(r.rho),
                   fma2(w, dup2(r.gru * r.u2), mul2(add2(a, z), dup2(r.u2))));
  float2 s = fma2(w, dup2(r.gru * r.H - r.c * r.c),
                  fma2(a, dup2(r.H - r.up * r.c), mul2(z, dup2(r.H + r.up * r.c))));
  if constexpr (DIM == 2) s = fma2(ch[1], dup2(-r.u1 * r.rho), s);
  if constexpr (DIM > 2) {
    // the two minor-wave products rounded before they are added, as in
    // to_physical
    s = add2(add2(mul2(ch[1], dup2(-r.u1 * r.rho)), mul2(ch[2], dup2(r.rho * r.u2))), s);
  }
  out[ENERGY] = s;
}

// ---- the fast build's FP64 characteristic frame ------------------------------
// The same Roe eigensystem with its rows factored. For a difference x =
// (rho, E, m) of conserved states (or of physical fluxes) let
//   Dp = mp - up rho, D1 = m1 - u1 rho, D2 = m2 - u2 rho,
//   V  = (E - H rho - up Dp - u1 D1 - u2 D2) / c^2;
// the characteristic values of the eigenvector matrices above are then
//   (u - c, u + c):  ((rho + gru V) -/+ Dp / c) / 2,  entropy wave: -V,
//   minor waves:     -D1 / rho_roe, D2 / rho_roe.
// 12 operations per difference against 19 with the rows multiplied out. The
// constant factors (1/2, 1/rho_roe) are left out of the values and go into the
// eps of their reconstruction instead (weno5_increments).
template <int DIM> struct CharFrame {
  double up, u1, u2, H, gru;       // Roe averages, gamma - 1
  double c, one_c, cc, one_cc;     // speed of sound, its inverse and squares
  double Hcc, wp, w1, w2;          // H / c^2, u / c^2
  double rho2;                     // Roe density squared (the product of the densities)
};

// Cell quantities of the frame: 1/rho, velocities, pressure, enthalpy, c^2.
template <int DIM> struct CharCell {
  double one, up, u1, u2, p, H, cc;
};

template <int DIM, int DIR>
__device__ __forceinline__ CharCell<DIM> char_cell(Eos const &e, double const (&c)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
  CharCell<DIM> r;
  r.one = inv(c[MASS]);
  r.up = c[mP] * r.one;
  double um = r.up * c[mP];
  r.u1 = r.u2 = 0.0;
  if constexpr (DIM > 1) {
    r.u1 = c[m1] * r.one;
    um = fma(r.u1, c[m1], um);
  }
  if constexpr (DIM > 2) {
    r.u2 = c[m2] * r.one;
    um = fma(r.u2, c[m2], um);
  }
  double const gB = e.gamma * e.B;
  double oneH = r.one;
  if (e.safe && !(c[MASS] > DBL_EPSILON)) {
    // StiffenedGasSafe divides by max(rho, eps)
    oneH = 1.0 / DBL_EPSILON;
    um *= c[MASS] * oneH;
  }
  r.p = fma(e.gamma - 1.0, fma(-0.5, um, c[ENERGY]), -gB);
  if (e.safe) r.p = dmax(r.p, -e.B + DBL_EPSILON);
  r.H = (c[ENERGY] + r.p) * oneH;
  r.cc = fma(e.gamma, r.p, gB) * r.one;
  return r;
}

// Roe average of the cells t (left) and n: with the weights w_t = 1 / (1 +
// lambda), lambda = sqrt(rho_n / rho_t), and w_n = lambda w_t, an average is
// a_n + w_t (a_t - a_n), and c^2 = avg(c^2) + (gamma - 1) w_t w_n |du|^2 / 2
// (psi + gru p / rho of eigendecomposition.h:262-300 is a cell's own c^2).
template <int DIM, int DIR>
__device__ __forceinline__ CharFrame<DIM> char_frame(Eos const &e, CharCell<DIM> const &t,
                                                     CharCell<DIM> const &n, double rho_t,
                                                     double rho_n) {
  CharFrame<DIM> r;
  double const ratio = rho_n * t.one;
  double const lambda = ratio * rsqrt_nr(ratio);
  double const wt = inv(1.0 + lambda);
  double const du = t.up - n.up;
  r.up = fma(wt, du, n.up);
  double d2 = du * du;
  r.u1 = r.u2 = 0.0;
  if constexpr (DIM > 1) {
    double const d = t.u1 - n.u1;
    r.u1 = fma(wt, d, n.u1);
    d2 = fma(d, d, d2);
  }
  if constexpr (DIM > 2) {
    double const d = t.u2 - n.u2;
    r.u2 = fma(wt, d, n.u2);
    d2 = fma(d, d, d2);
  }
  r.H = fma(wt, t.H - n.H, n.H);
  r.gru = e.gamma - 1.0;
  r.cc = fma((0.5 * r.gru) * (lambda * (wt * wt)), d2, fma(wt, t.cc - n.cc, n.cc));
  r.one_c = rsqrt_nr(r.cc);
  r.c = r.cc * r.one_c;
  r.one_cc = r.one_c * r.one_c;
  r.Hcc = r.H * r.one_cc;
  r.wp = r.up * r.one_cc;
  r.w1 = r.u1 * r.one_cc;
  r.w2 = r.u2 * r.one_cc;
  r.rho2 = rho_t * rho_n;
  return r;
}

// Scaled characteristic values of a difference x (conserved-field order) in
// wave order: 2 (u - c), minor waves -rho_roe / +rho_roe, -entropy, 2 (u + c).
template <int DIM, int DIR>
__device__ __forceinline__ void char_project(CharFrame<DIM> const &r, double const (&x)[DIM + 2],
                                             double (&ch)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
  double const rho = x[MASS];
  double const Dp = fma(-r.up, rho, x[mP]);
  double V = fma(-r.wp, Dp, fma(-r.Hcc, rho, r.one_cc * x[ENERGY]));
  if constexpr (DIM > 1) {
    ch[1] = fma(-r.u1, rho, x[m1]);
    V = fma(-r.w1, ch[1], V);
  }
  if constexpr (DIM > 2) {
    ch[2] = fma(-r.u2, rho, x[m2]);
    V = fma(-r.w2, ch[2], V);
  }
  double const s = fma(r.gru, V, rho);
  ch[DIM] = V;
  ch[0] = fma(-r.one_c, Dp, s);
  ch[DIM + 1] = fma(r.one_c, Dp, s);
}

// Whether wave n is one of the minor waves.
template <int DIM> __host__ __device__ constexpr bool minor_wave(int n) {
  return n > 0 && n < DIM;
}

// The minor waves' values carry a factor rho_roe: momentum-sized, they span more
// than the other waves' values, so their reconstruction takes a reciprocal per side
// (weno5_finish). Where the product rho2 of the densities is below kMinorRho2, the
// fourth power of its eps would leave the double range all the same.
constexpr double kMinorRho2 = 1.0e-60;

// Square of the factor on the characteristic values of wave n in these scales,
// minor_scale that of the minor waves.
template <int DIM>
__device__ __forceinline__ double char_scale(double minor_scale, int n) {
  return n == 0 || n == DIM + 1 ? 4.0 : (n == DIM ? 1.0 : minor_scale);
}

// Flux splitting takes any positive density: below the line the minor waves'
// values are multiplied by `unit`, a power of two near 1 / rho_roe, for their
// reconstruction. (The finite-volume forms refuse reconstructed densities below
// 2.2e-16 and keep kMinorRho2 as the least scale: on the faces they accept that
// changes the weights of minor values below 1e-33 only, nothing beside the momenta
// of such densities. The branch cost FV char 3 % through its registers, flux
// splitting 1 %.)
struct MinorUnits {
  double scale, unit, back;
  bool tiny;
};
__device__ __forceinline__ MinorUnits minor_units(double rho2) {
  MinorUnits u{rho2, 1.0, 1.0, !(rho2 > kMinorRho2)};
  if (__builtin_expect(u.tiny, 0)) {
    int const h = (1023 - ((__double2hiint(rho2) >> 20) & 0x7ff)) / 2;
    u.unit = __hiloint2double((1023 + h) << 20, 0);
    u.back = __hiloint2double((1023 - h) << 20, 0);
    u.scale = (rho2 * u.unit) * u.unit;
  }
  return u;
}

// base + sgn (the conserved difference whose scaled characteristic values are ch).
template <int DIM, int DIR>
__device__ __forceinline__ void char_restore(CharFrame<DIM> const &r, double const (&base)[DIM + 2],
                                             double const (&ch)[DIM + 2], double sgn,
                                             double (&out)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  constexpr int m1 = MOMX + (DIM > 1 ? Minor<DIR>::m1 : 0);
  constexpr int m2 = MOMX + (DIM > 2 ? Minor<DIR>::m2 : 0);
  double const h = 0.5 * sgn;
  double const rho = fma(h, ch[0] + ch[DIM + 1], (-sgn * r.gru) * ch[DIM]);
  double const cd = (h * r.c) * (ch[DIM + 1] - ch[0]);
  out[MASS] = base[MASS] + rho;
  out[mP] = fma(r.up, rho, base[mP] + cd);
  double E = fma(r.H, rho, fma(r.up, cd, fma(sgn * r.cc, ch[DIM], base[ENERGY])));
  if constexpr (DIM > 1) {
    double const d = sgn * ch[1];
    out[m1] = fma(r.u1, rho, base[m1] + d);
    E = fma(r.u1, d, E);
  }
  if constexpr (DIM > 2) {
    double const d = sgn * ch[2];
    out[m2] = fma(r.u2, rho, base[m2] + d);
    E = fma(r.u2, d, E);
  }
  out[ENERGY] = E;
}

// ---- HLLC with Einfeldt signal speeds -------------------------------------
// The fast build's FP64 HLLC: the upwind star flux alone. Where the reference
// averages the two (S* = 0) they are equal up to rounding: F*_L - F*_R =
// S* (U*_L - U*_R). With S the unclamped speed of the upwind side, Sc the
// clamped one, chi = (S - v) / (S - S*) and k = v + Sc (chi - 1), the fluxes are
//   mass rho k, momentum p + rho (v^2 + Sc (chi S* - v)), minor momenta q k,
//   energy E k + v p + Sc chi (S* - v) (rho S* + p / (Sc - v)).
struct HllcUpwind {
  bool right;        // the upwind side is the right one
  double rho, p, k;  // its density and pressure; the advecting speed
  double g, pe;      // momentum per density beside p; energy beside E k
};

// c^2 of a state (generic_stiffened_gas.h; the safe variant's floors)
__device__ __forceinline__ double eos_cc(Eos const &e, double rho, double p, double one_rho) {
  double const gp = e.gamma * (p + e.B);
  if (e.safe)
    return dmax(gp * (rho > DBL_EPSILON ? one_rho : inv(dmax(rho, DBL_EPSILON))), DBL_EPSILON);
  return gp * one_rho;
}

__device__ __forceinline__ HllcUpwind hllc_upwind(Eos const &e, double rl, double rr, double pl,
                                                  double pr, double vl, double vr, double one_l,
                                                  double one_r) {
  double const ccl = eos_cc(e, rl, pl, one_l), ccr = eos_cc(e, rr, pr, one_r);
  // Einfeldt: Roe weights wl = 1 / (1 + lambda), wr = lambda wl, lambda = sqrt(rr / rl)
  double const ratio = rr * one_l;
  double const lambda = ratio * rsqrt_nr(ratio);
  double const wl = inv(1.0 + lambda);
  double const dv = vl - vr;
  double const u = fma(wl, dv, vr);
  double const ce2 = fma((0.5 * lambda) * (wl * wl), dv * dv, fma(wl, ccl - ccr, ccr));
  double const ce = ce2 * rsqrt_nr(ce2);
  double const cl = ccl * rsqrt_nr(ccl), cr = ccr * rsqrt_nr(ccr);
  double const sl = dmin(u - ce, vl - cl), sr = dmax(u + ce, vr + cr);
  double const al = rl * (sl - vl), ar = rr * (sr - vr);
  double const ss = fma(vl, al, fma(-vr, ar, pr - pl)) * inv(al - ar);
  HllcUpwind h;
  h.right = ss < 0.0;
  h.rho = h.right ? rr : rl;
  h.p = h.right ? pr : pl;
  double const v = h.right ? vr : vl;
  double const s = h.right ? sr : sl;
  double const sc = h.right ? dmax(sr, 0.0) : dmin(sl, 0.0);
  double const dss = ss - v;
  double const dchi = dss * inv(s - ss);  // chi - 1
  h.k = fma(sc, dchi, v);
  double const chi = 1.0 + dchi;
  h.g = fma(v, v, sc * fma(dchi, ss, dss));
  h.pe = fma(v, h.p, (sc * (chi * dss)) * fma(h.rho, ss, h.p * inv(sc - v)));
  return h;
}

// Flux of the upwind star state from its side's conserved state.
template <int DIM, int DIR>
__device__ __forceinline__ void hllc_flux(HllcUpwind const &h, double const (&cl)[DIM + 2],
                                          double const (&cr)[DIM + 2], double (&flux)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  flux[MASS] = h.rho * h.k;
  flux[mP] = fma(h.rho, h.g, h.p);
  flux[ENERGY] = fma(h.right ? cr[ENERGY] : cl[ENERGY], h.k, h.pe);
#pragma unroll
  for (int d = 0; d < DIM - 1; ++d) {
    int const mm = MOMX + (d == 0 ? Minor<DIR>::m1 : Minor<DIR>::m2);
    flux[mm] = (h.right ? cr[mm] : cl[mm]) * h.k;
  }
}

// Sum of a[d] b[d] over the axes, the principal one fused onto the sum of the two
// minor products, each rounded on its own: the same bits with the minor axes
// exchanged (the fast build's primitive form; one operation more than a chain).
template <int DIM, int DIR>
__device__ __forceinline__ double axis_dot(double const (&a)[DIM], double const (&b)[DIM]) {
  if constexpr (DIM == 1) return a[0] * b[0];
  else if constexpr (DIM == 2) return fma(a[DIR], b[DIR], rmul(a[1 - DIR], b[1 - DIR]));
  else
    return fma(a[DIR], b[DIR],
               rmul(a[Minor<DIR>::m1], b[Minor<DIR>::m1]) +
                   rmul(a[Minor<DIR>::m2], b[Minor<DIR>::m2]));
}

// Its flux from prime states (Density, Pressure, VelocityX..): the upwind side's
// conserved quantities alone.
template <int DIM, int DIR>
__device__ __forceinline__ void hllc_flux_primes(Eos const &e, HllcUpwind const &h,
                                                 double const (&pm)[DIM + 2],
                                                 double const (&pp)[DIM + 2],
                                                 double (&flux)[DIM + 2]) {
  flux[MASS] = h.rho * h.k;
  double v[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    v[d] = h.right ? pp[VELX + d] : pm[VELX + d];
    flux[MOMX + d] = d == DIR ? fma(h.rho, h.g, h.p) : v[d] * flux[MASS];
  }
  double const q = axis_dot<DIM, DIR>(v, v);
  double const E = fma(0.5 * h.rho, q, (h.p + e.gamma * e.B) * inv(e.gamma - 1.0));
  flux[ENERGY] = fma(E, h.k, h.pe);
}

// CalculateSignalSpeed, Einfeldt (hll_signal_speed_calculator.h:77-101) and
// HllcRiemannSolver::SolveRiemannProblemImplementation (hllc_riemann_solver.h:52-198)
// one_rl, one_rr: 1/density of the two states as returned by inv()
// As the reference writes it: the strict build's form.
template <int DIM, int DIR, typename T>
__device__ __forceinline__ void hllc_ordered(Eos const &e, T const (&cl)[DIM + 2],
                                             T const (&cr)[DIM + 2], T pres_l, T pres_r, T vel_l,
                                             T vel_r, T one_rl, T one_rr, T (&flux)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  T const c_l = eos_speed_of_sound<T>(e, cl[MASS], pres_l, one_rl);
  T const c_r = eos_speed_of_sound<T>(e, cr[MASS], pres_r, one_rr);
  T const srl = tsqrt(cl[MASS]);
  T const srr = tsqrt(cr[MASS]);
  T const rho_div = quot(T(1), srl + srr);
  T const u_roe = ((vel_l * srl) + (vel_r * srr)) * rho_div;
  T const c_e = tsqrt(((c_l * c_l * srl) + (c_r * c_r * srr)) * rho_div +
                     (T(0.5) * srl * srr * rho_div * rho_div) * (vel_r - vel_l) * (vel_r - vel_l));
  T const sls = dmin(u_roe - c_e, vel_l - c_l);
  T const srs = dmax(u_roe + c_e, vel_r + c_r);
  T const s_star = quot((pres_r - pres_l) + (cl[mP] * (sls - vel_l) - cr[mP] * (srs - vel_r)),
                        cl[MASS] * (sls - vel_l) - cr[MASS] * (srs - vel_r));
  T const sl = dmin(sls, T(0));
  T const sr = dmax(srs, T(0));
  T const chi_l = quot(sls - vel_l, sls - s_star);
  T const chi_r = quot(srs - vel_r, srs - s_star);
  T const rchi_l = cl[MASS] * chi_l, rchi_r = cr[MASS] * chi_r;
  T const sg = T((T(0) < s_star) - (s_star < T(0)));
  T const wl = T(0.5) * (T(1) + sg), wr = T(0.5) * (T(1) - sg);
  // mass
  {
    T const fsl = cl[mP] + (sl * (rchi_l - cl[MASS]));
    T const fsr = cr[mP] + (sr * (rchi_r - cr[MASS]));
    flux[MASS] = wl * fsl + wr * fsr;
  }
  // principal momentum
  {
    T const fl = ((cl[mP] * cl[mP]) * one_rl) + pres_l;
    T const fr = ((cr[mP] * cr[mP]) * one_rr) + pres_r;
    T const fsl = fl + (sl * (rchi_l * s_star - cl[mP]));
    T const fsr = fr + (sr * (rchi_r * s_star - cr[mP]));
    flux[mP] = wl * fsl + wr * fsr;
  }
  // energy (the star-state pressure term uses the clamped speeds, :131-144)
  {
    T const el = rchi_l * (cl[ENERGY] * one_rl +
                           (s_star - vel_l) * (s_star + quot(pres_l, cl[MASS] * (sl - vel_l))));
    T const er = rchi_r * (cr[ENERGY] * one_rr +
                           (s_star - vel_r) * (s_star + quot(pres_r, cr[MASS] * (sr - vel_r))));
    T const fl = vel_l * (cl[ENERGY] + pres_l);
    T const fr = vel_r * (cr[ENERGY] + pres_r);
    T const fsl = fl + (sl * (el - cl[ENERGY]));
    T const fsr = fr + (sr * (er - cr[ENERGY]));
    flux[ENERGY] = wl * fsl + wr * fsr;
  }
  // minor momenta
#pragma unroll
  for (int d = 0; d < DIM - 1; ++d) {
    int const mm = MOMX + (d == 0 ? Minor<DIR>::m1 : Minor<DIR>::m2);
    T const fsl = vel_l * cl[mm] + (sl * (chi_l * cl[mm] - cl[mm]));
    T const fsr = vel_r * cr[mm] + (sr * (chi_r * cr[mm] - cr[mm]));
    flux[mm] = wl * fsl + wr * fsr;
  }
}

template <int DIM, int DIR, typename T>
__device__ __forceinline__ void hllc(Eos const &e, T const (&cl)[DIM + 2], T const (&cr)[DIM + 2],
                                     T pres_l, T pres_r, T vel_l, T vel_r, T one_rl, T one_rr,
                                     T (&flux)[DIM + 2]) {
  if constexpr (ALP_FAST)
    hllc_flux<DIM, DIR>(hllc_upwind(e, cl[MASS], cr[MASS], pres_l, pres_r, vel_l, vel_r, one_rl,
                                    one_rr),
                        cl, cr, flux);
  else
    hllc_ordered<DIM, DIR, T>(e, cl, cr, pres_l, pres_r, vel_l, vel_r, one_rl, one_rr, flux);
}

// hllc_upwind of the FP32-flux form: wave speeds, the contact speed and the
// increments against the upwind state's physical flux in float, that flux and
// the sums in double. Uses chi - 1 = (S* - v) / (S - S*), so no increment is
// formed by cancellation.
__device__ __forceinline__ HllcUpwind hllc_upwind_mixed(Eos const &e, double rl, double rr,
                                                        double pl, double pr, double vl, double vr,
                                                        double one_l, double one_r) {
  float const ccl = float(eos_cc(e, rl, pl, one_l)), ccr = float(eos_cc(e, rr, pr, one_r));
  float const frl = float(rl), frr = float(rr), ul = float(vl), ur = float(vr);
  float const srl = tsqrt(frl), srr = tsqrt(frr);
  float const one = inv(srl + srr);
  float const wl = srl * one, wr = srr * one;
  float const du = float(vl - vr);
  float const u = fmaf(wl, du, ur);
  float const ce = tsqrt(fmaf(0.5f * (wl * wr), du * du, fmaf(wl, ccl - ccr, ccr)));
  float const sl = dmin(u - ce, ul - tsqrt(ccl)), sr = dmax(u + ce, ur + tsqrt(ccr));
  float const al = frl * (sl - ul), ar = frr * (sr - ur);
  float const ss = fmaf(ul, al, fmaf(-ur, ar, float(pr - pl))) * inv(al - ar);
  HllcUpwind h;
  h.right = ss < 0.0f;
  h.rho = h.right ? rr : rl;
  h.p = h.right ? pr : pl;
  double const v = h.right ? vr : vl;
  float const fu = h.right ? ur : ul, s = h.right ? sr : sl;
  float const sc = h.right ? dmax(sr, 0.0f) : dmin(sl, 0.0f);
  float const dss = ss - fu;
  float const dchi = dss * inv(s - ss);
  h.k = v + double(sc * dchi);
  h.g = fma(v, v, double(sc * fmaf(dchi, ss, dss)));
  h.pe = fma(v, h.p, double((sc * ((1.0f + dchi) * dss)) *
                            fmaf(h.right ? frr : frl, ss, float(h.p) * inv(sc - fu))));
  return h;
}

// HLLC for the strict build's FP32-flux form (same approximate Riemann solver as hllc():
// Einfeldt speeds, Toro star states, the reference's clamped-speed energy
// term). Wave speeds, the contact speed and the star-state increments
// q* - q are computed in float; the physical fluxes F(q) that carry the mean
// and their sum F + S (q* - q) are evaluated in double. Uses
// chi - 1 = (S* - u) / (S - S*), so no increment is formed by cancellation.
template <int DIM, int DIR>
__device__ __forceinline__ void hllc_mixed(Eos const &e, double const (&cl)[DIM + 2],
                                           double const (&cr)[DIM + 2], double pres_l,
                                           double pres_r, double vel_l, double vel_r,
                                           double one_rl, double one_rr, double (&flux)[DIM + 2]) {
  constexpr int mP = MOMX + DIR;
  float const g = float(e.gamma), B = float(e.B);
  float const rl = float(cl[MASS]), rr = float(cr[MASS]);
  float const ul = float(vel_l), ur = float(vel_r);
  float const cc_l = g * (float(pres_l) + B) * float(one_rl);
  float const cc_r = g * (float(pres_r) + B) * float(one_rr);
  float const c_l = tsqrt(cc_l), c_r = tsqrt(cc_r);
  float const srl = tsqrt(rl), srr = tsqrt(rr);
  float const rho_div = __fdividef(1.0f, srl + srr);
  float const u_roe = (ul * srl + ur * srr) * rho_div;
  float const c_e = tsqrt((cc_l * srl + cc_r * srr) * rho_div +
                          (0.5f * srl * srr * rho_div * rho_div) * (ur - ul) * (ur - ul));
  float const sls = dmin(u_roe - c_e, ul - c_l);
  float const srs = dmax(u_roe + c_e, ur + c_r);
  float const dpr = float(pres_r - pres_l);
  float const s_star = __fdividef(dpr + (rl * ul * (sls - ul) - rr * ur * (srs - ur)),
                                  rl * (sls - ul) - rr * (srs - ur));
  float const sl = dmin(sls, 0.0f), sr = dmax(srs, 0.0f);
  float const dchi_l = __fdividef(s_star - ul, sls - s_star);  // chi_l - 1
  float const dchi_r = __fdividef(s_star - ur, srs - s_star);
  float const chi_l = 1.0f + dchi_l, chi_r = 1.0f + dchi_r;
  float const sg = float((0.0f < s_star) - (s_star < 0.0f));
  double const wl = 0.5 * (1.0 + sg), wr = 0.5 * (1.0 - sg);
  // star-state increments q* - q
  float dq_l[DIM + 2], dq_r[DIM + 2];
  dq_l[MASS] = rl * dchi_l;
  dq_r[MASS] = rr * dchi_r;
  dq_l[mP] = rl * ((s_star - ul) + dchi_l * s_star);
  dq_r[mP] = rr * ((s_star - ur) + dchi_r * s_star);
  dq_l[ENERGY] = float(cl[ENERGY]) * dchi_l +
                 rl * chi_l * (s_star - ul) *
                     (s_star + __fdividef(float(pres_l), rl * (sl - ul)));
  dq_r[ENERGY] = float(cr[ENERGY]) * dchi_r +
                 rr * chi_r * (s_star - ur) *
                     (s_star + __fdividef(float(pres_r), rr * (sr - ur)));
#pragma unroll
  for (int d = 0; d < DIM - 1; ++d) {
    int const mm = MOMX + (d == 0 ? Minor<DIR>::m1 : Minor<DIR>::m2);
    dq_l[mm] = dchi_l * float(cl[mm]);
    dq_r[mm] = dchi_r * float(cr[mm]);
  }
  // physical fluxes in double
  double fl[DIM + 2], fr[DIM + 2];
  fl[MASS] = cl[mP];
  fr[MASS] = cr[mP];
  fl[mP] = cl[mP] * cl[mP] * one_rl + pres_l;
  fr[mP] = cr[mP] * cr[mP] * one_rr + pres_r;
  fl[ENERGY] = vel_l * (cl[ENERGY] + pres_l);
  fr[ENERGY] = vel_r * (cr[ENERGY] + pres_r);
#pragma unroll
  for (int d = 0; d < DIM - 1; ++d) {
    int const mm = MOMX + (d == 0 ? Minor<DIR>::m1 : Minor<DIR>::m2);
    fl[mm] = vel_l * cl[mm];
    fr[mm] = vel_r * cr[mm];
  }
#pragma unroll
  for (int n = 0; n < DIM + 2; ++n)
    flux[n] = wl * (fl[n] + double(sl * dq_l[n])) + wr * (fr[n] + double(sr * dq_r[n]));
}

}  // namespace alp
