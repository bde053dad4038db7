// Block kernels beside the face fluxes (face_flux.cu, sweep.cu, ext_*.cu, pencil.cu):
// flux divergence, stage updates, halo fill, prime states, signal speed, time-step
// and commit records, initial conditions, interior copies. Data stays in the
// reference's block layout (layout.cuh).
#include <cfloat>
#include <cstdio>

#include "face_kernels.cuh"

namespace alp {

namespace {

// ---------------------------------------------------------------------------
// divergence, stage update
// ---------------------------------------------------------------------------

// Right-hand side of every cell of the blocks: zero in the halos
// (space_solver.cpp:58-70), the flux divergence inside. A CTA takes
// kDivergenceCells consecutive cells of one block and the threads walk its
// fields, so that the writes are the only pass over the buffer and a call of a
// few blocks still fills the chip.
// 125 blocks: 68 us with one CTA per block zeroing, then filling it.
constexpr int kDivergenceCells = 512;

template <int DIM>
__global__ void __launch_bounds__(256)
divergence_kernel(int const *__restrict__ work, BlockMeta const *__restrict__ meta, BlockMeta def,
                  double const *__restrict__ F, long long stride, long long dstride,
                  double *__restrict__ rhs) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  double *rb = rhs + (size_t)slot * G::BLOCK_DOUBLES;
  BlockMeta const bm = meta ? meta[slot] : def;
  double const ocs = inv(bm.cell_size);
  double const *Fb = F + (long long)item * stride;
  int const end = min(G::CELLS, (int)(blockIdx.y + 1) * kDivergenceCells);
  for (int x = blockIdx.y * kDivergenceCells + threadIdx.x; x < end; x += blockDim.x) {
    int const k = x % G::TCZ - G::fic(2), j = (x / G::TCZ) % G::TCY - G::fic(1);
    int const i = x / (G::TCZ * G::TCY) - G::fic(0);
    bool const in = (unsigned)i < (unsigned)G::ICX && (unsigned)j < (unsigned)G::ICY &&
                    (unsigned)k < (unsigned)G::ICZ;
#pragma unroll
    for (int f = 0; f < G::NE; ++f) {
      double v = 0.0;
      if (in) {
        double const *fx = Fb + f * G::FACES;
        v = 0.0 + divergence<DIM>(fx, fx + dstride, fx + 2 * dstride, i, j, k, ocs);
      }
      rb[f * G::CELLS + x] = v;
    }
  }
}

// Uin: stage input, U0: state at the start of the step, Uout: stage output.
// Uout may alias U0 (each cell is read and written by the same thread) but
// not Uin, whose cells other blocks' stencils read during the stage.
template <int DIM>
__global__ void __launch_bounds__(256)
stage_update_kernel(double const *Uin, double const *U0, double *Uout,
                    int const *__restrict__ work, BlockMeta const *__restrict__ meta, BlockMeta def,
                    double const *__restrict__ F, long long stride, long long dstride, int stage,
                    CaseState const *__restrict__ cases, double dt_all) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  double const dt = cases ? cases[bm.case_id].dt : dt_all;
  if (!(dt > 0.0)) return;
  int const t = blockIdx.y * blockDim.x + threadIdx.x;
  if (t >= G::INTERIOR) return;
  stage_update_cell<DIM>(Uin, U0, Uout, F + (long long)item * stride, dstride, slot, t,
                         inv(bm.cell_size), rk_stage(stage, dt));
}

// Stage update from a reference-layout right-hand-side buffer.
template <int DIM>
__global__ void __launch_bounds__(256)
rk_stage_rhs_kernel(double *__restrict__ U, double *__restrict__ U0,
                    double const *__restrict__ rhs, int stage, double dt) {
  using G = Geo<DIM>;
  int const slot = blockIdx.x;
  int const t = blockIdx.y * blockDim.x + threadIdx.x;
  if (t >= G::INTERIOR) return;
  int i, j, k;
  interior_coords<DIM>(t, i, j, k);
  int const c = G::cell(i + G::fic(0), j + G::fic(1), k + G::fic(2));
  RkStage const rk = rk_stage(stage, dt);
  size_t const base = (size_t)slot * G::BLOCK_DOUBLES + c;
  // every load before the first store, so that a thread's loads are in flight
  // together
  double u[G::NE], u0[G::NE], r[G::NE];
#pragma unroll
  for (int f = 0; f < G::NE; ++f) {
    size_t const x = base + (size_t)f * G::CELLS;
    u[f] = U[x];
    u0[f] = rk.first ? 0.0 : U0[x];
    r[f] = rhs[x];
  }
#pragma unroll
  for (int f = 0; f < G::NE; ++f) {
    size_t const x = base + (size_t)f * G::CELLS;
    if (stage == 0) U0[x] = u[f];
    U[x] = rk_apply(rk, u[f], u0[f], r[f]);
  }
}

// ---------------------------------------------------------------------------
// halos
// ---------------------------------------------------------------------------

// Same-level halo regions (communication_types.h:45-132): for direction offset
// o = +1 the halo [HS+IC, TC) takes the neighbour's [HS, 2HS); o = -1 the halo
// [0, HS) takes the neighbour's [IC, IC+HS); o = 0 spans the interior. A halo
// cell's offset follows from its coordinates, and its source is the cell 16
// further inside along the offset. A CTA fills the halo cells of one x plane of
// one block (3D; the whole block in 1D and 2D), all fields, in storage order,
// so the stores are whole rows; halos of domain faces are left to
// zero_gradient_kernel. 125 blocks of 5 fields: 40 us with one CTA per region
// (26 of them, 4 cells wide along z) and the extents divided at run time.
template <int DIM>
__global__ void __launch_bounds__(256)
halo_region_kernel(double *__restrict__ U, int const *__restrict__ work,
                   int const *__restrict__ nbr26, BlockMeta const *__restrict__ meta,
                   CaseState const *__restrict__ cases, int faces_only, int nfields) {
  using G = Geo<DIM>;
  constexpr int PLANES = DIM == 3 ? TC : 1;
  // cells of an interior 3D plane that are halo: 8 whole rows, 8 cells of the others
  constexpr int ROWS = 2 * HS * TC, RING = ROWS + 2 * HS * IC;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  if (cases && meta && !(cases[meta[slot].case_id].dt > 0.0)) return;
  __shared__ int nb[27];
  if (threadIdx.x < 27)
    nb[threadIdx.x] = threadIdx.x == 13 ? -1
                                        : nbr26[(size_t)slot * 26 + threadIdx.x - (threadIdx.x > 13)];
  __syncthreads();
  int const plane = PLANES > 1 ? blockIdx.y : 0;
  bool const ring = PLANES > 1 && plane >= HS && plane < HS + IC;
  int const count = ring ? RING : G::CELLS / PLANES;
  double *dst = U + (size_t)slot * nfields * G::CELLS;
  for (int t = threadIdx.x; t < count; t += blockDim.x) {
    int c[3];
    if (ring) {
      c[0] = plane;
      if (t < ROWS) {
        int const r = t / TC;
        c[1] = r < HS ? r : r + IC;
        c[2] = t - r * TC;
      } else {
        int const r = (t - ROWS) / (2 * HS), q = (t - ROWS) % (2 * HS);
        c[1] = HS + r;
        c[2] = q < HS ? q : q + IC;
      }
    } else {
      c[2] = t % G::TCZ;
      c[1] = (t / G::TCZ) % G::TCY;
      c[0] = PLANES > 1 ? plane : t / (G::TCZ * G::TCY);
    }
    int o = 0, nonzero = 0, src[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int const off = d >= DIM ? 0 : (c[d] < HS ? -1 : (c[d] >= HS + IC ? 1 : 0));
      o = 3 * o + off + 1;
      nonzero += off != 0;
      src[d] = c[d] - IC * off;
    }
    int const n = nb[o];
    if (n < 0 || (faces_only && nonzero != 1)) continue;  // interior, domain face, or not asked for
    double const *sb = U + (size_t)n * nfields * G::CELLS + G::cell(src[0], src[1], src[2]);
    double *db = dst + G::cell(c[0], c[1], c[2]);
    int f = 0;
    for (; f + 5 <= nfields; f += 5) {  // loads first: the stores may alias them
      double v[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) v[q] = sb[(f + q) * G::CELLS];
#pragma unroll
      for (int q = 0; q < 5; ++q) db[(f + q) * G::CELLS] = v[q];
    }
    for (; f < nfields; ++f) db[f * G::CELLS] = sb[f * G::CELLS];
  }
}

// Zero-gradient halos of domain faces (boundary_constants.h:103-160, 211-252):
// the halo takes the value of the first / last interior plane. With
// faces_only the copy covers the interior extent of the face, otherwise the
// reference's full TC x TC slab. The faces of one block are applied one after
// the other in x, y, z order (CommunicationManager::NeighborsOfNode lists
// domain sides East, West, North, South, Top, Bottom), which fixes the values
// the overlapping slabs leave in edge and corner halos.
template <int DIM>
__global__ void __launch_bounds__(256)
zero_gradient_kernel(double *__restrict__ U, int const *__restrict__ work,
                     int const *__restrict__ nbr26, BlockMeta const *__restrict__ meta,
                     CaseState const *__restrict__ cases, int faces_only, int nfields) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  if (cases && meta && !(cases[meta[slot].case_id].dt > 0.0)) return;
  double *b = U + (size_t)slot * nfields * G::CELLS;
  for (int face = 0; face < 2 * DIM; ++face) {
    int const dir = face / 2, high = face & 1;
    int off[3] = {0, 0, 0};
    off[dir] = high ? 1 : -1;
    int const o = (off[0] + 1) * 9 + (off[1] + 1) * 3 + (off[2] + 1);
    int const nface = nbr26[(size_t)slot * 26 + (o < 13 ? o : o - 1)];
    if (nface >= 0) continue;
    bool const sym = nface == -2;  // symmetry wall: mirror, normal momentum negated
    int lo[3], ext[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = faces_only ? G::fic(d) : 0;
      ext[d] = faces_only ? G::ic(d) : G::tc(d);
    }
    lo[dir] = high ? HS + IC : 0;
    ext[dir] = HS;
    int const plane = high ? HS + IC - 1 : HS;
    int const mirror = high ? 2 * (HS + IC) - 1 : 2 * HS - 1;
    int const cells = ext[0] * ext[1] * ext[2];
    for (int x = threadIdx.x; x < cells * nfields; x += blockDim.x) {
      int const f = x / cells;
      int const r = x - f * cells;
      int c[3];
      c[2] = lo[2] + r % ext[2];
      c[1] = lo[1] + (r / ext[2]) % ext[1];
      c[0] = lo[0] + r / (ext[2] * ext[1]);
      int s[3] = {c[0], c[1], c[2]};
      s[dir] = sym ? mirror - c[dir] : plane;
      double const v = b[f * G::CELLS + G::cell(s[0], s[1], s[2])];
      // the momentum (or, for prime states, the velocity) normal to the wall is field 2 + dir
      b[f * G::CELLS + G::cell(c[0], c[1], c[2])] = (sym && f == 2 + dir) ? -1.0 * v : v;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// prime states, signal speed, dt
// ---------------------------------------------------------------------------

template <int DIM>
__global__ void __launch_bounds__(256)
prime_states_kernel(double const *__restrict__ U, int const *__restrict__ work,
                    BlockMeta const *__restrict__ meta, BlockMeta def, double *__restrict__ P) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  Eos const eos{bm.gamma, bm.B, bm.safe};
  double const *ub = U + (size_t)slot * G::BLOCK_DOUBLES;
  double *pb = P + (size_t)slot * G::BLOCK_DOUBLES;
  for (int x = blockIdx.y * blockDim.x + threadIdx.x; x < G::CELLS; x += gridDim.y * blockDim.x) {
    double c[G::NE];
#pragma unroll
    for (int f = 0; f < G::NE; ++f) c[f] = ub[f * G::CELLS + x];
    double const one_density = inv(c[MASS]);
    pb[RHO * G::CELLS + x] = c[MASS];
#pragma unroll
    for (int d = 0; d < DIM; ++d) pb[(VELX + d) * G::CELLS + x] = c[MOMX + d] * one_density;
    pb[PRES * G::CELLS + x] = eos_pressure<DIM>(eos, c[MASS], c[MOMX],
                                                DIM > 1 ? c[MOMX + (DIM > 1)] : 0.0,
                                                DIM > 2 ? c[MOMX + 2 * (DIM > 2)] : 0.0, c[ENERGY],
                                                one_density);
  }
}

// CTAs per block of the signal speed: four in 3D, four cells to a thread. 64
// blocks took 16.6 us with one CTA per block (a chain of 16 loads and square
// roots per thread).
__host__ __device__ constexpr int signal_parts(int dim) { return dim == 3 ? 4 : 1; }

// Signal speed of ComputeTimestepSize (modular_algorithm_assembler.cpp:1840-1870):
// max over interior cells of ConsistencyManagedSum(|u_d| + c).
template <int DIM>
__global__ void __launch_bounds__(256)
signal_speed_kernel(double const *__restrict__ U, int const *__restrict__ work,
                    BlockMeta const *__restrict__ meta, BlockMeta def, CaseState *cases,
                    unsigned long long *out) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  Eos const eos{bm.gamma, bm.B, bm.safe};
  double const *ub = U + (size_t)slot * G::BLOCK_DOUBLES;
  double smax = 0.0;
  int bad = 0;
  constexpr int PARTS = signal_parts(DIM);
  int const first = blockIdx.y * (G::INTERIOR / PARTS);
#pragma unroll 4
  for (int t = threadIdx.x; t < G::INTERIOR / PARTS; t += blockDim.x) {
    int i, j, k;
    interior_coords<DIM>(first + t, i, j, k);
    int const x = G::cell(i + G::fic(0), j + G::fic(1), k + G::fic(2));
    double c[G::NE];
#pragma unroll
    for (int f = 0; f < G::NE; ++f) c[f] = ub[f * G::CELLS + x];
    double const s = cell_signal_speed<DIM>(eos, c, bad);
    smax = dmax(smax, s);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0 && cases) atomicOr(&cases[bm.case_id].status, 1);
  // warp then CTA max (non-negative doubles order like their bit patterns)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) smax = dmax(smax, __shfl_xor_sync(0xffffffffu, smax, o));
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = smax;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) {
      unsigned long long *dst = cases ? &cases[bm.case_id].smax_bits : out;
      atomicMax(dst, (unsigned long long)__double_as_longlong(v));
    }
  }
}

// dt = CFL / (smax / dx_finest), clipped to the end time
// (modular_algorithm_assembler.cpp:1932, 1961-1982); 0 once t >= t_end or the
// step budget is spent, which makes every kernel skip the case.
// dt of every case from its smax (case_dt_finalize); dtflag, when given,
// marks each case's dt as ready for a tile-stage launch (its step 0).
__global__ void dt_finalize_kernel(CaseState *cases, int n, int *dtflag) {
  int const c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  case_dt_finalize(cases[c]);
  if (dtflag) dtflag[c] = 1;
}

__global__ void step_commit_kernel(CaseState *cases, int n) {
  int const c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  case_commit(cases[c]);
}

}  // namespace

// Initial conditions evaluated on the device for a regular block grid whose
// blocks occupy consecutive slots from `first` in C order (x slowest). Cell
// centres are ((block index * 16 + i + 0.5) * cell_size, ...). Prime states
// are converted with PrimeStatesToConservatives (prime_state_handler.h:195-275).
// Every cell of the block (halos too) is written; halos are refreshed before
// they are read.
template <int DIM>
__global__ void __launch_bounds__(256)
initial_condition_kernel(double *__restrict__ U, int first, int nbx, int nby, int nbz,
                         double cell_size, double gamma, double B, int type,
                         IcParams params) {
  using G = Geo<DIM>;
  int const b = blockIdx.x;
  int const bx = b / (nby * nbz), by = (b / nbz) % nby, bz = b % nbz;
  double *ub = U + (size_t)(first + b) * G::BLOCK_DOUBLES;
  Eos const eos{gamma, B, 0};
  for (int x = threadIdx.x; x < G::CELLS; x += blockDim.x) {
    int const k = x % G::TCZ, j = (x / G::TCZ) % G::TCY, i = x / (G::TCZ * G::TCY);
    double pos[3] = {0.0, 0.0, 0.0};
    pos[0] = (bx * IC + i - HS + 0.5) * cell_size;
    if (DIM > 1) pos[1] = (by * IC + j - HS + 0.5) * cell_size;
    if (DIM > 2) pos[2] = (bz * IC + k - HS + 0.5) * cell_size;
    double const *q = params.v;
    double rho, p, vel[3] = {0.0, 0.0, 0.0};
    if (type == IC_QUADRANTS) {
      // q: x0, y0, then (rho, u, v, p) for quadrants (x<x0,y<y0), (x>=x0,y<y0),
      // (x<x0,y>=y0), (x>=x0,y>=y0)
      int const quad = (pos[0] >= q[0] ? 1 : 0) + (pos[1] >= q[1] ? 2 : 0);
      double const *s = q + 2 + 4 * quad;
      rho = s[0];
      vel[0] = s[1];
      vel[1] = s[2];
      p = s[3];
    } else {
      // IC_BLAST: q: centre (3), radius, (rho, p) inside, (rho, p) outside
      double r2 = 0.0;
      for (int d = 0; d < DIM; ++d) r2 += (pos[d] - q[d]) * (pos[d] - q[d]);
      bool const in = r2 < q[3] * q[3];
      rho = in ? q[4] : q[6];
      p = in ? q[5] : q[7];
    }
    double c[G::NE];
    c[MASS] = rho;
#pragma unroll
    for (int d = 0; d < DIM; ++d) c[MOMX + d] = vel[d] * rho;
    c[ENERGY] = eos_energy<DIM, double>(eos, rho, vel[0], vel[1], vel[2], p);
#pragma unroll
    for (int f = 0; f < G::NE; ++f) ub[f * G::CELLS + x] = c[f];
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

namespace {

int interior_of(int dim) { return dim == 3 ? 4096 : (dim == 2 ? 256 : 16); }

}  // namespace

cudaError_t launch_divergence(Launch const &L, double const *F, long long stride,
                              long long dstride, double *rhs) {
  if (L.nwork <= 0) return cudaSuccess;
  int const cells = 24 * (L.dim > 1 ? 24 : 1) * (L.dim > 2 ? 24 : 1);
  dim3 grid(L.nwork, (cells + kDivergenceCells - 1) / kDivergenceCells);
  switch (L.dim) {
    case 1: divergence_kernel<1><<<grid, 256, 0, L.stream>>>(L.work, L.meta, L.def, F, stride, dstride, rhs); break;
    case 2: divergence_kernel<2><<<grid, 256, 0, L.stream>>>(L.work, L.meta, L.def, F, stride, dstride, rhs); break;
    case 3: divergence_kernel<3><<<grid, 256, 0, L.stream>>>(L.work, L.meta, L.def, F, stride, dstride, rhs); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_stage_update(Launch const &L, double const *U0, double *Uout, double const *F,
                                long long stride, long long dstride, int stage,
                                CaseState const *cases, double dt) {
  if (L.nwork <= 0) return cudaSuccess;
  if (stage < 0 || stage > 4) return cudaErrorInvalidValue;
  int const threads = 256;
  dim3 grid(L.nwork, (interior_of(L.dim) + threads - 1) / threads);
  switch (L.dim) {
    case 1: stage_update_kernel<1><<<grid, threads, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, L.def, F, stride, dstride, stage, cases, dt); break;
    case 2: stage_update_kernel<2><<<grid, threads, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, L.def, F, stride, dstride, stage, cases, dt); break;
    case 3: stage_update_kernel<3><<<grid, threads, 0, L.stream>>>(L.U, U0, Uout, L.work, L.meta, L.def, F, stride, dstride, stage, cases, dt); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_rk_stage_rhs(int dim, double *U, double *U0, double const *rhs, int nb,
                                int stage, double dt, cudaStream_t stream) {
  if (nb <= 0) return cudaSuccess;
  if (stage < 0 || stage > 2) return cudaErrorInvalidValue;
  dim3 grid(nb, (interior_of(dim) + 255) / 256);
  switch (dim) {
    case 1: rk_stage_rhs_kernel<1><<<grid, 256, 0, stream>>>(U, U0, rhs, stage, dt); break;
    case 2: rk_stage_rhs_kernel<2><<<grid, 256, 0, stream>>>(U, U0, rhs, stage, dt); break;
    case 3: rk_stage_rhs_kernel<3><<<grid, 256, 0, stream>>>(U, U0, rhs, stage, dt); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_halo(Launch const &L, int const *nbr26, bool faces_only, int nfields,
                        CaseState const *cases) {
  if (L.nwork <= 0) return cudaSuccess;
  dim3 g1(L.nwork, L.dim == 3 ? TC : 1), g2(L.nwork);
  int const fo = faces_only ? 1 : 0;
  switch (L.dim) {
    case 1:
      halo_region_kernel<1><<<g1, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      zero_gradient_kernel<1><<<g2, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      break;
    case 2:
      halo_region_kernel<2><<<g1, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      zero_gradient_kernel<2><<<g2, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      break;
    case 3:
      halo_region_kernel<3><<<g1, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      zero_gradient_kernel<3><<<g2, 256, 0, L.stream>>>(L.U, L.work, nbr26, L.meta, cases, fo, nfields);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_prime_states(Launch const &L, double *P) {
  if (L.nwork <= 0) return cudaSuccess;
  dim3 grid(L.nwork, 8);
  switch (L.dim) {
    case 1: prime_states_kernel<1><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, P); break;
    case 2: prime_states_kernel<2><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, P); break;
    case 3: prime_states_kernel<3><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, P); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_signal_speed(Launch const &L, CaseState *cases, unsigned long long *out) {
  if (L.nwork <= 0) return cudaSuccess;
  dim3 grid(L.nwork, signal_parts(L.dim));
  switch (L.dim) {
    case 1: signal_speed_kernel<1><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, cases, out); break;
    case 2: signal_speed_kernel<2><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, cases, out); break;
    case 3: signal_speed_kernel<3><<<grid, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, cases, out); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_initial_condition(int dim, double *U, int first, int const nblocks[3],
                                     double cell_size, double gamma, double B, int type,
                                     IcParams const &params, cudaStream_t stream) {
  int const nb = nblocks[0] * nblocks[1] * nblocks[2];
  if (nb <= 0) return cudaSuccess;
  if (type != IC_QUADRANTS && type != IC_BLAST) return cudaErrorInvalidValue;
  switch (dim) {
    case 1: initial_condition_kernel<1><<<nb, 256, 0, stream>>>(U, first, nblocks[0], nblocks[1], nblocks[2], cell_size, gamma, B, type, params); break;
    case 2: initial_condition_kernel<2><<<nb, 256, 0, stream>>>(U, first, nblocks[0], nblocks[1], nblocks[2], cell_size, gamma, B, type, params); break;
    case 3: initial_condition_kernel<3><<<nb, 256, 0, stream>>>(U, first, nblocks[0], nblocks[1], nblocks[2], cell_size, gamma, B, type, params); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_dt_finalize(CaseState *cases, int n, cudaStream_t stream, int *dtflag) {
  if (n <= 0) return cudaSuccess;
  dt_finalize_kernel<<<(n + 127) / 128, 128, 0, stream>>>(cases, n, dtflag);
  return cudaGetLastError();
}

cudaError_t launch_step_commit(CaseState *cases, int n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  step_commit_kernel<<<(n + 127) / 128, 128, 0, stream>>>(cases, n);
  return cudaGetLastError();
}

namespace {
__device__ unsigned long long g_glf_stateless[4];

__device__ __forceinline__ double max_keep(double m, double v) { return (m < v) ? v : m; }

// One CTA per block: the block's maxima of |u - c|, |u|, |u + c| (x velocity,
// interior cells with positive density; std::max keeps the running maximum
// against a NaN as the reference's does), then one atomicMax per value on
// its case's slot (bit patterns of non-negative doubles order like the values).
template <int DIM>
__global__ void __launch_bounds__(256)
glf_maxima_kernel(double const *__restrict__ U, int const *__restrict__ work,
                  BlockMeta const *__restrict__ meta, BlockMeta def,
                  unsigned long long *__restrict__ glf) {
  using G = Geo<DIM>;
  int const item = blockIdx.x;
  int const slot = slot_of(work, item);
  BlockMeta const bm = meta ? meta[slot] : def;
  Eos const eos{bm.gamma, bm.B, bm.safe};
  double const *ub = U + (size_t)slot * G::BLOCK_DOUBLES;
  double m[3] = {0.0, 0.0, 0.0};
  for (int c = threadIdx.x; c < G::INTERIOR; c += blockDim.x) {
    int const k = c % G::ICZ, j = (c / G::ICZ) % G::ICY, i = c / (G::ICZ * G::ICY);
    int const x = ((i + HS) * G::TCY + (j + (DIM > 1 ? HS : 0))) * G::TCZ + (k + (DIM > 2 ? HS : 0));
    double cons[G::NE];
#pragma unroll
    for (int f = 0; f < G::NE; ++f) cons[f] = ub[f * G::CELLS + x];
    auto const pr = cell_prims<DIM, 0>(eos, cons);
    if (!(pr.rho > 0.0)) continue;
    double const cs = eos_speed_of_sound<double>(eos, pr.rho, pr.p, pr.one_rho);
    m[0] = max_keep(m[0], fabs(pr.up - cs));
    m[1] = max_keep(m[1], fabs(pr.up));
    m[2] = max_keep(m[2], fabs(pr.up + cs));
  }
  __shared__ double red[3][8];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double v = m[q];
    for (int o = 16; o > 0; o >>= 1) v = max_keep(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v = max_keep(v, red[threadIdx.x][w]);
    atomicMax(&glf[4 * bm.case_id + threadIdx.x], (unsigned long long)__double_as_longlong(v));
  }
}
}  // namespace

cudaError_t launch_glf_maxima(Launch const &L, unsigned long long *glf, int ncases) {
  if (ncases <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(glf, 0, sizeof(unsigned long long) * 4 * ncases, L.stream);
  if (e != cudaSuccess || L.nwork <= 0) return e;
  switch (L.dim) {
    case 1: glf_maxima_kernel<1><<<L.nwork, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, glf); break;
    case 2: glf_maxima_kernel<2><<<L.nwork, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, glf); break;
    default: glf_maxima_kernel<3><<<L.nwork, 256, 0, L.stream>>>(L.U, L.work, L.meta, L.def, glf); break;
  }
  return cudaGetLastError();
}

// The address is looked up on every call (a symbol lookup in the loaded
// module): after cudaDeviceReset the module loads again, possibly at another
// address, so an address kept from an earlier call could be stale.
unsigned long long *glf_stateless_slot() {
  void *addr = nullptr;
  if (cudaGetSymbolAddress(&addr, g_glf_stateless) != cudaSuccess) return nullptr;
  return static_cast<unsigned long long *>(addr);
}

namespace {
// packed [b][field][ICX][ICY][ICZ] <-> the interiors of pool blocks first + b
// (one thread per cell; consecutive threads take consecutive z cells).
template <int DIM>
__global__ void interior_copy_kernel(double *U, int first, int nb, double *P, bool to_pool) {
  using G = Geo<DIM>;
  long long const n = (long long)nb * G::NE * G::INTERIOR;
  for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n;
       x += (long long)gridDim.x * blockDim.x) {
    int const c = int(x % G::INTERIOR);
    long long const bf = x / G::INTERIOR;  // b * NE + field
    int const k = c % G::ICZ, j = (c / G::ICZ) % G::ICY, i = c / (G::ICZ * G::ICY);
    long long const u = ((long long)first * G::NE + bf) * G::CELLS +
                        G::cell(i + G::fic(0), j + G::fic(1), k + G::fic(2));
    if (to_pool) U[u] = P[x];
    else P[x] = U[u];
  }
}
}  // namespace

cudaError_t launch_interior_copy(int dim, double *U, int first, int nb, double *packed,
                                 bool to_pool, cudaStream_t stream) {
  if (nb <= 0) return cudaSuccess;
  int const grid = 148 * 8, threads = 256;
  switch (dim) {
    case 1: interior_copy_kernel<1><<<grid, threads, 0, stream>>>(U, first, nb, packed, to_pool); break;
    case 2: interior_copy_kernel<2><<<grid, threads, 0, stream>>>(U, first, nb, packed, to_pool); break;
    default: interior_copy_kernel<3><<<grid, threads, 0, stream>>>(U, first, nb, packed, to_pool); break;
  }
  return cudaGetLastError();
}

}  // namespace alp
