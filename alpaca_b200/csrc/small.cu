// Whole steps of a small 1D or 2D work list in one launch of one thread-block
// cluster. With a few hundred to a few thousand faces a stage's work takes a few
// microseconds, less than the nine dependent launches of a step cost; here the
// phases of a step (signal speed, dt, per stage the face fluxes and the stage
// update) are separated by the cluster's hardware barrier instead, and one
// launch runs many steps. The CTAs of a cluster are scheduled together, so the
// barrier needs no bound. Cells and fluxes written by other CTAs are read
// through L2. The arithmetic is that of the launches it replaces (face_flux,
// stage_update_cell, cell_signal_speed, case_dt_finalize), so are the bits.
#include "face_kernels.cuh"

namespace alp {
namespace {

struct SmallArgs {
  double *in[3], *out[3];  // stage input and output pools
  double *U, *F;
  int const *work;
  int nwork;
  BlockMeta const *meta;
  int const *nbr26;
  CaseState *cases;
  int ncases, nsteps, nst, s0;
  bool commit;
  long long stride, dstride;
};

constexpr int kSmallThreads = 256;  // at most, per CTA
constexpr int kSmallCtas = 16;      // the largest cluster (beyond 8: opt-in)
constexpr int kSmallSteps = 256;  // steps per launch

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}

// Case c's record, read through L2 (other CTAs' atomics changed it).
__device__ __forceinline__ CaseState load_case(CaseState const *c) {
  static_assert(sizeof(CaseState) % 8 == 0, "");
  CaseState s;
  auto const *src = reinterpret_cast<unsigned long long const *>(c);
  auto *dst = reinterpret_cast<unsigned long long *>(&s);
#pragma unroll
  for (int k = 0; k < (int)(sizeof(CaseState) / 8); ++k) dst[k] = __ldcg(src + k);
  return s;
}

template <int DIM, int SCHEME, typename T>
__global__ void __launch_bounds__(kSmallThreads) small_steps_kernel(SmallArgs a) {
  using G = Geo<DIM>;
  constexpr int NE = G::NE, COUNT = FaceMap<DIM, 0>::COUNT;
  int const nth = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
  for (int step = 0; step < a.nsteps; ++step) {
    // signal speed: 16 consecutive cells belong to one block, hence to one case
    for (int x = tid; x < a.nwork * G::INTERIOR; x += nth) {
      int const item = x / G::INTERIOR;
      int const slot = a.work[item];
      BlockMeta const bm = a.meta[slot];
      int i, j, k, bad = 0;
      interior_coords<DIM>(x - item * G::INTERIOR, i, j, k);
      double const *u = a.U + (size_t)slot * G::BLOCK_DOUBLES +
                        G::cell(i + G::fic(0), j + G::fic(1), k + G::fic(2));
      double c[NE];
#pragma unroll
      for (int f = 0; f < NE; ++f) c[f] = __ldcg(u + f * G::CELLS);
      double s = cell_signal_speed<DIM>(Eos{bm.gamma, bm.B, bm.safe}, c, bad);
      s = dmax(0.0, s);  // signal_speed_kernel's running maximum starts at 0
      unsigned const half = 0xffffu << (threadIdx.x & 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s = dmax(s, __shfl_xor_sync(half, s, o));
      bool const any = __any_sync(half, bad);
      if ((threadIdx.x & 15) == 0) {
        atomicMax(&a.cases[bm.case_id].smax_bits, (unsigned long long)__double_as_longlong(s));
        if (any) atomicOr(&a.cases[bm.case_id].status, 1);
      }
    }
    cluster_sync();
    for (int c = tid; c < a.ncases; c += nth) {
      CaseState s = load_case(a.cases + c);
      case_dt_finalize(s);
      a.cases[c] = s;
    }
    cluster_sync();
    for (int st = 0; st < a.nst; ++st) {
      for (int x = tid; x < a.nwork * DIM * COUNT; x += nth) {
        int const item = x / (DIM * COUNT), r = x - item * DIM * COUNT;
        int const slot = a.work[item];
        BlockMeta const bm = a.meta[slot];
        if (!(__ldcg(&a.cases[bm.case_id].dt) > 0.0)) continue;
        if (DIM == 1 || r < COUNT)
          face_flux<DIM, 0, SCHEME, T, false, 2>(a.in[st], a.nbr26, slot, item, r, bm, a.F, a.stride);
        else
          face_flux<DIM, (DIM > 1 ? 1 : 0), SCHEME, T, false, 2>(
              a.in[st], a.nbr26, slot, item, r - COUNT, bm, a.F + a.dstride, a.stride);
      }
      cluster_sync();
      for (int x = tid; x < a.nwork * G::INTERIOR; x += nth) {
        int const item = x / G::INTERIOR;
        int const slot = a.work[item];
        BlockMeta const bm = a.meta[slot];
        double const dt = __ldcg(&a.cases[bm.case_id].dt);
        if (!(dt > 0.0)) continue;
        stage_update_cell<DIM, true>(a.in[st], a.U, a.out[st], a.F + (long long)item * a.stride,
                                     a.dstride, slot, x - item * G::INTERIOR, inv(bm.cell_size),
                                     rk_stage(a.s0 + st, dt));
      }
      cluster_sync();
    }
    if (a.commit)
      for (int c = tid; c < a.ncases; c += nth) {
        // the thread that finalized this case; only its own fields are stored
        // (the next signal speed is already under way)
        CaseState s = load_case(a.cases + c);
        case_commit(s);
        a.cases[c].t = s.t;
        a.cases[c].steps = s.steps;
      }
  }
}

template <int DIM, typename T>
void const *small_kernel(int scheme) {
  switch (scheme) {
    case FV_CHAR: return (void const *)small_steps_kernel<DIM, FV_CHAR, T>;
    case FV_PRIM: return (void const *)small_steps_kernel<DIM, FV_PRIM, T>;
    case FS_ROE: return (void const *)small_steps_kernel<DIM, FS_ROE, T>;
  }
  return nullptr;
}

long long stage_faces(int dim, int nwork) {
  return (long long)nwork * dim * (IC + 1) * (dim > 1 ? IC : 1);
}

}  // namespace

// One round of the largest cluster's threads. Step in us, launches against
// cluster: 1D 8 blocks 22.7 / 15.5, 64: 22.7 / 16.6, 128: 22.7 / 19.7, 256 (two
// rounds): 24.7 / 28.2; 2D 1 block 26.8 / 20.5, 4: 26.7 / 22.1, 6: 27.7 / 24.2,
// 8 (two rounds): 26.8 / 28.3.
bool small_pays(int dim, int nwork) {
  return dim < 3 && stage_faces(dim, nwork) <= kSmallCtas * kSmallThreads;
}

int small_launches(int n) { return n / kSmallSteps + (n % kSmallSteps != 0); }

cudaError_t launch_small_steps(Launch const &L, double *const in[3], double *const out[3],
                               double *F, long long stride, long long dstride, int const *nbr26,
                               CaseState *cases, int ncases, int nst, int s0, int n, bool commit) {
  if (L.nwork <= 0 || n <= 0) return cudaSuccess;
  if (!L.work || !L.meta || !nbr26 || !cases || nst < 1 || nst > 3) return cudaErrorInvalidValue;
  if (!L.opt.is_default() || L.dim < 1 || L.dim > 2) return cudaErrorInvalidValue;
  bool const f32 = L.precision == FP32_FLUX;
  void const *k = L.dim == 1 ? (f32 ? small_kernel<1, float>(L.scheme) : small_kernel<1, double>(L.scheme))
                             : (f32 ? small_kernel<2, float>(L.scheme) : small_kernel<2, double>(L.scheme));
  if (!k) return cudaErrorInvalidValue;
  // one face per thread; 128 threads a CTA while they suffice (four warps, one
  // to a scheduler: 1D 64 blocks 16.6 us against 19.6 with 256)
  long long const faces = stage_faces(L.dim, L.nwork);
  int const threads = faces <= kSmallCtas * 128 ? 128 : kSmallThreads;
  int ctas = 1;
  while (ctas < kSmallCtas && (long long)ctas * threads < faces) ctas *= 2;
  SmallArgs a{};
  for (int s = 0; s < nst; ++s) {
    a.in[s] = in[s];
    a.out[s] = out[s];
  }
  a.U = L.U;
  a.F = F;
  a.work = L.work;
  a.nwork = L.nwork;
  a.meta = L.meta;
  a.nbr26 = nbr26;
  a.cases = cases;
  a.ncases = ncases;
  a.nst = nst;
  a.s0 = s0;
  a.commit = commit;
  a.stride = stride;
  a.dstride = dstride;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = L.stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (ctas > 8) {
    // a partitioned GPU may not hold 16 CTAs in one cluster
    int fit = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();
      attr[0].val.clusterDim.x = 8;
      cfg.gridDim = dim3(8);
    }
  }
  for (; n > 0; n -= a.nsteps) {
    a.nsteps = n < kSmallSteps ? n : kSmallSteps;
    void *args[] = {&a};
    if (cudaError_t e = cudaLaunchKernelExC(&cfg, k, args)) return e;
  }
  return cudaSuccess;
}

}  // namespace alp
