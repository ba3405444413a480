// Launches of the 3-D FP64 gather and spreader (double3.cuh).
#include "double3.cuh"

namespace nfft {
namespace {

template <int L, bool TABLE> int gather_launch(const nfft_plan* p, const double2* g, double2* fhat) {
  const int pitch = gather3d_pitch(int(p->bs[0]) + L - 1);
  const size_t smem = Gather3D<L>::stage_bytes() +
                      sizeof(double2) * size_t(pitch) * size_t(p->bs[1] + L - 1) * size_t(p->bs[2] + L - 1);
  if (smem > 227 * 1024) return -1;
  auto kern = gather_double3_kernel<L, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  kern<<<unsigned(p->n_tasks), kD3GatherThreads, smem, p->stream>>>(make_geom<double>(p), make_nodes<double>(p),
                                                                    p->tasks, g, fhat, pitch);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

template <int L, bool TABLE> int spread_launch(const nfft_plan* p, const double2* fhat, double* g) {
  const int64_t rows = (p->bs[1] + L - 1) * (p->bs[2] + L - 1);
  const int64_t limit = (int64_t(227) * 1024 - int64_t(Spread3D<L>::STAGE)) / (16 * rows);
  const int P0 = int(p->bs[0]) + L - 1;
  if (P0 > limit) return -1;
  const int pitch = warp2_pitch(2 * p->m, 8, P0, limit);
  const size_t smem = Spread3D<L>::STAGE + 16 * size_t(pitch) * size_t(rows);
  auto kern = spread_double3_kernel<L, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  kern<<<unsigned(p->n_tasks), Spread3D<L>::THREADS, smem, p->stream>>>(make_geom<double>(p), make_nodes<double>(p),
                                                                       p->tasks, fhat, g, pitch);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

}  // namespace

// -1: not applicable (no task list, a tile that does not fit, or too few
// nodes per task, or in all, to pay for bringing their tile into shared
// memory.  Forward transform, us tiled / direct, m = 5: 4096 tasks, 20,000 nodes
// 486 / 332, 100,000 797 / 1014, 262,144 1.31 / 1.99 ms in the gather; 225 tasks, 20,000
// nodes 248 / 225, 100,000 785 / 903.  m = 3: 4096 tasks, 20,000 nodes 278 / 232, 100,000
// 332 / 468; 225 tasks, 4000 nodes 83 / 82, 100,000 262 / 359).  Compensated plans
// (tasks_suit): 80,000 radial nodes, 32^3, m = 4 595 / 347, m = 5 1552 / 861, uniform 259 /
// 327, 469 / 842; 300,000 radial m = 4 1210 / 1008, m = 5 1958 / 2167; 270,000 in 128 tiles
// m = 4 1150 / 905.
int launch_gather_double3(const nfft_plan* p, const void* g, void* fhat) {
  if (!p->tasks || p->n_tasks == 0 || p->M < 16 * p->n_tasks || p->M < 65536) return -1;
  if (!tasks_suit(p, 4)) return -1;
  if (p->m == 4 && p->prm.compensated && p->longest_task > 512 && p->M < (int64_t(1) << 19)) return -1;
#define NFFT_D3_GATHER(L)                                                                                \
  case L / 2:                                                                                            \
    return p->wtab ? gather_launch<L, true>(p, static_cast<const double2*>(g), static_cast<double2*>(fhat)) \
                   : gather_launch<L, false>(p, static_cast<const double2*>(g), static_cast<double2*>(fhat))
  switch (p->m) {
    NFFT_D3_GATHER(4);
    NFFT_D3_GATHER(6);
    NFFT_D3_GATHER(8);
    NFFT_D3_GATHER(10);
    NFFT_D3_GATHER(12);
    NFFT_D3_GATHER(14);
    NFFT_D3_GATHER(16);
  }
#undef NFFT_D3_GATHER
  return -1;
}

// Spreading into a zeroed grid (values in the caller's order); -1: m = 4 and m >= 6
// (spread_owned_kernel is as good or better there), fewer tasks than fill the
// GPU (a task's latency counts, and eight warps have less of it), m = 5 with few nodes in small
// tiles, or the tile and its staging do not fit in shared memory.  Adjoint, us here / there, 64^3, 4096
// tasks: m = 3, 24,576 uniform nodes 297 / 337, 196,608 549 / 624; m = 5 505 / 574,
// 1291 / 1540; m = 6 906 / 734, 2451 / 2402.  24^3, 150 tasks: m = 3, 3,600 radial
// nodes 133 / 127, m = 5 234 / 223, uniform 125 / 123.  32^3, tiles of 8 x 8 x 4, times as fast as there:
// m = 7, 2,000 / 20,000 / 150,000 uniform nodes 0.71 / 0.80 / 0.85; m = 5 0.89 / 1.0 / 1.09, 10,000 0.94.
int launch_spread_double3(const nfft_plan* p, const void* fhat, void* g) {
  if (p->n_tasks < 4 * int64_t(p->sms)) return -1;
  const auto* f = static_cast<const double2*>(fhat);
  double* gd = static_cast<double*>(g);
  switch (p->m) {
    case 2: return p->wtab ? spread_launch<4, true>(p, f, gd) : spread_launch<4, false>(p, f, gd);
    case 3: return p->wtab ? spread_launch<6, true>(p, f, gd) : spread_launch<6, false>(p, f, gd);
    case 5:
      if (p->bs[0] * p->bs[1] * p->bs[2] < 512 && p->M < 16 * p->n_tasks) return -1;
      return p->wtab ? spread_launch<10, true>(p, f, gd) : spread_launch<10, false>(p, f, gd);
  }
  return -1;
}

}  // namespace nfft
