// Spreading (convolve_transpose!): g[tap] += prod_d phi_d * fHat[j] over the
// (2m)^D window taps of every node, src/convolution.jl:349-520.
//
// The GB300 form of NFFT.jl's blocked adjoint (private padded block per
// block, then a locked wrap-add into g, :356-443):
//   * nodes are bin-sorted by home tile (bs[0] x bs[1] x bs[2] grid points);
//     one CTA per task = one home tile or a chunk of a hot tile;
//   * the CTA accumulates into the tile padded by 2m-1 points in shared
//     memory, so every tap of every node lands inside it: no per-tap bounds
//     tests and no wrap-around in the hot loop;
//   * D >= 2 (spread_owned_kernel): warp w owns the slices of the padded tile
//     along the last dimension with index = w mod 8 (x-y planes for D = 3, x
//     rows for D = 2).  Each tile point then has exactly one writer, so the
//     accumulation is a plain read-modify-write of a complex value (measured
//     ~17x the throughput of shared-memory float atomics on GB300), and can
//     carry a Kahan compensation term (compensated = 1).  Nodes are staged in
//     shared memory in batches (window values, x*y weight products, value);
//   * D = 1 (spread_pad1_kernel): 32/G nodes per warp, shared-memory atomics;
//     compensated (spread_line_kahan_kernel): one warp per task, lane l owns
//     the padded positions x = l mod 32, Kahan read-modify-writes;
//   * where they are faster (rules below, spread3.cu, double3.cu): D = 1 nodes sorted
//     by cell (line1.cuh), D = 2 one warp per task (warp2.cuh), D = 3 plane owners
//     (spread_plane3.cuh, double3.cuh);
//   * the padded tile is added to the zeroed grid with vector global atomics
//     (red.global.add.v2), wrapping periodically; all-zero points are skipped.
// The lock of the reference becomes the L2 atomics of the flush.
#include "spread_body.cuh"
#include "line1.cuh"
#include "spread_tile3.cuh"
#include "warp2.cuh"

namespace nfft {
namespace {

// D = 2, uncompensated: one warp per task (warp2.cuh); blockIdx.y: column of a multi-column launch.
template <int L, typename T, bool TABLE>
__global__ void __launch_bounds__(32) spread_warp2_kernel(Geom<T> G, Nodes<T> Nd, const int4* __restrict__ tasks,
                                                          const typename Cplx<T>::type* __restrict__ fhat,
                                                          T* __restrict__ g, int pitch, int64_t fcol, int64_t gcol,
                                                          const __grid_constant__ WinPoly<L, T, TABLE> wp) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  spread_warp2_body<L, T, TABLE>(G, Nd, __ldg(tasks + blockIdx.x), fhat + blockIdx.y * fcol, g + blockIdx.y * gcol,
                                 pitch, wp.c, smem_raw);
}

// 1-D: whether the sorting spreader (line1.cuh) is faster than the kernels of
// spread_body.cuh, atomics or, compensated, one warp per task.
//
// Up to 1024 cells (the counts and their scan outgrow
// the CTA) and from 3 nodes per 2 cells of the occupied tiles on: its sort
// and scan cost the same for few nodes (forward + adjoint, us, against the
// per-node kernels: 0.5 nodes per cell 173 / 162, 1.2 nodes 50 / 49, 2
// nodes 1233 / 1540 compensated, 30 nodes 180 / 222, 1500 nodes 243 / 448).
// Without compensation the atomics of short windows are cheaper than the sort,
// and in FP64 the serial window values and taps of a CTA's nodes cost more
// than atomics over all SMs until there are many CTAs.  Adjoint, times as fast as
// the per-node kernels: 300,000 nodes on 4,000 points (75 per cell), m = 2, 4, 5, 6, 8: FP32
// 0.77 0.90 1.20 1.09 1.14, compensated 1.15 1.19 1.31 1.34 1.47; FP64 1.17 1.24 0.95 0.83
// 0.71, compensated 1.05 1.01 0.72 0.72 0.72; 2e6 nodes on 200,000 points: FP32 0.85 0.90
// 1.32 1.40 1.16; FP64 0.93 1.02 1.46 1.26 0.94; 20,000 nodes 0.90 - 1.02.
//
// A tile of few cells keeps only as many of its CTA's lanes busy as it has
// positions, for all of its nodes.  That is made up for while the tasks do not fill
// the GPU anyway (300,000 nodes, grid of 256 points, 300 tasks: 1.2 to 1.5 times as
// fast), not by short or many tasks.  Adjoint, times as fast, compensated, tiles of 8 cells,
// grid of 8,000 points: 66,000 / 300,000 / 2e6 nodes m = 3 0.78 / 0.76 / 0.55, m = 5 0.82 / 0.87 /
// 0.68; 256 points, 900,000 / 2e6: m = 3 0.68 / 0.56; tiles of 32 cells 66,000 / 130,000 / 300,000:
// 0.96 / 1.04 / 1.18, FP64 m = 8, 2e6 0.72.  FP32 without compensation, m = 6, tiles of 8 or 32
// cells, about 1000 tasks, 66,000 to 900,000 nodes 0.81 to 0.89, 2e6 (2000 tasks) 1.14 to
// 1.23; m = 8 0.93 (64 nodes per task) to 1.2.  FP64, m = 4, tiles of 32 cells, 66,000 /
// 130,000 / 300,000 / 900,000 0.79 / 0.89 / 0.93 / 1.15, m = 3 0.87 / 0.98 / 1.04 / 1.35; 256 points, 66 to
// 130 tasks 0.79.
template <int L, typename T> bool line_sort_pays(const nfft_plan* p) {
  constexpr bool kDouble = sizeof(T) == 8;
  const bool comp = p->prm.compensated != 0;
  const int64_t bs = p->bs[0], M = p->M, tasks = p->n_tasks;
  if (bs > kLineMaxTile || 2 * M < 3 * std::min(tasks, p->ntiles_total) * bs) return false;
  if (M < (kDouble && L >= 10 ? int64_t(1) << 20 : 65536)) return false;
  if (!comp && (kDouble ? L == 4 || L == 16 : L <= 8)) return false;
  if (bs >= 64) return true;
  if (tasks <= 4 * int64_t(p->sms)) return comp || !kDouble || 2 * tasks >= 3 * int64_t(p->sms);
  if (comp) return bs >= 32 && M >= 96 * tasks && !(kDouble && L >= 12);
  if (!kDouble) return L == 16 ? M >= 128 * tasks : 2 * tasks >= 17 * int64_t(p->sms);
  return M >= (bs < 16 ? 96 : L == 8 ? 384 : 128) * tasks;
}

template <int L, typename T, bool TABLE, bool KAHAN>
int spread_line_launch(nfft_plan* p, const Geom<T>& G, const Nodes<T>& Nd, const typename Cplx<T>::type* fhat, T* g,
                       int ncols, int64_t fcol, int64_t gcol_t) {
  const size_t smem = Line1<L, T, KAHAN>::smem(int(p->bs[0]));
  if (smem > 227 * 1024) return -1;
  LinePoly<L, T, TABLE> wp{};
  if constexpr (!TABLE)
    for (int q = 0; q < L * (L + 1); ++q) wp.c[q] = T(p->coeffs_host[q]);
  auto kern = spread_line_kernel<L, T, TABLE, KAHAN>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), kLineThreads, smem, p->stream>>>(G, Nd, p->tasks, fhat, g, fcol,
                                                                                      gcol_t, wp);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

template <int L, typename T, bool TABLE>
int spread_warp2_launch(nfft_plan* p, const Geom<T>& G, const Nodes<T>& Nd, const typename Cplx<T>::type* fhat, T* g,
                        int ncols, int64_t fcol, int64_t gcol_t) {
  const int pitch = warp2_plan_pitch<L, T, TABLE>(p);
  const size_t smem = warp2_spread_bytes<L, T, TABLE>(p);
  WinPoly<L, T, TABLE> wp{};
  if constexpr (!TABLE)
    for (int q = 0; q < L * (L + 1); ++q) wp.c[q] = T(p->coeffs_host[q]);
  auto kern = spread_warp2_kernel<L, T, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), 32, smem, p->stream>>>(G, Nd, p->tasks, fhat, g, pitch, fcol,
                                                                            gcol_t, wp);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

// Whether the uncompensated 2-D spreading of ncols columns runs two warps per
// tile (spread_owned_kernel, on bin-sorted values) instead of one (warp2.cuh).
// FP64, tiles that fit in shared memory with the staging of the former but not
// with that of the latter, which is 2 to 5 KB larger (FP32: smaller).
// FP64, single plans: from m = 5 on, for few nodes, and for m = 4
// where the GPU is full anyway (a task's window values and taps keep one
// warp's FP64 operations in a row too long).  Adjoint, us one warp / two warps per task, 60,000 uniform nodes on a
// 300 x 263 image: m = 4 275 / 270, m = 5 307 / 297, m = 8 410 / 377; 3,000 radial
// nodes, 64 x 56: m = 4 109 / 96, m = 8 232 / 159.
// FP64, several columns: m = 8, and few node values in all, or, m >= 6, few nodes (times
// as fast with two warps, forward + adjoint of a 40 x 30 / 128 x 118 stack: m = 8, 6,000 nodes,
// 2 columns 1.16 / 1.12, 8 1.03 / 1.07, 64 1.03 / 1.08; m = 5, 2 columns of 12,000 1.08 /
// 1.03, of 24,000 1.01, 8 of 3,000 1.04 / 1.03, of 6,000 1.00 / 1.03; m = 7, 64 of 3,000 1.00 / 1.05,
// of 12,000 0.92 - 1.01; m = 4, 2 of 3,000 1.06).
template <int L, typename T> bool spread2_two_warps(const nfft_plan* p, int64_t ncols) {
  if (sizeof(T) == 4) return false;
  const bool table = p->prm.precompute != NFFT_PRECOMPUTE_POLYNOMIAL;
  if ((table ? warp2_spread_bytes<L, T, true>(p) : warp2_spread_bytes<L, T, false>(p)) > size_t(kSmemMost)) return true;
  if (ncols > 1) {
    const int64_t values = p->M * p->task_columns;
    return L == 16 || (L >= 10 && values < 32768) || (L >= 12 && p->M < 4096) || (L == 8 && values < 8192);
  }
  return L >= 10 || p->M < 4096 || (L == 8 && p->M >= 32768);
}

// fHat in bin-sorted order (node4[i].w = input index), for coalesced staging.
// blockIdx.y: column of a multi-column launch (input fhat + y fcol, output out + y M)
template <typename T>
__global__ void sort_values_kernel(const int4* __restrict__ node4, const typename Cplx<T>::type* __restrict__ fhat,
                                   typename Cplx<T>::type* __restrict__ out, int64_t M, int64_t fcol = 0) {
  fhat += blockIdx.y * fcol;
  out += blockIdx.y * M;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < M; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = __ldg(fhat + __ldg(node4 + i).w);
}

// fHat of every column in bin-sorted order (grid-stride, a few CTAs per SM).
template <typename T>
int sort_values(const nfft_plan* p, const typename Cplx<T>::type* fhat, typename Cplx<T>::type* out, int ncols,
                int64_t fcol) {
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                cudaSuccess || sms < 1)
    sms = 1;
  int64_t nb = (p->M + 255) / 256;
  const int64_t cap = (int64_t(sms) * 32 + ncols - 1) / ncols;
  if (nb > cap) nb = cap;
  if (nb < 1) nb = 1;
  sort_values_kernel<T><<<dim3(unsigned(nb), unsigned(ncols)), 256, 0, p->stream>>>(p->node4, fhat, out, p->M, fcol);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

template <int BX, int BY, int BZ>
int tile3_launch(nfft_plan* p, const Geom<float>& G, const Nodes<float>& Nd, const float2* fs, float* gp, int ncols,
                 int64_t fcol, int64_t gcol_t) {
  using TC = Tile3<BX, BY, BZ>;
  const CUtensorMap* map = (ncols == 1 && p->spread_tma) ? tile3_map<BX, BY, BZ>(p, gp) : nullptr;
  const int use_tma = map ? 1 : 0;
  CUtensorMap none{};
  auto kern = p->wtab ? spread_tile3_kernel<BX, BY, BZ, true> : spread_tile3_kernel<BX, BY, BZ, false>;
  NFFT_CUDA_TRY(allow_smem(kern, TC::SMEM));
  kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), TC::THREADS, TC::SMEM, p->stream>>>(
      map ? *map : none, use_tma, G, Nd, p->tasks, fs, gp, ncols > 1 ? fcol : 0, gcol_t);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

// The shape-specialised 3-D kernel when the plan's tiles have one of its
// shapes (FP32, m = 4, uncompensated, 8-warp layout); -1 = not applicable.
int spread_tile3(nfft_plan* p, const Geom<float>& G, const Nodes<float>& Nd, const float2* fs, float* gp, int ncols,
                 int64_t fcol, int64_t gcol_t) {
  if (!p->spread_tile3 || p->D != 3 || p->m != 4 || p->prm.compensated || p->spread_layout != 1) return -1;
  const int64_t bx = p->bs[0], by = p->bs[1], bz = p->bs[2];
  if (bz != 8) return -1;
  if (bx == 16 && by == 8) return tile3_launch<16, 8, 8>(p, G, Nd, fs, gp, ncols, fcol, gcol_t);
  if (bx == 16 && by == 16) return tile3_launch<16, 16, 8>(p, G, Nd, fs, gp, ncols, fcol, gcol_t);
  if (bx == 32 && by == 8) return tile3_launch<32, 8, 8>(p, G, Nd, fs, gp, ncols, fcol, gcol_t);
  if (bx == 8 && by == 8) return tile3_launch<8, 8, 8>(p, G, Nd, fs, gp, ncols, fcol, gcol_t);
  return -1;
}

// ncols columns in one launch (blockIdx.y): values fhat + c fcol, grids
// g + c gcol (complex elements; the grids must be contiguous, gcol = |Ntilde|),
// bin-sorted values in `sorted` (M x ncols); ncols = 1 uses the plan's own scratch.
template <int D, int L, typename T>
int spread_launch(nfft_plan* p, const void* fhat, void* g, int ncols, int64_t fcol, int64_t gcol, void* sorted) {
  Geom<T> G = make_geom<T>(p);
  Nodes<T> Nd = make_nodes<T>(p);
  using C = typename Cplx<T>::type;
  const size_t gbytes = size_t(p->Nt[0] * p->Nt[1] * p->Nt[2]) * sizeof(T) * 2;
  if (!p->skip_memset) NFFT_CUDA_TRY(cudaMemsetAsync(g, 0, gbytes * size_t(ncols), p->stream));
  if (p->n_tasks == 0) return NFFT_OK;
  const C* fp = static_cast<const C*>(fhat);
  T* gp = static_cast<T*>(g);
  const int64_t gcol_t = 2 * gcol;  // in T units
  if (ncols > 1 && (p->prm.compensated || (D == 3 && p->spread_layout == 2))) {
    set_error("multi-column spreading supports the default (uncompensated, 8-warp) tiles only");
    return NFFT_ERR_UNSUPPORTED;
  }
  if constexpr (D == 1) {
    if (line_sort_pays<L, T>(p)) {
      // FP32 TENSOR plans: Horner (2m multiply-adds a value) gives the table's own
      // values for less than reading them; FP64 units are too few for that
      const bool table = p->wtab && !(sizeof(T) == 4 && G.mode == WIN_POLY);
      const int rc =
          p->prm.compensated
              ? (table ? spread_line_launch<L, T, true, true>(p, G, Nd, fp, gp, ncols, fcol, gcol_t)
                       : spread_line_launch<L, T, false, true>(p, G, Nd, fp, gp, ncols, fcol, gcol_t))
              : (table ? spread_line_launch<L, T, true, false>(p, G, Nd, fp, gp, ncols, fcol, gcol_t)
                       : spread_line_launch<L, T, false, false>(p, G, Nd, fp, gp, ncols, fcol, gcol_t));
      if (rc != -1) return rc;
    }
    if (p->prm.compensated) {
      const size_t smem = ((sizeof(typename Acc<T, true>::type) * size_t(p->bs[0] + L - 1) + 31) & ~size_t(31)) +
                          sizeof(T) * size_t(2 * 32 * L + L * (L + 1));
      if (smem > 227 * 1024) {
        set_error("compensated spreading row of %zu bytes does not fit in shared memory; use a smaller blockSize",
                  smem);
        return NFFT_ERR_UNSUPPORTED;
      }
      auto kern = p->wtab ? spread_line_kahan_kernel<L, T, true> : spread_line_kahan_kernel<L, T, false>;
      NFFT_CUDA_TRY(allow_smem(kern, smem));
      kern<<<unsigned(p->n_tasks), 32, smem, p->stream>>>(G, Nd, p->tasks, fp, gp);
      NFFT_LAUNCH_CHECK();
      return NFFT_OK;
    }
    const size_t smem = 2 * sizeof(T) * size_t(p->bs[0] + L - 1);
    if (smem > 227 * 1024) {
      set_error("spreading row of %zu bytes does not fit in shared memory; use a smaller blockSize", smem);
      return NFFT_ERR_UNSUPPORTED;
    }
    auto kern = p->wtab ? spread_pad1_kernel<L, T, true> : spread_pad1_kernel<L, T, false>;
    NFFT_CUDA_TRY(allow_smem(kern, smem));
    kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), kSpreadThreads, smem, p->stream>>>(G, Nd, p->tasks, fp, gp,
                                                                                          fcol, gcol_t);
  } else {
    const bool comp = p->prm.compensated != 0;
    const size_t smem = owned_smem<D, L, T>(p, comp);
    if (smem > 227 * 1024) {
      set_error("padded spreading tile (%zu bytes) does not fit in shared memory; use a smaller blockSize", smem);
      return NFFT_ERR_UNSUPPORTED;
    }
    auto kern = p->wtab ? spread_owned_kernel<D, L, T, true, true> : spread_owned_kernel<D, L, T, false, true>;
    int threads = OwnedCfg<D, L>::THREADS;
    if constexpr (D == 2) {
      const bool two = spread2_two_warps<L, T>(p, ncols);
      // (FP64: m = 8, and from m = 5 on POLYNOMIAL windows, which no stack has, always run two)
      constexpr bool kTable = sizeof(T) == 4 || L < 16, kPoly = sizeof(T) == 4 || L <= 8;
      if (!comp && !two) {
        if constexpr (kTable)
          if (p->wtab) return spread_warp2_launch<L, T, true>(p, G, Nd, fp, gp, ncols, fcol, gcol_t);
        if constexpr (kPoly)
          if (!p->wtab) return spread_warp2_launch<L, T, false>(p, G, Nd, fp, gp, ncols, fcol, gcol_t);
      }
      if constexpr (sizeof(T) == 8)
        if (!comp) kern = p->wtab ? spread_owned_kernel<D, L, T, true, false> : spread_owned_kernel<D, L, T, false, false>;
    }
    if constexpr (D == 3) {
      if (!comp) kern = p->wtab ? spread_owned_kernel<D, L, T, true, false> : spread_owned_kernel<D, L, T, false, false>;
      if (!comp && p->spread_layout == 2) {  // 16 warps: slice group x row parity
        kern = p->wtab ? spread_owned_kernel<D, L, T, true, false, 2> : spread_owned_kernel<D, L, T, false, false, 2>;
        threads = OwnedCfg<D, L, 2>::THREADS;
      }
    }
    // (L = 8: eight warps with one full plane of a node each waste nothing in
    // spread_owned_kernel either, and flush twice as fast; 64^3 image, 100,000 nodes 543
    // against 580 us for the whole adjoint)
    if constexpr (D == 3 && sizeof(T) == 8 && L != 8) {
      if (!comp && p->spread_layout == 1 && ncols == 1) {
        const int rc = launch_spread_double3(p, fhat, g);
        if (rc != -1) return rc;
      }
    }
    if constexpr (D == 3 && sizeof(T) == 4 && L <= 12) {  // values read in the caller's order
      const int rc = launch_spread_plane3(p, fhat, g, ncols, fcol, gcol_t);
      if (rc != -1) return rc;
    }
    NFFT_CUDA_TRY(allow_smem(kern, smem));
    C* fs = static_cast<C*>(ncols > 1 ? sorted : p->fsorted);
    int rc = sort_values<T>(p, fp, fs, ncols, fcol);
    if (rc) return rc;
    if constexpr (D == 3 && L == 8 && sizeof(T) == 4) {
      rc = spread_tile3(p, G, Nd, fs, gp, ncols, p->M, gcol_t);
      if (rc != -1) return rc;
    }
    kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), threads, smem, p->stream>>>(G, Nd, p->tasks, fs, gp,
                                                                                   p->spread_pitch, p->M, gcol_t);
  }
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

#define NFFT_SPREAD_ARGS p, fhat, g, ncols, fcol, gcol, sorted
template <int D, typename T>
int spread_dispatch_l(nfft_plan* p, const void* fhat, void* g, int ncols, int64_t fcol, int64_t gcol, void* sorted) {
  switch (p->m) {
    case 2: return spread_launch<D, 4, T>(NFFT_SPREAD_ARGS);
    case 3: return spread_launch<D, 6, T>(NFFT_SPREAD_ARGS);
    case 4: return spread_launch<D, 8, T>(NFFT_SPREAD_ARGS);
    case 5: return spread_launch<D, 10, T>(NFFT_SPREAD_ARGS);
    case 6: return spread_launch<D, 12, T>(NFFT_SPREAD_ARGS);
    case 7: return spread_launch<D, 14, T>(NFFT_SPREAD_ARGS);
    case 8: return spread_launch<D, 16, T>(NFFT_SPREAD_ARGS);
  }
  set_error("m = %d not supported (2..8)", p->m);
  return NFFT_ERR_UNSUPPORTED;
}

template <typename T>
int spread_dispatch(nfft_plan* p, const void* fhat, void* g, int ncols, int64_t fcol, int64_t gcol, void* sorted) {
  switch (p->D) {
    case 1: return spread_dispatch_l<1, T>(NFFT_SPREAD_ARGS);
    case 2: return spread_dispatch_l<2, T>(NFFT_SPREAD_ARGS);
    case 3: return spread_dispatch_l<3, T>(NFFT_SPREAD_ARGS);
  }
  return NFFT_ERR_UNSUPPORTED;
}
#undef NFFT_SPREAD_ARGS

}  // namespace

// A zeroed buffer as large as the largest padded tile, copied into shared
// memory to clear each CTA's tile (allocated once per plan).
const float4* zero_tile_for(nfft_plan* p) {
  if (!p->zero_tile && p->spread_zero_copy) {
    // nothing is allocated while the caller captures a graph (the copy source
    // is made by the first call outside one): plain stores clear the tile
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(p->stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return nullptr;
    }
    if (cudaMalloc(&p->zero_tile, kZeroTileBytes) != cudaSuccess ||
        cudaMemsetAsync(p->zero_tile, 0, kZeroTileBytes, p->stream) != cudaSuccess) {
      cudaFree(p->zero_tile);
      p->zero_tile = nullptr;
      p->spread_zero_copy = false;  // plain stores clear the tile
      cudaGetLastError();
    }
  }
  return p->spread_zero_copy ? static_cast<const float4*>(p->zero_tile) : nullptr;
}

bool spread_cols_sorted(const nfft_plan* p, int64_t ncols) {
  if (p->D != 2) return p->D == 3;
  if (p->precision == 32) return false;
  switch (p->m) {
    case 2: return spread2_two_warps<4, double>(p, ncols);
    case 3: return spread2_two_warps<6, double>(p, ncols);
    case 4: return spread2_two_warps<8, double>(p, ncols);
    case 5: return spread2_two_warps<10, double>(p, ncols);
    case 6: return spread2_two_warps<12, double>(p, ncols);
    case 7: return spread2_two_warps<14, double>(p, ncols);
    default: return spread2_two_warps<16, double>(p, ncols);
  }
}

// Row pitch (in accumulator elements) of the padded tile: the smallest pitch
// >= the padded row length for which every shared-memory access phase of a
// warp step (lanes = L taps along x times the row slots) hits distinct banks.
int spread_pitch_for(int D, int m, int P0, int elem_bytes, int ny) {
  const int L = 2 * m;
  // lane -> (column ix, row slot ry); D = 3 rows are ny pitches apart (ny = 2:
  // row-parity ownership), D = 2 rows of one warp are 2 slices = 2 pitches apart
  const int RY = D == 3 ? 32 / L : (D == 2 ? (L + 1) / 2 : 1);
  const int rowmul = D == 2 ? 2 : (D == 3 ? ny : 1);
  const int words = elem_bytes / 4;       // 32-bit words per element
  const int lanes_per_phase = 32 / words;  // lanes served per shared-memory wavefront
  for (int pitch = P0; pitch < P0 + 64; ++pitch) {
    bool ok = true;
    for (int ph = 0; ph < words && ok; ++ph) {
      int used[32] = {};
      for (int l = ph * lanes_per_phase; l < (ph + 1) * lanes_per_phase && ok; ++l) {
        const int ix = l % L, ry = l / L;
        if (ry >= RY) continue;
        for (int w = 0; w < words; ++w) {
          const int bank = ((ix + pitch * rowmul * ry) * words + w) % 32;
          if (used[bank]++) ok = false;
        }
      }
    }
    if (ok) return pitch;
  }
  return P0;
}

int launch_spread(nfft_plan* p, const void* fhat, int, void* g, int) {
  return p->precision == 32 ? spread_dispatch<float>(p, fhat, g, 1, 0, 0, nullptr)
                            : spread_dispatch<double>(p, fhat, g, 1, 0, 0, nullptr);
}

int launch_spread_cols(nfft_plan* p, const void* fhat, void* g, int ncols, int64_t fcol, int64_t gcol,
                       void* sorted) {
  return p->precision == 32 ? spread_dispatch<float>(p, fhat, g, ncols, fcol, gcol, sorted)
                            : spread_dispatch<double>(p, fhat, g, ncols, fcol, gcol, sorted);
}

}  // namespace nfft
