// Launches of the plane-owner 3-D FP32 spreader (spread_plane3.cuh) for the
// tile shapes and window widths it is compiled for.
#include "spread_plane3.cuh"

#include <algorithm>

namespace nfft {
namespace {

template <int BX, int BY, int BZ, int L, int NW, bool TABLE>
int plane3_launch(nfft_plan* p, const Geom<float>& G, const Nodes<float>& Nd, const float2* fhat, float* gp, int ncols,
                  int64_t fcol, int64_t gcol_t) {
  using TC = Tile3<BX, BY, BZ, L>;
  using PC = Plane3<BX, BY, BZ, L, NW>;
  static_assert(TC::NACC * 8 <= kZeroTileBytes, "zero tile buffer");
  const CUtensorMap* map = (ncols == 1 && p->spread_tma) ? tile3_map<BX, BY, BZ, L>(p, gp) : nullptr;
  CUtensorMap none{};
  const float4* zeros = zero_tile_for(p);
  Plane3Poly<L, TABLE> wp{};
  if constexpr (!TABLE)
    for (int q = 0; q < L * (L + 1); ++q) wp.c[q] = float(p->coeffs_host[q]);
  auto kern = spread_plane3_kernel<BX, BY, BZ, L, NW, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, PC::SMEM));
  kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), PC::THREADS, PC::SMEM, p->stream>>>(
      map ? *map : none, map ? 1 : 0, G, Nd, p->tasks, fhat, gp, ncols > 1 ? fcol : 0, gcol_t, zeros, p->dflag + 1, wp);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

template <int BX, int BY, int BZ, int L, int NW>
int plane3_table(nfft_plan* p, const Geom<float>& G, const Nodes<float>& Nd, const float2* fhat, float* gp, int ncols,
                 int64_t fcol, int64_t gcol_t) {
  return p->wtab ? plane3_launch<BX, BY, BZ, L, NW, true>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t)
                 : plane3_launch<BX, BY, BZ, L, NW, false>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
}

// Two or four warps per tile.  Two read a node's weights half as often, four
// hide more latency where a tile has few nodes; L = 12's 79 KB tiles leave two CTAs per
// SM and want four.  Adjoint, us with two / four warps, uniform (radial) nodes:
//   m = 2: 64^3: 5,000 nodes 45 / 45 (40 / 42), 10^6 133 / 166 (124 / 160)
//   m = 3: 64^3: 50,000 67 / 63 (57 / 60), 200,000 97 / 102 (90 / 100), 4e6 875 / 1024;
//          128^3: 200,000 242 / 232 (182 / 188), 500,000 291 / 294 (242 / 254), 4e6 940 / 1094
//   m = 4: 64^3: 2e6 705 / 693 (686 / 708), 4e6 1275 / 1308 (1279 / 1322);
//          128^3: 10^6 519 / 499 (450 / 453), 4e6 1372 / 1399 (1310 / 1356)
//   m = 5: 128^3: 10^6 902 / 870 (789 / 796), 2e6 1482 / 1482, 4e6 2658 / 2723 (2573 / 2662)
template <int L> bool plane3_two_warps(const nfft_plan* p) {
  if (L == 4) return true;
  if (L == 6) return p->M >= (int64_t(1) << 17) && p->M >= 24 * p->n_tasks;
  return L < 12 && p->M >= 3 * (int64_t(1) << 20);
}

template <int BX, int BY, int BZ, int L>
int plane3_warps(nfft_plan* p, const Geom<float>& G, const Nodes<float>& Nd, const float2* fhat, float* gp, int ncols,
                 int64_t fcol, int64_t gcol_t) {
  if constexpr (L < 12)
    if (plane3_two_warps<L>(p)) return plane3_table<BX, BY, BZ, L, 2>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
  if constexpr (L > 4) return plane3_table<BX, BY, BZ, L, 4>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
  return -1;
}

template <int L>
int plane3_shape(nfft_plan* p, const Nodes<float>& Nd, const float2* fhat, float* gp, int ncols, int64_t fcol,
                 int64_t gcol_t) {
  const Geom<float> G = make_geom<float>(p);
  const int64_t bx = p->bs[0], by = p->bs[1];
  if (bx == 16 && by == 8) return plane3_warps<16, 8, 8, L>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
  if (bx == 8 && by == 8) return plane3_warps<8, 8, 8, L>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
  if constexpr (L == 8) {
    if (bx == 16 && by == 16) return plane3_warps<16, 16, 8, L>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
    if (bx == 32 && by == 8) return plane3_warps<32, 8, 8, L>(p, G, Nd, fhat, gp, ncols, fcol, gcol_t);
  }
  return -1;
}

}  // namespace

// Spreading of ncols columns (values in the caller's order) into zeroed
// grids; -1: the plan's tiles or window have no compiled kernel.
int launch_spread_plane3(nfft_plan* p, const void* fhat, void* g, int ncols, int64_t fcol, int64_t gcol_t) {
  if (!p->spread_tile3 || !p->spread_rec || p->D != 3 || p->precision != 32 || p->prm.compensated ||
      p->spread_layout != 1 || p->bs[2] != 8)
    return -1;
  const Nodes<float> Nd = make_nodes<float>(p);
  const float2* f = static_cast<const float2*>(fhat);
  float* gp = static_cast<float*>(g);
  switch (p->m) {
    case 2: return plane3_shape<4>(p, Nd, f, gp, ncols, fcol, gcol_t);
    case 3: return plane3_shape<6>(p, Nd, f, gp, ncols, fcol, gcol_t);
    case 4: return plane3_shape<8>(p, Nd, f, gp, ncols, fcol, gcol_t);
    case 5: return plane3_shape<10>(p, Nd, f, gp, ncols, fcol, gcol_t);
    case 6: return plane3_shape<12>(p, Nd, f, gp, ncols, fcol, gcol_t);
  }
  return -1;
}

}  // namespace nfft
