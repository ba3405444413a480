// 3-D FP32 gather from padded tiles in shared memory for any window width
// L = 2m = 4 .. 12 and the tile shapes fixed at compile time (tile3.cuh); for
// L = 8, grids whose tiles rarely wrap have their own kernel
// (interp_tile3_kernel, interp.cu).
//
// One CTA per task.  A tile inside the grid comes in by one bulk tensor copy, one
// that wraps around it by asynchronous 8-byte copies with the periodic
// index.  A half-warp takes a node's x-y planes as flat lists of L x L taps
// (t = (lane mod 16) + 16 step: conflict-free, the row pitch is L mod 16): it
// sums each of its taps' columns over z, weights the sums by phi_x phi_y and
// adds the lanes' partial sums of two nodes at once.  Nodes go through shared memory
// in warp-private batches of four, the next batch's records and window values in
// flight by cp.async; rows of window values are spaced so that two nodes' reads
// fall in distinct banks.
//
// Bound: shared-memory wavefronts and instruction issue.  L = 10: 95
// wavefronts a node (70 for the taps, 10 for the window values, 2 for the
// sums) at 76 % of one per clock and SM, 64 % of the issue slots.  240 x 216 x 180
// grid, 600,000 radial nodes: 528 us with the warp-per-node gather
// straight from L1 (30 of 32 lanes, shuffled weights), 263 with a whole warp
// per node of a tile, 251 now (128^3 transform, 10^6 uniform nodes, m = 6:
// 820 -> 772 us).  Without `act` the idle lanes of the last step read a tap's
// bank again: 19 wavefronts a node more; with rows of 32 floats 9 more, 261 us.
#include "tile3.cuh"
#include "warp2.cuh"

namespace nfft {
namespace {

constexpr int kG3Threads = 256;
constexpr int kG3Warps = kG3Threads / 32;

template <int BX, int BY, int BZ, int L, bool TABLE> struct Gather3 {
  using TC = Tile3<BX, BY, BZ, L>;
  static constexpr int NB = 4;                      // nodes per warp and batch
  static constexpr int TAPS = L * L;
  static constexpr int NSTEP = (TAPS + 15) / 16;    // of a half-warp
  static constexpr int NWIN = 3 * L;
  // staged window values of a node: the values of one dimension of two
  // neighbouring rows, read together, fall in distinct banks
  static constexpr int row_floats() {
    int w = NWIN;
    while (w % 32 < L || w % 32 > 32 - L) w += 2;
    return w;
  }
  static constexpr int WROW = row_floats();
  static constexpr int FRAC = TABLE ? 0 : 4;        // POLYNOMIAL: fractional offsets
  static constexpr int NODE_BYTES = 16 + WROW * 4 + FRAC * 4;
  static constexpr int SLOT = NB * NODE_BYTES;
  static_assert(SLOT % 16 == 0 && NB * WROW % 4 == 0, "16-byte records and offsets");
  static constexpr size_t STAGE_BYTES = size_t(kG3Warps) * 2 * SLOT;
  static constexpr size_t SMEM = TC::ACC_BYTES + 16 + STAGE_BYTES;
  static constexpr int PER_SM = int((227 * 1024) / (SMEM + 1024)) < 1 ? 1 : int((227 * 1024) / (SMEM + 1024));
};

template <int BX, int BY, int BZ, int L, bool TABLE>
__global__ void __launch_bounds__(kG3Threads, (Gather3<BX, BY, BZ, L, TABLE>::PER_SM > 3
                                                   ? 3
                                                   : Gather3<BX, BY, BZ, L, TABLE>::PER_SM))
    gather_plane3_kernel(const __grid_constant__ CUtensorMap tmap, int use_tma, Geom<float> G, Nodes<float> Nd,
                         const int4* __restrict__ tasks, const float2* __restrict__ g, float2* __restrict__ fhat,
                         int* status) {
  using TC = Tile3<BX, BY, BZ, L>;
  using GC = Gather3<BX, BY, BZ, L, TABLE>;
  constexpr int PITCH = TC::PITCH, PLANE = TC::PLANE, NB = GC::NB, NSTEP = GC::NSTEP;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(1024) unsigned char smem_g3[];
  float2* tile = reinterpret_cast<float2*>(smem_g3);
  const unsigned tile_s = static_cast<unsigned>(__cvta_generic_to_shared(tile));
  const unsigned mbar_s = static_cast<unsigned>(__cvta_generic_to_shared(smem_g3 + TC::ACC_BYTES));
  const int4 task = tasks[blockIdx.x];
  const int tc0 = task.x % G.ntiles[0];
  const int tc1 = (task.x / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = task.x / (G.ntiles[0] * G.ntiles[1]);
  const int o0 = tc0 * BX, o1 = tc1 * BY, o2 = tc2 * BZ;
  const int q0 = wrap_once(o0 + G.sh[0], G.Nt[0]), q1 = wrap_once(o1 + G.sh[1], G.Nt[1]);
  const int q2 = wrap_once(o2 + G.sh[2], G.Nt[2]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* stage_base = smem_g3 + TC::ACC_BYTES + 16 + warp * 2 * GC::SLOT;

  // a batch's records and window rows (or fractional offsets) into slot buf
  auto stage = [&](int buf, int b) {
    unsigned char* st = stage_base + buf * GC::SLOT;
    const int n = min(NB, task.z - b);
    if (n > 0) {
      if (lane < n) cp_async16(st + 16 * lane, Nd.node4 + b + lane);
      if constexpr (TABLE) {  // rows of 3L floats: 8-byte chunks (row starts are 8-byte aligned)
        constexpr int CH = GC::NWIN / 2;
        const float* src = Nd.wtab + int64_t(b) * GC::NWIN;
        for (int q = lane; q < n * CH; q += 32) {
          const int k = q / CH, c = q - k * CH;
          cp_async8(st + NB * 16 + k * GC::WROW * 4 + 8 * c, src + 2 * q);
        }
      } else if (lane < n) {
        cp_async16(st + NB * (16 + GC::WROW * 4) + 16 * lane, Nd.frac4 + 4 * int64_t(b + lane));
      }
    }
    cp_async_commit();
  };
  const bool bulk = use_tma && tile3_interior<BX, BY, BZ, L>(G, q0, q1, q2) && (tile_s & 127u) == 0;
  if (bulk) {
    if (threadIdx.x == 0) {
      mbar_init(mbar_s, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(mbar_s, unsigned(TC::NACC) * 8u);
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
          "[%5];" ::"r"(tile_s),
          "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(2 * (q0 - TC::XOFF)), "r"(q1 - (L / 2 - 1)),
          "r"(q2 - (L / 2 - 1)), "r"(mbar_s)
          : "memory");
    }
  } else {
    // columns [LEAD, P0) of every row, periodic in every dimension
    const int x0 = q0 - TC::XOFF, y0 = q1 - (L / 2 - 1), z0 = q2 - (L / 2 - 1);
    for (int r = warp; r < TC::P1 * TC::P2; r += kG3Warps) {
      const int z = r / TC::P1, y = r - z * TC::P1;
      const float2* row = g + int64_t(wrap_any(z0 + z, G.Nt[2])) * G.plane + int64_t(wrap_any(y0 + y, G.Nt[1])) * G.Nt[0];
      for (int x = TC::LEAD + lane; x < TC::P0; x += 32)
        cp_async8(tile + z * PLANE + y * PITCH + x, row + wrap_any(x0 + x, G.Nt[0]));
    }
    cp_async_commit();
  }
  const int first = task.y + NB * warp;
  stage(0, first);
  // POLYNOMIAL: value v = lane + 32 r of a node's 3L window values is column v mod L of dimension v / L
  constexpr int NR = (GC::NWIN + 31) / 32;
  float pc[TABLE ? 1 : NR][TABLE ? 1 : L + 1];
  if constexpr (!TABLE) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int v = lane + 32 * r;
#pragma unroll
      for (int i = 0; i <= L; ++i) pc[r][i] = v < GC::NWIN ? __ldg(G.coeffs + (v % L) * (L + 1) + i) : 0.f;
    }
  }
  // a half-warp per node: tap t = (lane mod 16) + 16 step of a plane
  const int half = lane >> 4;
  int lofs[NSTEP], ix[NSTEP], iy[NSTEP];
  bool act[NSTEP];
#pragma unroll
  for (int q = 0; q < NSTEP; ++q) {
    const int t = (lane & 15) + 16 * q;
    act[q] = GC::TAPS % 16 == 0 || t < GC::TAPS;
    const int tt = act[q] ? t : GC::TAPS - 1;
    iy[q] = tt / L;
    ix[q] = tt - iy[q] * L;
    lofs[q] = iy[q] * PITCH + ix[q] + TC::LEAD;
  }
  const unsigned origin = unsigned(o0) + unsigned(o1) * PITCH + unsigned(o2) * PLANE;
  bool ok = true;
  if (!bulk) asm volatile("cp.async.wait_group 1;" ::: "memory");  // this thread's part of the tile
  __syncthreads();
  if (bulk) ok = mbar_wait_bounded(mbar_s, 0);
  if (!ok) {  // no copy into shared memory outlives the CTA, as far as another bounded wait can tell
    if (lane == 0) atomicOr(status, 1);
    asm volatile("cp.async.wait_all;" ::: "memory");
    mbar_wait_bounded(mbar_s, 0);
    return;
  }
  int buf = 0;
  for (int b = first; b < task.z; b += NB * kG3Warps, buf ^= 1) {
    stage(buf ^ 1, b + NB * kG3Warps);
    cp_async_wait<1>();
    __syncwarp();
    const int n = min(NB, task.z - b);
    unsigned char* st = stage_base + buf * GC::SLOT;
    const int4* rec = reinterpret_cast<const int4*>(st);
    float* win = reinterpret_cast<float*>(st + NB * 16);
    if constexpr (!TABLE) {
      const float* fr = reinterpret_cast<const float*>(st + NB * (16 + GC::WROW * 4));
      for (int k = 0; k < n; ++k) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const int v = lane + 32 * r;
          if (v < GC::NWIN) {
            const float t = fr[4 * k + v / L] - 0.5f;
            float w = pc[r][L];
#pragma unroll
            for (int i = L - 1; i >= 0; --i) w = fmaf(w, t, pc[r][i]);
            win[k * GC::WROW + v] = w;
          }
        }
      }
      __syncwarp();
    }
    float ar[NB / 2], ai[NB / 2];
#pragma unroll
    for (int k = 0; k < NB / 2; ++k) {
      const int s = min(2 * k + half, n - 1);  // (nodes past the end repeat the last one and are dropped)
      const int4 nd = rec[s];
      const float* wn = win + s * GC::WROW;
      // (unsigned: PLANE times a grid index need not fit in 32 bits, its difference to the origin's does)
      const float2* p = tile + int(unsigned(nd.z) * PLANE + unsigned(nd.y) * PITCH + unsigned(nd.x) - origin);
      float sr[NSTEP], si[NSTEP];
#pragma unroll
      for (int q = 0; q < NSTEP; ++q) sr[q] = si[q] = 0.f;
#pragma unroll
      for (int iz = 0; iz < L; iz += 2) {
        const float2 wz = *reinterpret_cast<const float2*>(wn + 2 * L + iz);
#pragma unroll
        for (int q = 0; q < NSTEP; ++q)
          if (act[q]) {  // (idle lanes of the last step make no request)
            const float2 v0 = p[iz * PLANE + lofs[q]], v1 = p[(iz + 1) * PLANE + lofs[q]];
            sr[q] = fmaf(wz.x, v0.x, sr[q]);
            si[q] = fmaf(wz.x, v0.y, si[q]);
            sr[q] = fmaf(wz.y, v1.x, sr[q]);
            si[q] = fmaf(wz.y, v1.y, si[q]);
          }
      }
      float tr = 0.f, ti = 0.f;
#pragma unroll
      for (int q = 0; q < NSTEP; ++q) {
        const float w = (16 % L == 0 ? wn[ix[0]] : wn[ix[q]]) * wn[L + iy[q]];  // (idle lanes: zero sums)
        tr = fmaf(w, sr[q], tr);
        ti = fmaf(w, si[q], ti);
      }
      ar[k] = tr;
      ai[k] = ti;
    }
    // transposed butterfly: lanes l = 0, 8 (mod 16) end with pair l / 8 mod 2's node l / 16
    static_assert(NB == 4, "two pairs of nodes");
    const bool e = (lane & 8) != 0;
    float tr = (e ? ar[1] : ar[0]) + __shfl_xor_sync(FULL, e ? ar[0] : ar[1], 8);
    float ti = (e ? ai[1] : ai[0]) + __shfl_xor_sync(FULL, e ? ai[0] : ai[1], 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      tr += __shfl_xor_sync(FULL, tr, o);
      ti += __shfl_xor_sync(FULL, ti, o);
    }
    const int s = 2 * int(e) + half;
    if ((lane & 7) == 0 && s < n) fhat[rec[s].w] = make_float2(tr, ti);
    __syncwarp();  // the slot is read before it is staged again
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int BX, int BY, int BZ, int L, bool TABLE>
int gather3_launch(nfft_plan* p, const float2* g, float2* fhat) {
  using GC = Gather3<BX, BY, BZ, L, TABLE>;
  const CUtensorMap* map = p->gather_tma ? tile3_map<BX, BY, BZ, L>(p, const_cast<float2*>(g)) : nullptr;
  CUtensorMap none{};
  auto kern = gather_plane3_kernel<BX, BY, BZ, L, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, GC::SMEM));
  kern<<<unsigned(p->n_tasks), kG3Threads, GC::SMEM, p->stream>>>(map ? *map : none, map ? 1 : 0, make_geom<float>(p),
                                                                  make_nodes<float>(p), p->tasks, g, fhat,
                                                                  p->dflag + 1);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

template <int BX, int BY, int BZ, int L> int gather3_table(nfft_plan* p, const float2* g, float2* fhat) {
  return p->wtab ? gather3_launch<BX, BY, BZ, L, true>(p, g, fhat) : gather3_launch<BX, BY, BZ, L, false>(p, g, fhat);
}

template <int L> int gather3_shape(nfft_plan* p, const float2* g, float2* fhat) {
  if (p->bs[0] == 16 && p->bs[1] == 8) return gather3_table<16, 8, 8, L>(p, g, fhat);
  if (p->bs[0] == 8 && p->bs[1] == 8) return gather3_table<8, 8, 8, L>(p, g, fhat);
  return -1;
}

}  // namespace

// -1: the plan's tiles or window have no compiled kernel, or too few nodes per
// task to pay for bringing their tile (L = 10: 60 KB) into shared memory.
// Forward transform, us tiled / direct, uniform (radial) nodes:
//   m = 2: 64^3, 2048 tasks, 48 nodes per task 50 / 48 (41 / 47), 96: 55 / 62 (46 / 62);
//          128^3, 16,384 tasks, 48: 218 / 232 (167 / 227), 96: 252 / 357 (201 / 353)
//   m = 3: 64^3, 24: 56 / 46 (46 / 46), 48: 60 / 67 (50 / 66); 128^3, 24: 253 / 235
//          (180 / 229), 48: 290 / 357 (221 / 355)
//   m = 5: 64^3, 24: 79 / 75 (61 / 74), 48: 91 / 132 (72 / 130); 128^3, 12: 333 / 290
//          (198 / 285), 24: 364 / 448 (262 / 441)
//   m = 6: 64^3, 12: 97 / 87 (69 / 86), 24: 106 / 145 (82 / 145); 128^3, 12: 478 / 561
//          (255 / 561), 24: 535 / 931 (359 / 927)
// Compensated plans (tasks_suit): 65,536 radial nodes, 64^3, m = 3 49 / 42, m = 5 94 / 79;
// 300,000 86 / 125, 178 / 272; m = 4, any number of them, no slower than before.
// 27^3, 360 tasks (one or two CTAs per SM): m = 3, 34,560 nodes 46 / 44, m = 5, 17,280
// 52 / 50, 34,560 60 / 68.  m = 4, device times as fast as direct, uniform (radial) nodes: 30^3
// 66,000 0.97 (0.95), 80,000 1.18 (1.11), 150,000 1.25 (1.20), 300,000 1.45 (1.37); 60 x 54 x 45 0.88
// (0.91), 1.02 (1.03), 1.12 (1.11), 1.32 (1.27).
int launch_gather_plane3(const nfft_plan* cp, const void* g, void* fhat) {
  nfft_plan* p = const_cast<nfft_plan*>(cp);  // the tensor-map cache only
  if (!p->gather_tma || !p->tasks || p->n_tasks == 0 || p->D != 3 || p->precision != 32 || p->bs[2] != 8) return -1;
  const int per_task = p->m == 2 ? 64 : p->m <= 4 ? 48 : p->m == 5 ? 32 : 24;
  if (p->M < per_task * p->n_tasks || p->M < (p->m >= 5 ? 32768 : p->m == 4 ? 73728 : 65536)) return -1;
  if (p->m != 4 && !tasks_suit(p, 6)) return -1;
  const float2* gp = static_cast<const float2*>(g);
  float2* f = static_cast<float2*>(fhat);
  switch (p->m) {
    case 2: return gather3_shape<4>(p, gp, f);
    case 3: return gather3_shape<6>(p, gp, f);
    case 4: return gather3_shape<8>(p, gp, f);
    case 5: return gather3_shape<10>(p, gp, f);
    case 6: return gather3_shape<12>(p, gp, f);
  }
  return -1;
}

}  // namespace nfft
