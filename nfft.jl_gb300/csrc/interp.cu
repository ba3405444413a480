// Gather interpolation (convolve!): fHat[j] = sum over the (2m)^D window taps
// of prod_d phi_d * g[tap], src/convolution.jl:229-344 (blocked) and :56-99.
//
// D = 1: one thread per node (line1.cuh); D = 2: one warp per task from
// tiles in shared memory (warp2.cuh); D = 3: tiled (below, gather3.cu, double3.cuh); each
// where its rule finds enough nodes and tasks.
// Otherwise a warp per node, nodes visited in bin-sorted order; each CTA takes
// a contiguous chunk of the sorted nodes, so the nodes an SM visits close in time read overlapping grid
// neighbourhoods through L1, and a warp issues all of a node's grid loads
// before its sums (memory-level parallelism).  Window values come from the stored window
// tensor (TENSOR / FULL / LINEAR) or from the fitted polynomial evaluated with
// its coefficients held in registers (POLYNOMIAL).  Grid offsets within a
// plane are 32-bit; the plane offset is 64-bit.
#include "interp_body.cuh"
#include "line1.cuh"
#include "tile3.cuh"
#include "warp2.cuh"

#include <algorithm>

namespace nfft {
namespace {

constexpr int kInterpThreads = 256;

// 8- or 16-byte asynchronous global -> shared copy (cp.async, sm_80+).
template <typename C> __device__ __forceinline__ void cp_async_elem(C* smem, const C* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if constexpr (sizeof(C) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int D, int L, typename T, bool TABLE, bool COLS = false>
__global__ void __launch_bounds__(kInterpThreads) interp_kernel(Geom<T> G, Nodes<T> Nd,
                                                                 const typename Cplx<T>::type* __restrict__ g,
                                                                 typename Cplx<T>::type* __restrict__ fhat,
                                                                 int64_t gcol = 0, int64_t fcol = 0) {
  static_assert(D >= 2, "D = 1: line1.cuh");
  if constexpr (COLS) {  // column of a multi-column launch
    g += blockIdx.y * gcol;
    fhat += blockIdx.y * fcol;
  }
  const int lane = threadIdx.x & 31;
  PolyRegs<D, L, T> P;
  if constexpr (!TABLE) P.load(G.coeffs, lane);
  // each CTA takes a contiguous chunk of the bin-sorted nodes: nodes a CTA
  // visits close in time share their grid neighbourhood in L1
  const int64_t chunk = (Nd.M + gridDim.x - 1) / gridDim.x;
  const int64_t lo = int64_t(blockIdx.x) * chunk;
  const int64_t hi = lo + chunk < Nd.M ? lo + chunk : Nd.M;
  for (int64_t i = lo + (threadIdx.x >> 5); i < hi; i += blockDim.x >> 5)
    interp_node<D, L, T, TABLE>(G, Nd, P, i, lane, g, fhat);
}

// Tile-staged gather: one CTA per spreading task (home tile or chunk of a hot
// tile).  The CTA copies the tile's padded neighbourhood of the grid (with
// periodic wrap) into shared memory with coalesced row loads, then each warp
// interpolates one node at a time from shared memory: no wrap logic and no
// global addressing in the tap loop.
template <int D, int L, typename T, bool TABLE>
__global__ void __launch_bounds__(kInterpThreads) interp_tile_kernel(Geom<T> G, Nodes<T> Nd,
                                                                      const int4* __restrict__ tasks,
                                                                      const typename Cplx<T>::type* __restrict__ g,
                                                                      typename Cplx<T>::type* __restrict__ fhat,
                                                                      int pitch) {
  using C = typename Cplx<T>::type;
  using LN = Lanes<D, L>;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  C* tile = reinterpret_cast<C*>(smem_raw);
  const int4 task = tasks[blockIdx.x];
  const int t = task.x;
  const int tc0 = t % G.ntiles[0];
  const int tc1 = (t / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = t / (G.ntiles[0] * G.ntiles[1]);
  const int P0 = G.bs[0] + L - 1;
  const int P1 = D >= 2 ? G.bs[1] + L - 1 : 1;
  const int P2 = D == 3 ? G.bs[2] + L - 1 : 1;
  const int o0 = tc0 * G.bs[0], o1 = D >= 2 ? tc1 * G.bs[1] : 0, o2 = D == 3 ? tc2 * G.bs[2] : 0;
  const int plane = pitch * P1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int m1 = G.m - 1;
  // stage the padded tile with asynchronous copies (cp.async): every row
  // copy is issued before the single wait, so a warp keeps all of its rows'
  // loads in flight instead of one load-store round trip per row
  {
    const int rows = P1 * P2;
    int r = warp, y = r % P1, z = r / P1;
    for (; r < rows; r += nwarps) {
      const int gy = D >= 2 ? wrap_any(o1 + G.sh[1] - m1 + y, G.Nt[1]) : 0;
      const int gz = D == 3 ? wrap_any(o2 + G.sh[2] - m1 + z, G.Nt[2]) : 0;
      const C* grow = g + int64_t(gz) * G.plane + int64_t(gy) * G.Nt[0];
      C* srow = tile + z * plane + y * pitch;
      for (int x = lane; x < P0; x += 32) {
        const int gx = wrap_any(o0 + G.sh[0] - m1 + x, G.Nt[0]);
        cp_async_elem(srow + x, grow + gx);
      }
      y += nwarps;
      while (y >= P1) {
        y -= P1;
        ++z;
      }
    }
    cp_async_wait_all();
  }
  __syncthreads();
  PolyRegs<D, L, T> P;
  if constexpr (!TABLE) P.load(G.coeffs, lane);
  const int ix = lane % L, ry = lane / L;
  const bool xact = ry < LN::RY;
  for (int i = task.y + warp; i < task.z; i += nwarps) {
    const int4 nd = __ldg(Nd.node4 + i);
    T W[LN::NW];
    node_weights<D, L, T, TABLE>(Nd, P, i, lane, W);
    const T wx = wsel<D, L>(W, ix);
    const int px = nd.x - o0 + ix, py = nd.y - o1;
    int row[LN::NSTEP];
    T wxy[LN::NSTEP];
#pragma unroll
    for (int s = 0; s < LN::NSTEP; ++s) {
      const int iy = s * LN::RY + ry;
      const bool ok = xact && iy < L;
      const int iyc = ok ? iy : 0;
      const T wy = wsel<D, L>(W, L + iyc);  // every lane shuffles
      row[s] = (py + iyc) * pitch + px;
      wxy[s] = ok ? wx * wy : T(0);
    }
    T ar = T(0), ai = T(0);
    if constexpr (D == 2) {
#pragma unroll
      for (int s = 0; s < LN::NSTEP; ++s) {
        const C v = tile[row[s]];
        ar = fma(wxy[s], v.x, ar);
        ai = fma(wxy[s], v.y, ai);
      }
    } else {
      const C* pl = tile + (nd.z - o2) * plane;
#pragma unroll
      for (int iz = 0; iz < L; ++iz) {
        const T wz = wsel<D, L>(W, 2 * L + iz);
#pragma unroll
        for (int s = 0; s < LN::NSTEP; ++s) {
          const C v = pl[iz * plane + row[s]];
          const T w = wxy[s] * wz;
          ar = fma(w, v.x, ar);
          ai = fma(w, v.y, ai);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ar += __shfl_xor_sync(0xFFFFFFFFu, ar, o);
      ai += __shfl_xor_sync(0xFFFFFFFFu, ai, o);
    }
    if (lane == 0) {
      C r;
      r.x = ar;
      r.y = ai;
      fhat[nd.w] = r;
    }
  }
}

// ---------------------------------------------------------------------------
// Shape-specialised 3-D FP32 gather (m = 4, the tiles of tile3.cuh).  One CTA
// per spreading task; a tile whose padded box lies inside the grid is brought
// into shared memory by one bulk tensor copy (TMA, completion on an
// mbarrier), and each half-warp then interpolates one node at a time from
// shared memory: lane (x = lane mod 8, row = lane / 8 mod 2) reads its 8 z values of
// rows iy, iy + 2, iy + 4 and iy + 6 at constant offsets (32 loads, one
// wavefront each), sums over z and weights by phi_x phi_y; the half-warp adds the
// 16 partial sums of two nodes at once.  Window values come straight from the
// table (broadcast loads, two nodes to a wavefront): shuffles share the
// shared-memory pipe with the tile reads.  Tiles whose box wraps around the
// grid gather their nodes straight from L1/L2 as interp_kernel does.  The wait for
// the copy is bounded: on timeout the CTA raises status word 1 (reported by
// nfft_sync) and skips its nodes.
// Bound: 41.7 shared-memory wavefronts per node (32 for the taps) at 82 % of one
// per clock and SM, the rest waiting for tiles; 256^3, 4.2e6 radial
// nodes: 750 (46 wavefronts, a whole warp per node) -> 686 us.

// Per-warp staging of the TMA gather: NK nodes per group, WCH 16-byte chunks
// of window data per node (24 table values, or the 4 fractional offsets),
// one slot = NK records + NK window blocks; two slots per warp.
template <bool TABLE> struct Tile3Gather {
  static constexpr int NK = 4;
  static constexpr int WCH = TABLE ? 6 : 1;
  // records, window values (copied from the table, or evaluated by Horner
  // from the fractional offsets staged behind them)
  static constexpr int SLOT = NK * (16 + 96 + (TABLE ? 0 : 16));
  static constexpr int NS = 2;  // (3 slots measured the same, 4 cost a CTA per SM)
  static constexpr size_t STAGE_BYTES = size_t(kInterpThreads / 32) * NS * SLOT;
};

template <int BX, int BY, int BZ, bool TABLE>
__global__ void __launch_bounds__(kInterpThreads, 4) interp_tile3_kernel(const __grid_constant__ CUtensorMap tmap,
                                                                       Geom<float> G, Nodes<float> Nd,
                                                                       const int4* __restrict__ tasks,
                                                                       const float2* __restrict__ g,
                                                                       float2* __restrict__ fhat, int* status,
                                                                       int pf_dist) {
  using TC = Tile3<BX, BY, BZ>;
  using LN = Lanes<3, 8>;
  constexpr int PITCH = TC::PITCH, PLANE = TC::PLANE;
  constexpr unsigned BOX_BYTES = unsigned(2 * PITCH) * 4u * TC::P1 * TC::P2;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float2* tile = reinterpret_cast<float2*>(smem_raw);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + TC::ACC_BYTES);
  const int4 task = tasks[blockIdx.x];
  const int t = task.x;
  const int tc0 = t % G.ntiles[0];
  const int tc1 = (t / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = t / (G.ntiles[0] * G.ntiles[1]);
  const int o0 = tc0 * BX, o1 = tc1 * BY, o2 = tc2 * BZ;
  // the tile's origin in the (possibly centred) grid; a whole number of tiles
  const int q0 = wrap_once(o0 + G.sh[0], G.Nt[0]), q1 = wrap_once(o1 + G.sh[1], G.Nt[1]);
  const int q2 = wrap_once(o2 + G.sh[2], G.Nt[2]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NWARPS = kInterpThreads / 32;
  PolyRegs<3, 8, float> P;
  if constexpr (!TABLE) P.load(G.coeffs, lane);
  const unsigned tile_s = static_cast<unsigned>(__cvta_generic_to_shared(tile));
  const unsigned mbar_s = static_cast<unsigned>(__cvta_generic_to_shared(mbar));
  // the bulk copy's shared-memory destination must be 128-byte aligned
  if (!tile3_interior<BX, BY, BZ>(G, q0, q1, q2) || (tile_s & 127u) != 0) {
    for (int64_t i = task.y + warp; i < task.z; i += NWARPS) interp_node<3, 8, float, TABLE>(G, Nd, P, i, lane, g, fhat);
    return;
  }
  // Warp w takes the nodes task.y + NK w + NK NWARPS j + k, k < NK: the NK
  // nodes' partial sums are reduced together (transposed butterfly: 3
  // shuffles per node and component instead of 5).  The node records and
  // window data (table values, or fractional offsets for Horner) of the next
  // group are copied into the warp's other stage slot by cp.async while this
  // group is summed; the first group's while the tile arrives.
  constexpr int NK = Tile3Gather<TABLE>::NK, WCH = Tile3Gather<TABLE>::WCH, SLOT = Tile3Gather<TABLE>::SLOT;
  constexpr int NS = Tile3Gather<TABLE>::NS;
  // a half-warp per node: column lane mod 8, rows ry, ry + 2, ry + 4, ry + 6
  const int ix = lane & 7, ry = (lane >> 3) & 1, half = lane >> 4;
  unsigned char* stage_base = smem_raw + TC::ACC_BYTES + 16 + warp * NS * SLOT;
  // this lane's copy in a stage: window chunk c of node k (lanes < NK WCH)
  // or the record of node lane - 24 (lanes 24 .. 24 + NK - 1); node indices
  // within a task fit in 32 bits
  const bool win_lane = lane < NK * WCH, rec_lane = lane >= 24 && lane < 24 + NK;
  const int cp_k = win_lane ? lane / WCH : lane - 24, cp_c = win_lane ? lane % WCH : 0;
  const int cp_dst = win_lane ? (TABLE ? NK * 16 + cp_k * 96 + 16 * cp_c : NK * (16 + 96) + 16 * cp_k) : 16 * cp_k;
  auto stage = [&](int buf, int gbase) {
    const int id = gbase + cp_k;
    if ((win_lane || rec_lane) && id < task.z) {
      const float4* src = win_lane ? reinterpret_cast<const float4*>(TABLE ? Nd.wtab + int64_t(id) * 24 + 4 * cp_c
                                                                              : Nd.frac4 + 4 * int64_t(id))
                                   : reinterpret_cast<const float4*>(Nd.node4 + id);
      cp_async_elem(reinterpret_cast<float4*>(stage_base + buf * SLOT + cp_dst), src);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int b = 0; b + 1 < NS; ++b) stage(b, task.y + NK * warp + b * NK * NWARPS);
  if (threadIdx.x == 0) {
    mbar_init(mbar_s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_expect_tx(mbar_s, BOX_BYTES);
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(tile_s),
        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(2 * (q0 - 4)), "r"(q1 - 3), "r"(q2 - 3), "r"(mbar_s)
        : "memory");
  } else if (threadIdx.x == 32 && pf_dist > 0 && blockIdx.x + unsigned(pf_dist) < gridDim.x) {
    // the tile of the task about one wave of resident CTAs ahead, fetched
    // into L2 now so that its CTA's bulk copy need not wait on DRAM
    const int tn = tasks[blockIdx.x + pf_dist].x;
    if (tn != t) {
      const int p0 = wrap_once((tn % G.ntiles[0]) * BX + G.sh[0], G.Nt[0]);
      const int p1 = wrap_once(((tn / G.ntiles[0]) % G.ntiles[1]) * BY + G.sh[1], G.Nt[1]);
      const int p2 = wrap_once((tn / (G.ntiles[0] * G.ntiles[1])) * BZ + G.sh[2], G.Nt[2]);
      if (tile3_interior<BX, BY, BZ>(G, p0, p1, p2))
        asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                         reinterpret_cast<uint64_t>(&tmap)),
                     "r"(2 * (p0 - 4)), "r"(p1 - 3), "r"(p2 - 3)
                     : "memory");
    }
  }
  if (!mbar_wait_bounded(mbar_s, 0)) {  // no copy into shared memory outlives the CTA, as far as another bounded wait can tell
    if (lane == 0) atomicOr(status, 1);
    asm volatile("cp.async.wait_all;" ::: "memory");
    mbar_wait_bounded(mbar_s, 0);
    return;
  }
  int buf = 0;
  const int lane_off = ry * PITCH + ix + 1;  // the lane's tap in the window
  for (int base = task.y + NK * warp; base < task.z; base += NK * NWARPS) {
    stage(buf == 0 ? NS - 1 : buf - 1, base + (NS - 1) * NK * NWARPS);
    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");  // this group's slot has landed
    __syncwarp();
    unsigned char* st = stage_base + buf * SLOT;
    if constexpr (!TABLE) {
      // the group's 4 x 24 window values, three per lane: value q = lane + 32 r
      // is column q mod 8 = lane mod 8 (the lane's coefficients) of dimension
      // (q mod 24) / 8 of node q / 24, evalpoly(frac - 1/2, coefficients)
      const float* fr = reinterpret_cast<const float*>(st + NK * (16 + 96));
      float* wv = reinterpret_cast<float*>(st + NK * 16);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int q = lane + 32 * r, k = q / 24, d = (q % 24) / 8;
        if (base + k < task.z) wv[q] = P.eval(0, fr[4 * k + d]);
      }
      __syncwarp();
    }
    const int4* rec = reinterpret_cast<const int4*>(st);
    const float* win = reinterpret_cast<const float*>(st + NK * 16);
    float ar[NK / 2], ai[NK / 2];
    // node k's partial sums (tail groups: nodes past the task end add zero)
    auto node = [&](int j, bool valid) {
      const int k = 2 * j + half;
      const int4 nd = rec[k];
      // window values: x at the lane's column, y at its four rows, all 8 z
      const float* wt = win + k * 24;
      const float wx = wt[ix];
      float wy[4], wz[8];
#pragma unroll
      for (int r = 0; r < 4; ++r) wy[r] = wt[8 + ry + 2 * r];
      const float4 z0 = *reinterpret_cast<const float4*>(wt + 16);
      const float4 z1 = *reinterpret_cast<const float4*>(wt + 20);
      wz[0] = z0.x, wz[1] = z0.y, wz[2] = z0.z, wz[3] = z0.w;
      wz[4] = z1.x, wz[5] = z1.y, wz[6] = z1.z, wz[7] = z1.w;
      // (a node past the task end reads tap 0 of the tile and is dropped)
      // (the tile's origin first: PLANE times a grid index need not fit in 32 bits)
      const float2* bp = tile + (valid ? (nd.z - o2) * PLANE + (nd.y - o1) * PITCH + (nd.x - o0) + lane_off : 0);
      float sr[4], si[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) sr[r] = si[r] = 0.f;
#pragma unroll
      for (int iz = 0; iz < 8; ++iz)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float2 v = bp[iz * PLANE + 2 * r * PITCH];
          sr[r] = fmaf(wz[iz], v.x, sr[r]);
          si[r] = fmaf(wz[iz], v.y, si[r]);
        }
      float tr = 0.f, ti = 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        tr = fmaf(wy[r], sr[r], tr);
        ti = fmaf(wy[r], si[r], ti);
      }
      ar[j] = valid ? wx * tr : 0.f;
      ai[j] = valid ? wx * ti : 0.f;
    };
    if (base + NK <= task.z) {
#pragma unroll
      for (int j = 0; j < NK / 2; ++j) node(j, true);
    } else {
#pragma unroll
      for (int j = 0; j < NK / 2; ++j) node(j, base + 2 * j + half < task.z);
    }
    // transposed reduction within the half-warps: lanes l = 0, 8 (mod 16) end
    // with pair (l / 8) mod 2's node l / 16
    const bool e = (lane & 8) != 0;
    float sr = (e ? ar[1] : ar[0]) + __shfl_xor_sync(0xFFFFFFFFu, e ? ar[0] : ar[1], 8);
    float si = (e ? ai[1] : ai[0]) + __shfl_xor_sync(0xFFFFFFFFu, e ? ai[0] : ai[1], 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xFFFFFFFFu, sr, o);
      si += __shfl_xor_sync(0xFFFFFFFFu, si, o);
    }
    const int kk = 2 * int(e) + half;
    if ((lane & 7) == 0 && base + kk < task.z) fhat[rec[kk].w] = make_float2(sr, si);
    __syncwarp();  // the slot is read before it is staged again
    buf = buf + 1 == NS ? 0 : buf + 1;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int BX, int BY, int BZ>
int interp_tile3_launch(const nfft_plan* p, const CUtensorMap* map, const Geom<float>& G, const Nodes<float>& Nd,
                        const float2* g, float2* fhat) {
  using TC = Tile3<BX, BY, BZ>;
  const size_t smem =
      TC::ACC_BYTES + 16 + (p->wtab ? Tile3Gather<true>::STAGE_BYTES : Tile3Gather<false>::STAGE_BYTES);
  auto kern = p->wtab ? interp_tile3_kernel<BX, BY, BZ, true> : interp_tile3_kernel<BX, BY, BZ, false>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 0;
  kern<<<unsigned(p->n_tasks), kInterpThreads, smem, p->stream>>>(*map, G, Nd, p->tasks, g, fhat, p->dflag + 1,
                                                                   p->gather_pf * sms);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

// Whether the kernel above is the right one for an m = 4 plan.  It moves tiles
// inside the grid only (nodes of wrapping tiles gather from L1, on one CTA per
// task), so it wants few nodes in wrapping tiles (counted by nodes!), fewer
// still where gather3.cu has many nodes per task to pay for its own tiles; with
// under 20 nodes per task, 13 where there are 25 tasks for every SM, the direct
// gather is faster (forward, device us here / direct, uniform nodes: 64^3, 2048 tasks, 16 /
// 20 / 23 nodes per task 32.4 / 30.9, 34.9 / 34.6, 37.4 / 37.9; 80^3, 4000 tasks, 12 / 16 / 23 68 /
// 67, 72 / 73, 80 / 90; 100^3, 8125 tasks, 9 / 12 / 15 / 23 132 / 130, 135 / 143, 140 / 147, 153 /
// 170; 128^3, 16,384 tasks, 8 / 12 / 16 / 23 162 / 144, 171 / 170, 180 / 192, 202 / 237).  Forward, us, here /
// gather3.cu / direct: 128^3, 10^6 uniform nodes, 23 % in wrapping tiles 351 / 371 /
// 477; 64^3, 43 %: 100,000 nodes 64 / 71 / 72, 10^6 351 / 212 / 382; 240 x 216 x 180 grid
// (not centred), 10^6 radial nodes 495 / 331 / 495; 256^3 grid, 8192 tasks, 100,000
// nodes 175 / - / 156, 300,000 207 / - / 220.
bool tile3_pays(const nfft_plan* p) {
  if (p->M < (p->n_tasks >= 25 * int64_t(p->sms) ? 13 : 20) * p->n_tasks) return false;
  if (p->bs[1] != 8 || p->bs[0] > 16) return true;  // tile shapes that gather3.cu does not have
  const int64_t w = p->wrap_nodes;
  return 4 * w <= p->M || (2 * w <= p->M && p->M < 96 * p->n_tasks);
}

// The TMA-tiled 3-D gather when the plan has one of the fixed tile shapes and
// the grid's tensor map can be made; -1 = not applicable.
int interp_tile3(const nfft_plan* cp, const Geom<float>& G, const Nodes<float>& Nd, const float2* g, float2* fhat) {
  nfft_plan* p = const_cast<nfft_plan*>(cp);  // the tensor-map cache only
  if (!p->gather_tma || !p->tasks || p->n_tasks == 0 || !tile3_shape(p)) return -1;
  void* gv = const_cast<float2*>(g);
  const int64_t bx = p->bs[0], by = p->bs[1];
  const CUtensorMap* map = nullptr;
  if (bx == 16 && by == 8) return (map = tile3_map<16, 8, 8>(p, gv)) ? interp_tile3_launch<16, 8, 8>(p, map, G, Nd, g, fhat) : -1;
  if (bx == 16 && by == 16)
    return (map = tile3_map<16, 16, 8>(p, gv)) ? interp_tile3_launch<16, 16, 8>(p, map, G, Nd, g, fhat) : -1;
  if (bx == 32 && by == 8) return (map = tile3_map<32, 8, 8>(p, gv)) ? interp_tile3_launch<32, 8, 8>(p, map, G, Nd, g, fhat) : -1;
  if (bx == 8 && by == 8) return (map = tile3_map<8, 8, 8>(p, gv)) ? interp_tile3_launch<8, 8, 8>(p, map, G, Nd, g, fhat) : -1;
  return -1;
}

// D = 2: one warp per task (warp2.cuh); blockIdx.y: column of a multi-column launch.
template <int L, typename T, bool TABLE>
__global__ void __launch_bounds__(32) gather_warp2_kernel(Geom<T> G, Nodes<T> Nd, const int4* __restrict__ tasks,
                                                          const typename Cplx<T>::type* __restrict__ g,
                                                          typename Cplx<T>::type* __restrict__ fhat, int pitch,
                                                          int64_t gcol, int64_t fcol,
                                                          const __grid_constant__ WinPoly<L, T, TABLE> wp) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  gather_warp2_body<L, T, TABLE>(G, Nd, __ldg(tasks + blockIdx.x), g + blockIdx.y * gcol, fhat + blockIdx.y * fcol,
                                 pitch, wp.c, smem_raw);
}

// -1: not applicable (no task list, tile too large, or too few nodes per
// task to pay for bringing their tile into shared memory).
template <int L, typename T, bool TABLE>
int gather_warp2_launch(const nfft_plan* p, const Geom<T>& G, const Nodes<T>& Nd, const typename Cplx<T>::type* g,
                        typename Cplx<T>::type* fhat, int ncols, int64_t gcol, int64_t fcol) {
  using W = Warp2<L, T, TABLE>;
  if (!p->tasks || p->n_tasks == 0) return -1;
  const int P0 = int(p->bs[0]) + L - 1, P1 = int(p->bs[1]) + L - 1;
  if (p->M * 256 < p->n_tasks * int64_t(P0) * P1) return -1;
  // (few nodes: a warp per node spreads them over more SMs, which in FP64 is
  // what counts: the window values alone are 2 L (L + 1) operations of a unit with
  // two lanes per SM.  Forward, us tiled / direct, POLYNOMIAL: 3,000 radial nodes, 64 x 56,
  // m = 5, FP64 145 / 65; FP64, 16,384 nodes, 64 x 56: m = 3 1.06 times as
  // fast, m = 5 0.89, m = 8 0.77; 60,000 nodes, 300 x 263 (86 per task): m = 5 266 / 283,
  // m = 8 1.02; 900 x 788 (11 per task): m = 5 1932 / 1913)
  // (also with several columns: 8 and 64 of 3,000 nodes; 2 of 6,000 and 4 of 4,200, forward + adjoint 0.93 to 0.96 times as fast)
  if (sizeof(T) == 8 && (p->M < 4096 || (ncols > 1 && p->M * p->task_columns < 20480))) return -1;
  if (!tasks_suit(p, sizeof(T) == 8 && L <= 6 ? 2 : 1)) return -1;
  // FP32, few nodes: a task's first loads (tile, records, window values) take longer than a
  // warp per node needs for all of them.  Forward, device us tiled / direct: 4,200 nodes, 14^2
  // m = 5 14.4 / 10.7, 400^2 radial m = 3 24.8 / 21.0; 8,000 nodes 14.5 / 12.0, 25.2 / 22.2; 16,000
  // 14.8 / 13.7, 25.1 / 23.4, 128^2 uniform m = 5 11.7 / 12.4; m = 8, 44^2, 8,000 16.9 / 14.9, 16,000 16.9 /
  // 17.9, 20,000 16.9 / 19.4.
  if (ncols == 1 && (p->M < (sizeof(T) == 8 ? 4096 : L >= 14 ? 10240 : 14336) ||
                     (sizeof(T) == 8 && (p->M < (L >= 10 ? 49152 : 16384) || p->M < 12 * p->n_tasks))))
    return -1;
  const int pitch = warp2_plan_pitch<L, T, TABLE>(p);
  const size_t smem = W::GATHER_STAGE + 2 * sizeof(T) * size_t(pitch) * P1;
  if (smem > 227 * 1024) return -1;
  WinPoly<L, T, TABLE> wp{};
  if constexpr (!TABLE)
    for (int q = 0; q < L * (L + 1); ++q) wp.c[q] = T(p->coeffs_host[q]);
  auto kern = gather_warp2_kernel<L, T, TABLE>;
  NFFT_CUDA_TRY(allow_smem(kern, smem));
  kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols)), 32, smem, p->stream>>>(G, Nd, p->tasks, g, fhat, pitch, gcol,
                                                                            fcol, wp);
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

// D = 1 (line1.cuh).  A tile row of 1024 points is 8 KB: with fewer than 32 nodes per
// task the nodes read the grid themselves.
template <int L, typename T, bool TABLE>
int gather_line_launch(const nfft_plan* p, const Geom<T>& G, const Nodes<T>& Nd, const typename Cplx<T>::type* g,
                       typename Cplx<T>::type* fhat, int ncols, int64_t gcol, int64_t fcol) {
  LinePoly<L, T, TABLE> wp{};
  if constexpr (!TABLE)
    for (int q = 0; q < L * (L + 1); ++q) wp.c[q] = T(p->coeffs_host[q]);
  // forward, device us, a thread / a lane per tap: 1,000 nodes, 256 points m = 5 22.8 / 20.6, m = 8 28.8 /
  // 21.5, 400,000 points 131.9 / 124.6; 4,000 nodes m = 5 23.0 / 22.2, m = 8 28.8 / 23.8; 10,000 no difference
  if constexpr (sizeof(T) == 8 && !TABLE && L >= 10)
    if (ncols == 1 && p->M < 6144) {
      const int64_t per = kLineWarps * Lanes<1, L>::NPW;
      gather_lanes_kernel<L, T><<<unsigned((p->M + per - 1) / per), kLineThreads, 0, p->stream>>>(G, Nd, g, fhat);
      NFFT_LAUNCH_CHECK();
      return NFFT_OK;
    }
  const size_t smem = 2 * sizeof(T) * size_t(p->bs[0] + L - 1);
  // (and with few tasks per SM the nodes spread better without them: FP64, m = 8,
  // 20,000 nodes 1.1 times as fast.  Forward, device us with tiles / without, FP32: 32,000 nodes in
  // about 40 tasks, m = 3 7.1 / 5.9, m = 8 10.3 / 6.3; 64,000 in 64 7.4 / 5.9, 10.4 / 6.7; 1024 tasks of
  // 31 nodes 12.8 / 12.0, 15.3 / 12.5)
  if (p->tasks && p->n_tasks > 0 && p->M >= 32 * p->n_tasks && p->M >= (sizeof(T) == 8 ? 131072 : 16384) &&
      3 * p->n_tasks >= 2 * int64_t(p->sms) && smem <= 227 * 1024) {
    auto kern = gather_line_kernel<L, T, TABLE, true>;
    NFFT_CUDA_TRY(allow_smem(kern, smem));
    // phases of the scattered stores: about 32 MB of output each from 64 MB on
    // (2^24 nodes, 134 MB: 478 us in one phase, 291 in four; forward + adjoint
    // 1356 / 1245 / 1233 / 1298 us with 1 / 2 / 4 / 8, 2^23 nodes 639 / 624 / 615 / 649)
    const int64_t out = int64_t(2 * sizeof(T)) * p->M;
    int64_t phases = out >= (int64_t(64) << 20) ? (out + (int64_t(32) << 20) - 1) / (int64_t(32) << 20) : 1;
    phases = std::max<int64_t>(1, std::min<int64_t>(phases, p->M / (p->n_tasks * 64)));
    kern<<<dim3(unsigned(p->n_tasks), unsigned(ncols), unsigned(phases)), kLineThreads, smem, p->stream>>>(
        G, Nd, p->tasks, g, fhat, gcol, fcol, wp);
  } else {
    // (few nodes: one warp per CTA, so that they reach all SMs)
    const int nt = p->M < int64_t(kLineThreads) * p->sms ? 32 : kLineThreads;
    const unsigned blocks = unsigned((p->M + nt - 1) / nt);
    gather_line_kernel<L, T, TABLE, false><<<dim3(blocks, unsigned(ncols)), nt, 0, p->stream>>>(
        G, Nd, nullptr, g, fhat, gcol, fcol, wp);
  }
  NFFT_LAUNCH_CHECK();
  return NFFT_OK;
}

// ncols columns in one launch (blockIdx.y): grids g + c gcol, values fhat + c fcol.
template <int D, int L, typename T>
int interp_launch(const nfft_plan* p, const void* g, void* fhat, int ncols, int64_t gcol, int64_t fcol) {
  Geom<T> G = make_geom<T>(p);
  Nodes<T> Nd = make_nodes<T>(p);
  if (Nd.M == 0) return NFFT_OK;
  using C = typename Cplx<T>::type;
  const C* gp = static_cast<const C*>(g);
  C* fp = static_cast<C*>(fhat);
  if constexpr (D == 1) {
    // FP32 TENSOR plans: as in the spreader (spread.cu), Horner instead of the table's rows
    return p->wtab && !(sizeof(T) == 4 && G.mode == WIN_POLY)
               ? gather_line_launch<L, T, true>(p, G, Nd, gp, fp, ncols, gcol, fcol)
               : gather_line_launch<L, T, false>(p, G, Nd, gp, fp, ncols, gcol, fcol);
  } else {
    const int64_t per_block = kInterpThreads / 32;
    int64_t blocks = (Nd.M + per_block - 1) / per_block;
    int dev = 0, sms = 1;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                  cudaSuccess || sms < 1)
      sms = 1;
    const int64_t cap = (int64_t(sms) * 64 + ncols - 1) / ncols;
    if (blocks > cap) blocks = cap;
    if constexpr (D == 2) {
      const int rc = p->wtab ? gather_warp2_launch<L, T, true>(p, G, Nd, gp, fp, ncols, gcol, fcol)
                             : gather_warp2_launch<L, T, false>(p, G, Nd, gp, fp, ncols, gcol, fcol);
      if (rc != -1) return rc;
    }
    if (ncols > 1) {
      const dim3 grid{unsigned(blocks), unsigned(ncols), 1u};
      if (p->wtab)
        interp_kernel<D, L, T, true, true><<<grid, kInterpThreads, 0, p->stream>>>(G, Nd, gp, fp, gcol, fcol);
      else
        interp_kernel<D, L, T, false, true><<<grid, kInterpThreads, 0, p->stream>>>(G, Nd, gp, fp, gcol, fcol);
      NFFT_LAUNCH_CHECK();
      return NFFT_OK;
    }
    if constexpr (D == 3 && sizeof(T) == 8) {
      const int rc = launch_gather_double3(p, g, fhat);
      if (rc != -1) return rc;
    }
    if constexpr (D == 3 && sizeof(T) == 4) {
      const int rc = L == 8 && tile3_pays(p) ? interp_tile3(p, G, Nd, gp, fp) : launch_gather_plane3(p, g, fhat);
      if (rc != -1) return rc;
    }
    if (p->tasks && p->gather_tiled) {
      const int P1 = D >= 2 ? int(p->bs[1]) + L - 1 : 1;
      const int P2 = D == 3 ? int(p->bs[2]) + L - 1 : 1;
      const size_t smem = sizeof(C) * size_t(p->gather_pitch) * P1 * P2;
      if (smem <= 227 * 1024 && p->n_tasks > 0) {
        auto kern = p->wtab ? interp_tile_kernel<D, L, T, true> : interp_tile_kernel<D, L, T, false>;
        NFFT_CUDA_TRY(allow_smem(kern, smem));
        kern<<<unsigned(p->n_tasks), kInterpThreads, smem, p->stream>>>(G, Nd, p->tasks, gp, fp, p->gather_pitch);
        NFFT_LAUNCH_CHECK();
        return NFFT_OK;
      }
    }
    if (p->wtab)
      interp_kernel<D, L, T, true><<<unsigned(blocks), kInterpThreads, 0, p->stream>>>(G, Nd, gp, fp);
    else
      interp_kernel<D, L, T, false><<<unsigned(blocks), kInterpThreads, 0, p->stream>>>(G, Nd, gp, fp);
    NFFT_LAUNCH_CHECK();
    return NFFT_OK;
  }
}

#define NFFT_INTERP_ARGS p, g, fhat, ncols, gcol, fcol
template <int D, typename T>
int interp_dispatch_l(const nfft_plan* p, const void* g, void* fhat, int ncols, int64_t gcol, int64_t fcol) {
  switch (p->m) {
    case 2: return interp_launch<D, 4, T>(NFFT_INTERP_ARGS);
    case 3: return interp_launch<D, 6, T>(NFFT_INTERP_ARGS);
    case 4: return interp_launch<D, 8, T>(NFFT_INTERP_ARGS);
    case 5: return interp_launch<D, 10, T>(NFFT_INTERP_ARGS);
    case 6: return interp_launch<D, 12, T>(NFFT_INTERP_ARGS);
    case 7: return interp_launch<D, 14, T>(NFFT_INTERP_ARGS);
    case 8: return interp_launch<D, 16, T>(NFFT_INTERP_ARGS);
  }
  set_error("m = %d not supported (2..8)", p->m);
  return NFFT_ERR_UNSUPPORTED;
}

template <typename T>
int interp_dispatch(const nfft_plan* p, const void* g, void* fhat, int ncols, int64_t gcol, int64_t fcol) {
  switch (p->D) {
    case 1: return interp_dispatch_l<1, T>(NFFT_INTERP_ARGS);
    case 2: return interp_dispatch_l<2, T>(NFFT_INTERP_ARGS);
    case 3: return interp_dispatch_l<3, T>(NFFT_INTERP_ARGS);
  }
  return NFFT_ERR_UNSUPPORTED;
}
#undef NFFT_INTERP_ARGS

}  // namespace

int launch_interp(const nfft_plan* p, const void* g, int, void* fhat, int) {
  return p->precision == 32 ? interp_dispatch<float>(p, g, fhat, 1, 0, 0) : interp_dispatch<double>(p, g, fhat, 1, 0, 0);
}

int launch_interp_cols(const nfft_plan* p, const void* g, void* fhat, int ncols, int64_t gcol, int64_t fcol) {
  return p->precision == 32 ? interp_dispatch<float>(p, g, fhat, ncols, gcol, fcol)
                            : interp_dispatch<double>(p, g, fhat, ncols, gcol, fcol);
}

}  // namespace nfft
