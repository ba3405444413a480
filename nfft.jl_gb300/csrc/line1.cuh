// 1-D gather and spreading.
//
// Gather (gather_line_kernel): one thread per bin-sorted node; a task's padded
// tile row (bs + 2m - 1 grid values) sits in shared memory, a node reads its 2m
// neighbours there (about 2 wavefronts a node with random conflicts) and
// evaluates or reads its window values itself, so nothing is shuffled or
// summed across lanes.  Task lists with few nodes per tile read the grid
// directly, FP64 POLYNOMIAL plans of few nodes with a lane per tap.  Node values go back to the caller's order, 8 or 16 bytes at a time:
// when they exceed a part of L2, a task's nodes (in input order) are taken in
// phases, all tasks' first shares first, so that the stores of a phase fall
// into a window of the output that stays in L2 until its sectors are full.
//
// Spreading (spread_line_kernel): output-driven.  A CTA takes one task in
// batches of at most 512 nodes, sorts a batch by grid cell in shared memory
// (stable: ranks from warp matches and per-warp cell counts, then a scan over
// the cells), and groups of eight lanes own eight neighbouring positions: a
// group walks the sorted nodes of the 8 + 2m - 1 cells that reach them and
// each lane adds its tap in registers, plainly or with a Kahan compensation.
// No atomics, and a fixed order of additions (cell, then input order).
// 2^24 nodes on 2^23 points, L = 10, compensated: 1019 -> 668 us against one warp
// per tile whose lanes own the positions mod 32 (10 of 32 lanes on a tap); the
// instruction issue and the sort's latency bound it (31 warp instructions a node, of
// which the taps are 14; 64 % of the issue slots; 6.1 shared-memory wavefronts a node, a third
// of them bank conflicts).  Measured slower: batches of 768 nodes with four
// lanes owning eight positions (748 us).
#pragma once

#include "spread_body.cuh"
#include "warpnode.cuh"

namespace nfft {
namespace {

constexpr int kLineThreads = 256;
constexpr int kLineWarps = kLineThreads / 32;
constexpr int kLineBatch = 512;    // nodes sorted at a time
constexpr int kLineMaxTile = 1024;  // largest tile of the sorting spreader

// The polynomial window's coefficients by value (uniform reads hit the constant bank).
template <int L, typename T, bool TABLE> struct LinePoly {
  T c[TABLE ? 1 : L * (L + 1)];
};

// The 2m window values of bin-sorted node i: its table row, or evalpoly at its fractional offset.
template <int L, typename T, bool TABLE>
__device__ __forceinline__ void line_weights(const Nodes<T>& Nd, int64_t i, T frac, const T* coeffs, T (&w)[L]) {
  using C = typename Cplx<T>::type;
  if constexpr (TABLE) {
    const C* row = reinterpret_cast<const C*>(Nd.wtab + i * L);
#pragma unroll
    for (int l = 0; l < L; l += 2) {
      const C v = __ldg(row + l / 2);
      w[l] = v.x;
      w[l + 1] = v.y;
    }
  } else {
    const T t = frac - T(0.5);
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const T* c = coeffs + l * (L + 1);
      T v = c[L];
#pragma unroll
      for (int q = L - 1; q >= 0; --q) v = fma(v, t, c[q]);
      w[l] = v;
    }
  }
}

// blockIdx.y: column of a multi-column launch.  TILE: one CTA per task; otherwise
// blockIdx.x runs over the nodes and the grid is read directly.
template <int L, typename T, bool TABLE, bool TILE>
__global__ void __launch_bounds__(kLineThreads) gather_line_kernel(Geom<T> G, Nodes<T> Nd,
                                                                    const int4* __restrict__ tasks,
                                                                    const typename Cplx<T>::type* __restrict__ g,
                                                                    typename Cplx<T>::type* __restrict__ fhat,
                                                                    int64_t gcol, int64_t fcol,
                                                                    const __grid_constant__ LinePoly<L, T, TABLE> wp) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  g += blockIdx.y * gcol;
  fhat += blockIdx.y * fcol;
  const int m1 = G.m - 1;
  if constexpr (TILE) {
    C* tile = reinterpret_cast<C*>(smem_raw);
    const int4 task = __ldg(tasks + blockIdx.x);
    const int o0 = task.x * G.bs[0], P0 = G.bs[0] + L - 1;
    for (int x = threadIdx.x; x < P0; x += kLineThreads) tile[x] = __ldg(g + wrap_any(o0 + G.sh[0] - m1 + x, G.Nt[0]));
    __syncthreads();
    // phase blockIdx.z of gridDim.z: an equal share of the task's nodes
    const int64_t n = task.z - task.y;
    const int lo = task.y + int(n * blockIdx.z / gridDim.z), hi = task.y + int(n * (blockIdx.z + 1) / gridDim.z);
    for (int i = lo + int(threadIdx.x); i < hi; i += kLineThreads) {
      const int4 nd = __ldg(Nd.node4 + i);
      T w[L];
      line_weights<L, T, TABLE>(Nd, i, TABLE ? T(0) : __ldg(Nd.frac4 + 4 * int64_t(i)), wp.c, w);
      const C* p = tile + (nd.x - o0);
      C s;
      s.x = s.y = T(0);
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const C v = p[l];
        s.x = fma(w[l], v.x, s.x);
        s.y = fma(w[l], v.y, s.y);
      }
      fhat[nd.w] = s;
    }
  } else {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= Nd.M) return;
    const int4 nd = __ldg(Nd.node4 + i);
    T w[L];
    line_weights<L, T, TABLE>(Nd, i, TABLE ? T(0) : __ldg(Nd.frac4 + 4 * i), wp.c, w);
    int x = wrap_any(nd.x + G.sh[0] - m1, G.Nt[0]);
    C s;
    s.x = s.y = T(0);
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const C v = __ldg(g + x);
      s.x = fma(w[l], v.x, s.x);
      s.y = fma(w[l], v.y, s.y);
      x = x + 1 == G.Nt[0] ? 0 : x + 1;
    }
    fhat[nd.w] = s;
  }
}

// The same gather with a node's taps on neighbouring lanes (32 / G1 nodes per warp, G1 the
// power of two >= L), each lane evaluating its own column: FP64 POLYNOMIAL plans of few nodes,
// where the L (L + 1) operations of a thread's window values in a row are the whole time.
template <int L, typename T>
__global__ void __launch_bounds__(kLineThreads) gather_lanes_kernel(Geom<T> G, Nodes<T> Nd,
                                                                     const typename Cplx<T>::type* __restrict__ g,
                                                                     typename Cplx<T>::type* __restrict__ fhat) {
  using C = typename Cplx<T>::type;
  using LN = Lanes<1, L>;
  const int lane = threadIdx.x & 31, slot = lane / LN::G1, ix = lane % LN::G1;
  const bool act = ix < L;
  T c[L + 1];
#pragma unroll
  for (int q = 0; q <= L; ++q) c[q] = act ? __ldg(G.coeffs + ix * (L + 1) + q) : T(0);
  const int64_t i = (int64_t(blockIdx.x) * kLineWarps + (threadIdx.x >> 5)) * LN::NPW + slot;
  const bool ok = slot < LN::NPW && i < Nd.M;
  int4 nd = make_int4(0, 0, 0, 0);
  C s;
  s.x = s.y = T(0);
  if (ok) {
    nd = __ldg(Nd.node4 + i);
    if (act) {
      const T t = __ldg(Nd.frac4 + 4 * i) - T(0.5);
      T w = c[L];
#pragma unroll
      for (int q = L - 1; q >= 0; --q) w = fma(w, t, c[q]);
      const C v = __ldg(g + wrap_any(nd.x + G.sh[0] - G.m + 1 + ix, G.Nt[0]));
      s.x = w * v.x;
      s.y = w * v.y;
    }
  }
#pragma unroll
  for (int o = LN::G1 / 2; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xFFFFFFFFu, s.x, o);
    s.y += __shfl_xor_sync(0xFFFFFFFFu, s.y, o);
  }
  if (ok && ix == 0) fhat[nd.w] = s;
}

// A sorted node: value and tile cell.
template <typename T> struct LineNode;
template <> struct __align__(16) LineNode<float> {
  float re, im;
  int x, pad;
};
template <> struct __align__(16) LineNode<double> {
  double re, im;
  int x, pad0, pad1, pad2;
};

template <int L, typename T, bool KAHAN> struct Line1 {
  using A = typename Acc<T, KAHAN>::type;
  // shared memory of a tile of bs cells
  static size_t acc_bytes(int bs) { return (sizeof(A) * size_t(bs + L - 1) + 31) & ~size_t(31); }
  static size_t smem(int bs) {
    return acc_bytes(bs) + size_t(kLineBatch) * (sizeof(LineNode<T>) + sizeof(T) * L) +
           sizeof(int) * size_t(((bs + 7) & ~7) + 4) + sizeof(uint16_t) * size_t(kLineWarps) * ((bs + 7) & ~7);
  }
};

template <int L, typename T, bool TABLE, bool KAHAN>
__global__ void __launch_bounds__(kLineThreads) spread_line_kernel(Geom<T> G, Nodes<T> Nd,
                                                                    const int4* __restrict__ tasks,
                                                                    const typename Cplx<T>::type* __restrict__ fhat,
                                                                    T* __restrict__ g, int64_t fcol, int64_t gcol,
                                                                    const __grid_constant__ LinePoly<L, T, TABLE> wp) {
  using C = typename Cplx<T>::type;
  using A = typename Acc<T, KAHAN>::type;
  constexpr int NPT = kLineBatch / kLineThreads;  // nodes per thread and batch
  constexpr unsigned FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ int s_warp[kLineWarps];
  fhat += blockIdx.y * fcol;  // column of a multi-column launch
  g += blockIdx.y * gcol;
  const int4 task = __ldg(tasks + blockIdx.x);
  const int bs = G.bs[0], o0 = task.x * bs, P0 = bs + L - 1;
  const int cells = (bs + 7) & ~7;
  A* acc = reinterpret_cast<A*>(smem_raw);
  LineNode<T>* s_node = reinterpret_cast<LineNode<T>*>(smem_raw + ((sizeof(A) * size_t(P0) + 31) & ~size_t(31)));
  T* s_w = reinterpret_cast<T*>(s_node + kLineBatch);
  int* s_start = reinterpret_cast<int*>(s_w + kLineBatch * L);            // [cells + 1]
  uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_start + cells + 4);  // [warp][cells]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    A zero;
    memset(&zero, 0, sizeof(A));
    for (int q = tid; q < P0; q += kLineThreads) acc[q] = zero;
  }
  const int total = task.z - task.y;
  const int nbatch = (total + kLineBatch - 1) / kLineBatch;
  const int per = nbatch > 0 ? (total + nbatch - 1) / nbatch : 0;  // batches of equal size
  for (int b = task.y; b < task.z; b += per) {
    const int n = min(per, task.z - b);
    const int wn = (n + kLineWarps - 1) / kLineWarps;  // each warp ranks wn consecutive nodes
    {
      uint4* z = reinterpret_cast<uint4*>(s_cnt);
      for (int q = tid; q < kLineWarps * cells / 8; q += kLineThreads) z[q] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    int node[NPT], cell[NPT], rank[NPT];
    C val[NPT];
    T frac[NPT];
    static_assert((kLineBatch / kLineWarps + 31) / 32 <= NPT, "rounds of 32 nodes per warp");
#pragma unroll
    for (int r = 0; r < NPT; ++r) {
      const int q = r * 32 + lane;
      const int i = warp * wn + q;
      const bool ok = q < wn && i < n;
      node[r] = -1;
      cell[r] = -1;
      if (ok) {
        node[r] = b + i;
        const int4 nd = __ldg(Nd.node4 + b + i);
        cell[r] = nd.x - o0;
        val[r] = __ldg(fhat + nd.w);
        frac[r] = TABLE ? T(0) : __ldg(Nd.frac4 + 4 * int64_t(b + i));
      }
    }
#pragma unroll
    for (int r = 0; r < NPT; ++r) {
      if (r * 32 < wn) {  // (uniform in the warp)
        const unsigned peers = __match_any_sync(FULL, cell[r]);
        uint16_t* cnt = s_cnt + warp * cells;
        const int before = cell[r] >= 0 ? cnt[cell[r]] : 0;
        rank[r] = before + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (cell[r] >= 0 && (peers >> lane) == 1u) cnt[cell[r]] = uint16_t(before + __popc(peers));  // last of its cell
        __syncwarp();
      }
    }
    __syncthreads();
    // counts -> exclusive offsets over the warps; cell totals -> exclusive
    // scan.  Two cells (one 32-bit word of the counts, no carry: a batch has
    // fewer than 2^16 nodes) at a time.
    {
      constexpr int CPT = kLineMaxTile / 2 / kLineThreads;  // consecutive words per thread (most)
      const int words = cells / 2, cpt = (words + kLineThreads - 1) / kLineThreads;
      uint32_t* cnt2 = reinterpret_cast<uint32_t*>(s_cnt);
      uint32_t tot[CPT];
      int sum = 0;
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        tot[c] = 0;
        const int x = tid * cpt + c;
        if (c < cpt && x < words) {
          uint32_t run = 0;
#pragma unroll
          for (int w = 0; w < kLineWarps; ++w) {
            const uint32_t v = cnt2[w * words + x];
            cnt2[w * words + x] = run;
            run += v;
          }
          tot[c] = run;
        }
        sum += int(tot[c] & 0xFFFFu) + int(tot[c] >> 16);
      }
      int inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += v;
      }
      if (lane == 31) s_warp[warp] = inc;
      __syncthreads();
      int at = inc - sum;
#pragma unroll
      for (int w = 0; w < kLineWarps; ++w)
        if (w < warp) at += s_warp[w];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const int x = tid * cpt + c;
        if (c < cpt && x < words) {
          s_start[2 * x] = at;
          s_start[2 * x + 1] = at + int(tot[c] & 0xFFFFu);
          at += int(tot[c] & 0xFFFFu) + int(tot[c] >> 16);
        }
      }
      // (cells past the tile are empty: s_start[bs ..] = n)
      if (tid == 0) s_start[cells] = n;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NPT; ++r) {
      if (cell[r] >= 0) {
        const int pos = s_start[cell[r]] + s_cnt[warp * cells + cell[r]] + rank[r];
        LineNode<T> nd;
        nd.re = val[r].x;
        nd.im = val[r].y;
        nd.x = cell[r];
        s_node[pos] = nd;
        T w[L];
        line_weights<L, T, TABLE>(Nd, node[r], frac[r], wp.c, w);
        C* row = reinterpret_cast<C*>(s_w + pos * L);
#pragma unroll
        for (int l = 0; l < L; l += 2) row[l / 2] = {w[l], w[l + 1]};
      }
    }
    __syncthreads();
    // eight lanes own eight neighbouring positions
    for (int p0 = (tid >> 3) * 8; p0 < P0; p0 += kLineThreads) {
      const int p = p0 + (tid & 7);
      const int lo = s_start[max(0, p0 - L + 1)], hi = s_start[min(bs, p0 + 8)];
      A a;
      if (p < P0) a = acc[p];
      for (int i = lo; i < hi; ++i) {
        const LineNode<T> nd = s_node[i];
        const unsigned l = unsigned(p - nd.x);
        if (l < unsigned(L)) {
          const T w = s_w[i * L + int(l)];
          if constexpr (KAHAN) {
            kahan_add<A, T>(a, w * nd.re, w * nd.im);
          } else {
            a.x = fma(w, nd.re, a.x);
            a.y = fma(w, nd.im, a.y);
          }
        }
      }
      if (p < P0) acc[p] = a;
    }
    __syncthreads();
  }
  flush_tile<1, T, KAHAN, kLineWarps>(G, acc, g, o0, 0, 0, P0, 1, 1, P0);
}

}  // namespace
}  // namespace nfft
