// 2-D spreading and gathering with one warp per task (a home tile or a chunk
// of a hot one), shared by the single-plan and multi-column launches
// (spread.cu, interp.cu) and the batched ones (batch.cu).
//
// Both directions hold the tile padded by the window in shared memory.
// Spreading treats a node's L x L taps (L = 2m) as one flat list t = lane + 32
// step: tap t is column t mod L of row t div L.  With a row pitch = L (mod the
// elements of one 128-byte wavefront) tap t lies in bank t (mod the same), so
// every access of a step is free of conflicts for any L and any node, and
// L x L taps take ceil(L L / 32) steps without idle rows.  Gathering gives each
// half-warp a node of its own, 16 div L rows (one for L > 8) a step: one column per
// lane, so that the x window value is read once and multiplied in at the end, and the
// weights of two nodes share a wavefront.
//
// A warp works alone: no CTA barrier, its tasks are independent, and as many
// warps as shared memory allows hide each other's latencies.  Nodes go through
// shared memory in batches of 32 (lane = node): record (first tap's offset,
// value), window values (table rows copied by cp.async one batch ahead, or
// evaluated by Horner, lane = node).
//
// What bounds it (FP32, L = 8): shared-memory wavefronts at 89 % (gather) and
// 94 % (spread) of one per clock and SM.  A spread node takes 13.7: 8 for the
// taps' read-modify-writes, 4 for record and window values, the rest staging,
// zero fill and flush.  A gathered one takes 8.5: 4 for its taps, 2 for record and window
// values, 1.25 for the sums over the half-warp of eight nodes together, the rest
// staging.  (One node per warp and step took 14.6 and 11.6.)
// 64 slices of a 256^2 stack, 8.4e6 node values: gather 876 us straight from L1 with a
// warp per node -> 361 us from the tile with 32 lanes per node -> 269 us
// with 16; spreading 618 (with the value sort, two warps sharing a tile) -> 437
// -> 412 us; a radial 300 x 210 image with 98,304 nodes, m = 5: spreading 118 -> 13 us.
// 400,000 uniform nodes on a 512^2 grid, forward transform with 32 and with 16
// lanes per node: m = 2 41.6 -> 31.5, m = 5 56.5 -> 48.0, m = 7 83.3 -> 57.1, m = 8 74.6 ->
// 62.2 us; FP64 m = 2 224 -> 156, m = 5 570 -> 503, m = 8 1068 -> 856 us (FP64:
// 2 + 2 / (rows per lane) operations per tap instead of 3).
#pragma once

#include "spread_body.cuh"
#include "warpnode.cuh"

namespace nfft {
namespace {

// Row pitch of the padded tile: >= the padded width, = want modulo `mod`
// elements.  `limit` is the pitch beyond which the tile would not fit
// (then the plain width, with conflicts).
inline int warp2_pitch(int want, int mod, int P0, int64_t limit) {
  int pitch = P0;
  while (pitch % mod != want % mod) ++pitch;
  return pitch <= limit ? pitch : P0;
}

template <int L, typename T, bool TABLE> struct Warp2 {
  using C = typename Cplx<T>::type;
  static constexpr int NB = 32;
  static constexpr int TAPS = L * L;
  static constexpr int NSTEP = (TAPS + 31) / 32;
  static constexpr int V = 16 / int(sizeof(T));
  // staged window values of a node: x then y.  Table rows are copied as they
  // are (16-byte chunks); rows written lane = node are padded so that the
  // 16-byte stores of eight lanes fall in distinct banks.
  static constexpr int pad_row(int n) {
    while (n % V != 0 || (n / V) % 2 != 1) ++n;
    return n;
  }
  static constexpr int ROW = TABLE ? 2 * L : pad_row(2 * L);
  static constexpr int NBUF = TABLE ? 2 : 1;
  // L = 8, 16: a lane's taps of two successive steps lie in successive rows, so
  // that their y window values are one 8-byte read.  L = 8 (FP32) then has
  // rows two apart in one wavefront: pitch = 2 (mod 4) keeps those on
  // distinct banks.
  static constexpr bool PAIR = L == 8 || L == 16;
  // FP64 spreading: c times the y window values per node (the FP64 units
  // bound it: one product per row instead of one per tap)
  static constexpr int CROW = pad_row(2 * L);
  static constexpr size_t WIN_BYTES = size_t(NBUF) * NB * ROW * sizeof(T);
  struct alignas(16) Rec {
    int off, dst;
    T re, im;
  };
  static constexpr size_t REC_BYTES = NB * sizeof(Rec);
  static constexpr size_t CY_BYTES = sizeof(T) == 8 ? size_t(NB) * CROW * sizeof(T) : 0;
  static constexpr size_t GATHER_STAGE = WIN_BYTES + REC_BYTES;
  static constexpr size_t SPREAD_STAGE = WIN_BYTES + REC_BYTES + CY_BYTES;
};

// The pitch of a plan's tiles: both directions use the one that fits the spreader.
template <int L, typename T, bool TABLE> int warp2_plan_pitch(const nfft_plan* p) {
  const int P0 = int(p->bs[0]) + L - 1, P1 = int(p->bs[1]) + L - 1;
  const int64_t room = int64_t(227) * 1024 - int64_t(Warp2<L, T, TABLE>::SPREAD_STAGE);
  const bool apart = L == 8 && sizeof(T) == 4;
  return warp2_pitch(apart ? 2 : L, apart ? 4 : 128 / int(2 * sizeof(T)), P0, room / (int64_t(2 * sizeof(T)) * P1));
}

// Shared memory of the spreader for a plan's tiles.
template <int L, typename T, bool TABLE> size_t warp2_spread_bytes(const nfft_plan* p) {
  return Warp2<L, T, TABLE>::SPREAD_STAGE +
         2 * sizeof(T) * size_t(warp2_plan_pitch<L, T, TABLE>(p)) * size_t(p->bs[1] + L - 1);
}

// The polynomial window's coefficients passed by value (uniform reads hit
// the constant bank); empty for table windows.
template <int L, typename T, bool TABLE> struct WinPoly {
  T c[TABLE ? 1 : L * (L + 1)];
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One lane's node of a batch and the batch's window values.
template <int L, typename T, bool TABLE> struct Warp2Stage {
  using W = Warp2<L, T, TABLE>;
  using C = typename Cplx<T>::type;
  int4 nd;
  T fx, fy;

  // the table rows of nodes [b, b + n) into buffer buf (one commit group)
  static __device__ __forceinline__ void copy_rows(const Nodes<T>& Nd, T* win, int b, int end, int buf, int lane) {
    if constexpr (TABLE) {
      const int n = min(W::NB, end - b);
      constexpr int CH = 2 * L / W::V;  // 16-byte chunks per node
      const T* src = Nd.wtab + int64_t(b) * (2 * L);
      T* dst = win + buf * W::NB * W::ROW;
      for (int q = lane; q < n * CH; q += 32) cp_async16(dst + q * W::V, src + q * W::V);
      cp_async_commit();
    }
  }
  // the node of this lane (idle lanes: the batch's last node, in range)
  __device__ __forceinline__ void load(const Nodes<T>& Nd, int b, int end, int lane) {
    const int i = min(b + lane, end - 1);
    nd = __ldg(Nd.node4 + i);
    if constexpr (!TABLE) {
      const C f = __ldg(reinterpret_cast<const C*>(Nd.frac4 + 4 * int64_t(i)));
      fx = f.x;
      fy = f.y;
    }
  }
  // POLYNOMIAL: this lane's 2L window values, evalpoly(frac - 1/2, coefficients of column l)
  static __device__ __forceinline__ T horner(const T* c, T t) {
    T v = c[L];
#pragma unroll
    for (int i = L - 1; i >= 0; --i) v = fma(v, t, c[i]);
    return v;
  }
};

// A vector of 16 bytes of T.
template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };
__device__ __forceinline__ float4 vec16(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ double2 vec16(const double* v) { return make_double2(v[0], v[1]); }

// Window values of the lane's node into its row (POLYNOMIAL only).
template <int L, typename T>
__device__ __forceinline__ void warp2_eval_row(T* row, const T* coeffs, T fx, T fy) {
  using V = typename Vec16<T>::type;
  constexpr int VN = 16 / int(sizeof(T));
  const T tx = fx - T(0.5), ty = fy - T(0.5);
#pragma unroll
  for (int q = 0; q < 2 * L; q += VN) {
    T v[VN];
#pragma unroll
    for (int u = 0; u < VN; ++u) {
      const int l = q + u;
      v[u] = Warp2Stage<L, T, false>::horner(coeffs + (l % L) * (L + 1), l < L ? tx : ty);
    }
    *reinterpret_cast<V*>(row + q) = vec16(v);
  }
}

// Spreads one task's nodes into its padded tile and adds the tile to the grid.
// fhat: node values in the caller's order.  smem: SPREAD_STAGE bytes, then
// pitch x (bs[1] + L - 1) accumulators.
template <int L, typename T, bool TABLE>
__device__ __forceinline__ void spread_warp2_body(const Geom<T>& G, const Nodes<T>& Nd, const int4 task,
                                                  const typename Cplx<T>::type* __restrict__ fhat,
                                                  T* __restrict__ g, int pitch, const T* coeffs, unsigned char* smem) {
  using W = Warp2<L, T, TABLE>;
  using C = typename Cplx<T>::type;
  using St = Warp2Stage<L, T, TABLE>;
  constexpr bool CY = sizeof(T) == 8;
  constexpr bool PAIR = W::PAIR && !CY;
  typename W::Rec* rec = reinterpret_cast<typename W::Rec*>(smem);
  T* win = reinterpret_cast<T*>(smem + W::REC_BYTES);
  T* cy = reinterpret_cast<T*>(smem + W::REC_BYTES + W::WIN_BYTES);
  C* acc = reinterpret_cast<C*>(smem + W::SPREAD_STAGE);
  const int lane = threadIdx.x & 31;
  const int tc0 = task.x % G.ntiles[0], tc1 = task.x / G.ntiles[0];
  const int P0 = G.bs[0] + L - 1, P1 = G.bs[1] + L - 1;
  const int o0 = tc0 * G.bs[0], o1 = tc1 * G.bs[1];
  if (task.y >= task.z) return;

  St st;
  C val;
  St::copy_rows(Nd, win, task.y, task.z, 0, lane);
  st.load(Nd, task.y, task.z, lane);
  val = __ldg(fhat + st.nd.w);
  {
    const int nacc = pitch * P1;
    C zero;
    zero.x = zero.y = T(0);
    for (int q = lane; q < nacc; q += 32) acc[q] = zero;
  }
  // this lane's taps: offset in the tile, column and row in the window
  int lofs[W::NSTEP], ix[W::NSTEP], iy[W::NSTEP];
  bool act[W::NSTEP];
#pragma unroll
  for (int s = 0; s < W::NSTEP; ++s) {
    const int t = lane + 32 * s;
    act[s] = W::TAPS % 32 == 0 || t < W::TAPS;
    const int tt = act[s] ? t : W::TAPS - 1;
    iy[s] = tt / L;
    ix[s] = tt - iy[s] * L;
    if constexpr (L == 8 && PAIR) iy[s] = 4 * ((lane >> 3) & 1) + 2 * (lane >> 4) + s;
    if constexpr (L == 16 && PAIR) iy[s] = 4 * (s / 2) + 2 * (lane >> 4) + (s & 1);
    lofs[s] = iy[s] * pitch + ix[s];
  }
  int buf = 0;
  for (int b = task.y; b < task.z; b += W::NB) {
    const int n = min(W::NB, task.z - b);
    T* wb = win + buf * W::NB * W::ROW;
    typename W::Rec r;
    r.off = (st.nd.y - o1) * pitch + (st.nd.x - o0);
    r.dst = 0;
    r.re = val.x;
    r.im = val.y;
    rec[lane] = r;
    if constexpr (!TABLE) warp2_eval_row<L, T>(wb + lane * W::ROW, coeffs, st.fx, st.fy);
    const bool more = b + W::NB < task.z;
    if (more) {  // the next batch's loads overlap this batch's taps
      st.load(Nd, b + W::NB, task.z, lane);
      val = __ldg(fhat + st.nd.w);
      St::copy_rows(Nd, win, b + W::NB, task.z, buf ^ 1, lane);
    }
    if constexpr (TABLE) {
      if (more) cp_async_wait<1>();
      else cp_async_wait<0>();
    }
    __syncwarp();
    if constexpr (CY) {  // lane = node: value times the y window values
      if (lane < n) {
        const T* wr = wb + lane * W::ROW + L;
#pragma unroll
        for (int l = 0; l < L; ++l) {
          const T w = wr[l];
          *reinterpret_cast<C*>(cy + lane * W::CROW + 2 * l) = {r.re * w, r.im * w};
        }
      }
      __syncwarp();
    }
    // taps; the next node's record and weights are loaded during this node's
    int off;
    C c;
    T wx[W::NSTEP], wy[W::NSTEP];
    C cw[W::NSTEP];
    auto fetch = [&](int s) {
      off = rec[s].off;
      if constexpr (!CY) {
        c.x = rec[s].re;
        c.y = rec[s].im;
      }
      const T* row = wb + s * W::ROW;
#pragma unroll
      for (int q = 0; q < W::NSTEP; ++q) {
        wx[q] = (32 % L == 0 && q > 0) ? wx[0] : row[ix[q]];
        if constexpr (CY) cw[q] = *reinterpret_cast<const C*>(cy + s * W::CROW + 2 * iy[q]);
        else if constexpr (!PAIR) wy[q] = row[L + iy[q]];
        else if (q % 2 == 0) {
          const C v = *reinterpret_cast<const C*>(row + L + iy[q]);
          wy[q] = v.x;
          wy[q + 1] = v.y;
        }
      }
    };
    fetch(0);
    for (int s = 0; s < n; ++s) {
      C* p = acc + off;
      T vr[W::NSTEP], vi[W::NSTEP];
#pragma unroll
      for (int q = 0; q < W::NSTEP; ++q) {
        if constexpr (CY) {
          vr[q] = cw[q].x;
          vi[q] = cw[q].y;
        } else {
          vr[q] = c.x * wy[q];
          vi[q] = c.y * wy[q];
        }
      }
      T wxc[W::NSTEP];
#pragma unroll
      for (int q = 0; q < W::NSTEP; ++q) wxc[q] = wx[q];
      C a[W::NSTEP];
#pragma unroll
      for (int q = 0; q < W::NSTEP; ++q)
        if (act[q]) a[q] = p[lofs[q]];
      fetch(s + 1 < n ? s + 1 : s);
#pragma unroll
      for (int q = 0; q < W::NSTEP; ++q)
        if (act[q]) {
          a[q].x = fma(wxc[q], vr[q], a[q].x);
          a[q].y = fma(wxc[q], vi[q], a[q].y);
          p[lofs[q]] = a[q];
        }
      __syncwarp();  // another lane may read these points for the next node
    }
    __syncwarp();
    if constexpr (TABLE) buf ^= 1;
  }
  flush_tile<2, T, false, 1>(G, acc, g, o0, o1, 0, P0, P1, 1, pitch);
}

// The task's padded tile by asynchronous copies with the periodic wrap (not committed).
template <int L, typename T>
__device__ __forceinline__ void warp2_load_tile(const Geom<T>& G, const typename Cplx<T>::type* __restrict__ g,
                                                typename Cplx<T>::type* tile, int pitch, int o0, int o1, int P0, int P1,
                                                int lane) {
  using C = typename Cplx<T>::type;
  const int x0 = o0 + G.sh[0] - (L / 2 - 1), y0 = o1 + G.sh[1] - (L / 2 - 1);
  for (int x = lane; x < P0; x += 32) {
    const int gx = wrap_any(x0 + x, G.Nt[0]);
    int gy = wrap_any(y0, G.Nt[1]);
    for (int y = 0; y < P1; ++y) {
      const C* src = g + int64_t(gy) * G.Nt[0] + gx;
      if constexpr (sizeof(C) == 8) cp_async8(tile + y * pitch + x, src);
      else cp_async16(tile + y * pitch + x, src);
      gy = gy + 1 == G.Nt[1] ? 0 : gy + 1;
    }
  }
}

// Sums two values of eight nodes over the warp together (transposed
// butterfly, 18 shuffles): lane l ends with node l / 4's sums in a[0], b[0].
template <typename T> __device__ __forceinline__ void warp2_reduce8(T (&a)[8], T (&b)[8], int lane) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0, h4 = (lane & 4) != 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T sa = h16 ? a[k] : a[k + 4], sb = h16 ? b[k] : b[k + 4];
    a[k] = (h16 ? a[k + 4] : a[k]) + __shfl_xor_sync(FULL, sa, 16);
    b[k] = (h16 ? b[k + 4] : b[k]) + __shfl_xor_sync(FULL, sb, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const T sa = h8 ? a[k] : a[k + 2], sb = h8 ? b[k] : b[k + 2];
    a[k] = (h8 ? a[k + 2] : a[k]) + __shfl_xor_sync(FULL, sa, 8);
    b[k] = (h8 ? b[k + 2] : b[k]) + __shfl_xor_sync(FULL, sb, 8);
  }
  {
    const T sa = h4 ? a[0] : a[1], sb = h4 ? b[0] : b[1];
    a[0] = (h4 ? a[1] : a[0]) + __shfl_xor_sync(FULL, sa, 4);
    b[0] = (h4 ? b[1] : b[0]) + __shfl_xor_sync(FULL, sb, 4);
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    a[0] += __shfl_xor_sync(FULL, a[0], o);
    b[0] += __shfl_xor_sync(FULL, b[0], o);
  }
}

// Gathers one task's nodes from its padded tile, brought into shared memory by
// asynchronous copies with the periodic wrap.  smem: GATHER_STAGE bytes, then
// pitch x (bs[1] + L - 1) grid values.
template <int L, typename T, bool TABLE>
__device__ __forceinline__ void gather_warp2_body(const Geom<T>& G, const Nodes<T>& Nd, const int4 task,
                                                  const typename Cplx<T>::type* __restrict__ g,
                                                  typename Cplx<T>::type* __restrict__ fhat, int pitch,
                                                  const T* coeffs, unsigned char* smem) {
  using W = Warp2<L, T, TABLE>;
  using C = typename Cplx<T>::type;
  using St = Warp2Stage<L, T, TABLE>;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int NK = 8;  // nodes reduced together
  typename W::Rec* rec = reinterpret_cast<typename W::Rec*>(smem);
  T* win = reinterpret_cast<T*>(smem + W::REC_BYTES);
  C* tile = reinterpret_cast<C*>(smem + W::GATHER_STAGE);
  const int lane = threadIdx.x & 31;
  const int tc0 = task.x % G.ntiles[0], tc1 = task.x / G.ntiles[0];
  const int P0 = G.bs[0] + L - 1, P1 = G.bs[1] + L - 1;
  const int o0 = tc0 * G.bs[0], o1 = tc1 * G.bs[1];
  if (task.y >= task.z) return;
  warp2_load_tile<L, T>(G, g, tile, pitch, o0, o1, P0, P1, lane);
  cp_async_commit();
  St st;
  St::copy_rows(Nd, win, task.y, task.z, 0, lane);
  st.load(Nd, task.y, task.z, lane);
  // a half-warp per node, RP rows at a time: lane -> column, row of the step
  constexpr int RP = L <= 8 ? 16 / L : 1, NS = L / RP;
  constexpr bool PAIRS = RP == 1 || W::PAIR;  // rows of steps 2i, 2i + 1 are neighbours in a lane
  const int half = lane >> 4;
  const bool act = (lane & 15) < RP * L;
  const int ix = act ? (lane & 15) % L : L - 1, ir = act ? (lane & 15) / L : 0;
  const int iy0 = PAIRS ? ir * NS : ir;            // this lane's first row
  const int lofs = iy0 * pitch + ix, step = PAIRS ? pitch : RP * pitch;
  int buf = 0;
  for (int b = task.y; b < task.z; b += W::NB) {
    const int n = min(W::NB, task.z - b);
    T* wb = win + buf * W::NB * W::ROW;
    {
      int2 r = make_int2((st.nd.y - o1) * pitch + (st.nd.x - o0), st.nd.w);
      *reinterpret_cast<int2*>(&rec[lane]) = r;
    }
    if constexpr (!TABLE) warp2_eval_row<L, T>(wb + lane * W::ROW, coeffs, st.fx, st.fy);
    const bool more = b + W::NB < task.z;
    if (more) {
      st.load(Nd, b + W::NB, task.z, lane);
      St::copy_rows(Nd, win, b + W::NB, task.z, buf ^ 1, lane);
    }
    if (TABLE && more) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncwarp();
    for (int s0 = 0; s0 < n; s0 += NK) {
      T ar[NK / 2], ai[NK / 2];
#pragma unroll
      for (int k = 0; k < NK / 2; ++k) {
        const int s = min(s0 + 2 * k + half, n - 1);  // (nodes past the end repeat the last one and are dropped)
        const C* p = tile + rec[s].off + lofs;
        const T* row = wb + s * W::ROW;
        T sr = T(0), si = T(0), wy[NS];
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          if constexpr (!PAIRS) wy[q] = row[L + iy0 + q * RP];
          else if (q % 2 == 0) {
            const C v = *reinterpret_cast<const C*>(row + L + iy0 + q);
            wy[q] = v.x;
            wy[q + 1] = v.y;
          }
        }
        const T wx = row[ix];
        if constexpr (NS == 1) wy[0] *= wx;
#pragma unroll
        for (int q = 0; q < NS; ++q, p += step)
          if (act) {  // (idle lanes make no request)
            const C v = *p;
            sr = fma(wy[q], v.x, sr);
            si = fma(wy[q], v.y, si);
          }
        ar[k] = NS == 1 ? sr : sr * wx;
        ai[k] = NS == 1 ? si : si * wx;
      }
      // transposed butterfly within the half-warps: lane l ends with the sums
      // of pair 2 (l & 8) / 8 + (l & 4) / 4, node l / 16 of it
      const bool h8 = (lane & 8) != 0, h4 = (lane & 4) != 0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const T sa = h8 ? ar[k] : ar[k + 2], sb = h8 ? ai[k] : ai[k + 2];
        ar[k] = (h8 ? ar[k + 2] : ar[k]) + __shfl_xor_sync(FULL, sa, 8);
        ai[k] = (h8 ? ai[k + 2] : ai[k]) + __shfl_xor_sync(FULL, sb, 8);
      }
      {
        const T sa = h4 ? ar[0] : ar[1], sb = h4 ? ai[0] : ai[1];
        ar[0] = (h4 ? ar[1] : ar[0]) + __shfl_xor_sync(FULL, sa, 4);
        ai[0] = (h4 ? ai[1] : ai[0]) + __shfl_xor_sync(FULL, sb, 4);
      }
#pragma unroll
      for (int o = 2; o > 0; o >>= 1) {
        ar[0] += __shfl_xor_sync(FULL, ar[0], o);
        ai[0] += __shfl_xor_sync(FULL, ai[0], o);
      }
      const int s = s0 + 2 * (2 * int(h8) + int(h4)) + half;
      if ((lane & 3) == 0 && s < n) {
        C r;
        r.x = ar[0];
        r.y = ai[0];
        fhat[rec[s].dst] = r;
      }
    }
    __syncwarp();
    if constexpr (TABLE) buf ^= 1;
  }
}

}  // namespace
}  // namespace nfft
