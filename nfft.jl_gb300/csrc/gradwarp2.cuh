// 2-D node gradient with one warp per task, on the tile and tap layout of
// warp2.cuh: the padded tile of the forward grid in shared memory, a node's
// L x L taps as a flat conflict-free list.  A lane forms the real product
// Re(conj(w_j) g[tap]) first, so a node needs two real sums (the x and the y
// derivative) instead of two complex ones.  Window values and derivatives are
// evaluated by the lane of the node, 32 nodes at a time.
#pragma once

#include "warp2.cuh"

namespace nfft {
namespace {

template <int L, typename T> struct GradWarp2 {
  using W = Warp2<L, T, false>;
  static constexpr int ROW = W::pad_row(4 * L);  // x, y, dx, dy window values of a node
  static constexpr size_t WIN_BYTES = size_t(32) * ROW * sizeof(T);
  static constexpr size_t STAGE = W::REC_BYTES + WIN_BYTES;
};

// POLY: Horner for value and derivative with the coefficients passed by value;
// otherwise tap_weight_deriv (LUT, window function).
template <int L, typename T, bool POLY>
__global__ void __launch_bounds__(32) grad_warp2_kernel(Geom<T> G, Nodes<T> Nd, const int4* __restrict__ tasks,
                                                        const typename Cplx<T>::type* __restrict__ g,
                                                        const typename Cplx<T>::type* __restrict__ wv,
                                                        T* __restrict__ dk, int pitch,
                                                        const __grid_constant__ WinPoly<L, T, !POLY> wp) {
  using GW = GradWarp2<L, T>;
  using W = typename GW::W;
  using C = typename Cplx<T>::type;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int NK = 8;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  auto* rec = reinterpret_cast<typename W::Rec*>(smem_raw);
  T* win = reinterpret_cast<T*>(smem_raw + W::REC_BYTES);
  C* tile = reinterpret_cast<C*>(smem_raw + GW::STAGE);
  const int lane = threadIdx.x;
  const int4 task = __ldg(tasks + blockIdx.x);
  const int tc0 = task.x % G.ntiles[0], tc1 = task.x / G.ntiles[0];
  const int P0 = G.bs[0] + L - 1, P1 = G.bs[1] + L - 1;
  const int o0 = tc0 * G.bs[0], o1 = tc1 * G.bs[1];
  warp2_load_tile<L, T>(G, g, tile, pitch, o0, o1, P0, P1, lane);
  cp_async_commit();
  int lofs[W::NSTEP], ix[W::NSTEP], iy[W::NSTEP];
  bool act[W::NSTEP];
#pragma unroll
  for (int s = 0; s < W::NSTEP; ++s) {
    const int t = lane + 32 * s;
    act[s] = W::TAPS % 32 == 0 || t < W::TAPS;
    const int tt = act[s] ? t : W::TAPS - 1;
    iy[s] = tt / L;
    ix[s] = tt - iy[s] * L;
    lofs[s] = iy[s] * pitch + ix[s];
  }
  const T n0 = T(G.Nt[0]), n1 = T(G.Nt[1]);
  for (int b = task.y; b < task.z; b += 32) {
    const int n = min(32, task.z - b);
    {
      const int i = b + min(lane, n - 1);
      const int4 nd = __ldg(Nd.node4 + i);
      const C f = __ldg(reinterpret_cast<const C*>(Nd.frac4 + 4 * int64_t(i)));
      const C w = __ldg(wv + nd.w);
      typename W::Rec r;
      r.off = (nd.y - o1) * pitch + (nd.x - o0);
      r.dst = nd.w;
      r.re = w.x;
      r.im = w.y;
      rec[lane] = r;
      T* row = win + lane * GW::ROW;
      if constexpr (POLY) {
#pragma unroll
        for (int q = 0; q < 2 * L; ++q) {
          const T* c = wp.c + (q % L) * (L + 1);
          const T t = (q < L ? f.x : f.y) - T(0.5);
          T v = c[L], d = T(0);
#pragma unroll
          for (int i2 = L - 1; i2 >= 0; --i2) {
            d = fma(d, t, v);
            v = fma(v, t, c[i2]);
          }
          row[q] = v;
          row[2 * L + q] = d;
        }
      } else {
#pragma unroll 1
        for (int q = 0; q < 2 * L; ++q) {
          T v, d;
          tap_weight_deriv<T>(G, G.coeffs, q < L ? f.x : f.y, q < L ? q : q - L, v, d);
          row[q] = v;
          row[2 * L + q] = d;
        }
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    for (int s0 = 0; s0 < n; s0 += NK) {
      T ax[NK], ay[NK];
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int s = min(s0 + k, n - 1);  // (nodes past the end repeat the last one and are dropped)
        const C* p = tile + rec[s].off;
        const T wr = rec[s].re, wi = rec[s].im;
        const T* row = win + s * GW::ROW;
        T sx = T(0), sy = T(0);
#pragma unroll
        for (int q = 0; q < W::NSTEP; ++q) {
          const T wx = row[ix[q]], wy = row[L + iy[q]], dx = row[2 * L + ix[q]], dy = row[3 * L + iy[q]];
          if (act[q]) {
            const C v = p[lofs[q]];
            const T t = fma(wr, v.x, wi * v.y);
            sx = fma(dx * wy, t, sx);
            sy = fma(wx * dy, t, sy);
          }
        }
        ax[k] = sx;
        ay[k] = sy;
      }
      warp2_reduce8(ax, ay, lane);
      const int s = s0 + (lane >> 2);
      if ((lane & 3) == 0 && s < n) {
        const int64_t j = rec[s].dst;
        dk[2 * j] = n0 * ax[0];
        dk[2 * j + 1] = n1 * ay[0];
      }
    }
    __syncwarp();
  }
}

}  // namespace
}  // namespace nfft
