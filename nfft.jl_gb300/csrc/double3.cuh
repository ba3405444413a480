// 3-D FP64 gather and spreading for any window width L = 2m (the spreader is
// launched for L = 4, 6, 10, double3.cu).
//
// GB300 has two FP64 lanes per SM and clock (a warp instruction occupies them
// for 16 cycles), so both kernels are bound by the number of FP64 warp
// instructions per node and are laid out to waste few lanes and operations:
//
// Gather: the padded tile sits in shared memory; a lane takes one window row
// (node, iy) -- floor(32 / L) nodes per warp -- and sums it over x with the x
// window values in registers and over z, 2 L (L + 1) multiply-adds, then the L
// rows of a node are added by shuffles.  Polynomial windows: lane (node, l)
// evaluates column l of all three dimensions.  L = 10: 88 FP64 warp instructions a
// node (73 for the taps), where the warp-per-node gather had 150 (x-y taps over
// 30 of 32 lanes in 4 steps, half-idle evaluation, a five-step sum per node).
//
// Spreading: four warps own the tile's z planes mod 4, as in
// spread_plane3.cuh; a warp's planes of a node (two or three for L = 10) form
// one flat tap list t = lane + 32 step, so that only its last step has idle
// lanes: 34 steps a node against 40 with a list per plane.  x-y products and
// value x z window values are staged once per node.
#pragma once

#include <type_traits>

#include "spread_body.cuh"
#include "warp2.cuh"

namespace nfft {
namespace {

constexpr int kD3GatherThreads = 256;

template <int L> struct Gather3D {
  static constexpr int NPW = 32 / L;     // nodes per warp
  static constexpr int WROW = 2 * L;     // staged window values of a node: x then z
  static constexpr size_t stage_bytes() { return size_t(kD3GatherThreads / 32) * NPW * WROW * sizeof(double); }
};

// Row pitch of the gather tile in points: odd, so that eight rows' 16-byte reads fall in distinct banks.
inline int gather3d_pitch(int P0) { return P0 | 1; }

template <int L, bool TABLE>
__global__ void __launch_bounds__(kD3GatherThreads, 2) gather_double3_kernel(Geom<double> G, Nodes<double> Nd,
                                                                             const int4* __restrict__ tasks,
                                                                             const double2* __restrict__ g,
                                                                             double2* __restrict__ fhat, int pitch) {
  using GC = Gather3D<L>;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* win = reinterpret_cast<double*>(smem_raw) + warp * GC::NPW * GC::WROW;
  double2* tile = reinterpret_cast<double2*>(smem_raw + GC::stage_bytes());
  const int4 task = __ldg(tasks + blockIdx.x);
  const int tc0 = task.x % G.ntiles[0], tc1 = (task.x / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = task.x / (G.ntiles[0] * G.ntiles[1]);
  const int o0 = tc0 * G.bs[0], o1 = tc1 * G.bs[1], o2 = tc2 * G.bs[2];
  const int P0 = G.bs[0] + L - 1, P1 = G.bs[1] + L - 1, P2 = G.bs[2] + L - 1;
  const int plane = pitch * P1;
  {
    const int x0 = o0 + G.sh[0] - (L / 2 - 1), y0 = o1 + G.sh[1] - (L / 2 - 1), z0 = o2 + G.sh[2] - (L / 2 - 1);
    for (int r = warp; r < P1 * P2; r += kD3GatherThreads / 32) {
      const int z = r / P1, y = r - z * P1;
      const double2* row = g + int64_t(wrap_any(z0 + z, G.Nt[2])) * G.plane +
                           int64_t(wrap_any(y0 + y, G.Nt[1])) * G.Nt[0];
      for (int x = lane; x < P0; x += 32) cp_async16(tile + z * plane + y * pitch + x, row + wrap_any(x0 + x, G.Nt[0]));
    }
    cp_async_commit();
  }
  const int k = lane / L, l = lane - k * L;  // this lane's node of a group and window row (or column)
  const bool act = k < GC::NPW;
  double c[TABLE ? 1 : L + 1];  // column l of the polynomial window
  if constexpr (!TABLE) {
#pragma unroll
    for (int i = 0; i <= L; ++i) c[i] = __ldg(G.coeffs + l * (L + 1) + i);
  }
  cp_async_wait<0>();
  __syncthreads();
  const int step = (kD3GatherThreads / 32) * GC::NPW;
  for (int b = task.y + warp * GC::NPW; b < task.z; b += step) {
    const int i = b + k;
    const bool ok = act && i < task.z;
    int4 nd = make_int4(0, 0, 0, 0);
    double wx = 0, wy = 0, wz = 0;
    if (ok) {
      nd = __ldg(Nd.node4 + i);
      if constexpr (TABLE) {
        const double* wt = Nd.wtab + int64_t(i) * (3 * L) + l;
        wx = __ldg(wt);
        wy = __ldg(wt + L);
        wz = __ldg(wt + 2 * L);
      } else {
        const double2* fr = reinterpret_cast<const double2*>(Nd.frac4 + 4 * int64_t(i));
        const double2 f = __ldg(fr);
        const double tx = f.x - 0.5, ty = f.y - 0.5, tz = __ldg(fr + 1).x - 0.5;
        wx = wy = wz = c[L];
#pragma unroll
        for (int q = L - 1; q >= 0; --q) {
          wx = fma(wx, tx, c[q]);
          wy = fma(wy, ty, c[q]);
          wz = fma(wz, tz, c[q]);
        }
      }
    }
    __syncwarp();  // the previous group's window values have been read
    if (act) {
      win[k * GC::WROW + l] = wx;
      win[k * GC::WROW + L + l] = wz;
    }
    __syncwarp();
    double sr = 0, si = 0;
    if (ok) {
      const double2* wn = reinterpret_cast<const double2*>(win + k * GC::WROW);
      double x[L];
#pragma unroll
      for (int q = 0; q < L; q += 2) {
        const double2 v = wn[q / 2];
        x[q] = v.x;
        x[q + 1] = v.y;
      }
      const double* wzp = win + k * GC::WROW + L;
      const double2* p = tile + (nd.z - o2) * plane + (nd.y - o1 + l) * pitch + (nd.x - o0);
      for (int iz = 0; iz < L; ++iz, p += plane) {
        double rr = 0, ri = 0;
#pragma unroll
        for (int q = 0; q < L; ++q) {
          const double2 v = p[q];
          rr = fma(x[q], v.x, rr);
          ri = fma(x[q], v.y, ri);
        }
        const double w = wzp[iz];
        sr = fma(w, rr, sr);
        si = fma(w, ri, si);
      }
      sr *= wy;
      si *= wy;
    }
    // the sum over a node's L lanes, halving the span (the middle lane of an odd span waits)
#pragma unroll
    for (int span = L; span > 1; span = (span + 1) / 2) {
      const int half = (span + 1) / 2;
      const double a = __shfl_down_sync(FULL, sr, half), bb = __shfl_down_sync(FULL, si, half);
      if (l + half < span) {
        sr += a;
        si += bb;
      }
    }
    if (ok && l == 0) fhat[nd.w] = make_double2(sr, si);
  }
}

template <int L> struct Spread3D {
  static constexpr int NW = 4, THREADS = NW * 32, NB = 16;
  static constexpr int TAPS = L * L;
  static constexpr int KS = (L + NW - 1) / NW;            // planes of a node per warp (most)
  static constexpr int STEPS = (KS * TAPS + 31) / 32;     // of a warp with KS planes
  static constexpr int STEPS1 = ((KS - 1) * TAPS + 31) / 32;  // of a warp with one fewer
  static constexpr size_t XY = size_t(NB) * TAPS * 8;
  static constexpr size_t CZ = size_t(NB) * NW * KS * 16;  // value x z window value of the warps' planes
  static constexpr size_t REC = size_t(NB) * NW * 8;       // {first tap's offset, planes}
  static constexpr size_t WIN = size_t(NB) * 3 * L * 8;    // window values of a batch
  static constexpr size_t STAGE = XY + CZ + REC + WIN;
};

template <int L, bool TABLE>
__global__ void __launch_bounds__(128, 2) spread_double3_kernel(Geom<double> G, Nodes<double> Nd,
                                                                const int4* __restrict__ tasks,
                                                                const double2* __restrict__ fhat,
                                                                double* __restrict__ g, int pitch) {
  using SC = Spread3D<L>;
  constexpr int NB = SC::NB, TAPS = SC::TAPS, KS = SC::KS, STEPS = SC::STEPS;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  double* s_xy = reinterpret_cast<double*>(smem_raw);                       // [NB][TAPS]
  double2* s_cz = reinterpret_cast<double2*>(smem_raw + SC::XY);            // [NB][4][KS]
  int2* s_rec = reinterpret_cast<int2*>(smem_raw + SC::XY + SC::CZ);        // [NB][4]
  double* s_w = reinterpret_cast<double*>(smem_raw + SC::XY + SC::CZ + SC::REC);  // [NB][3L]
  double2* acc = reinterpret_cast<double2*>(smem_raw + SC::STAGE);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4 task = __ldg(tasks + blockIdx.x);
  const int tc0 = task.x % G.ntiles[0], tc1 = (task.x / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = task.x / (G.ntiles[0] * G.ntiles[1]);
  const int o0 = tc0 * G.bs[0], o1 = tc1 * G.bs[1], o2 = tc2 * G.bs[2];
  const int P0 = G.bs[0] + L - 1, P1 = G.bs[1] + L - 1, P2 = G.bs[2] + L - 1;
  const int plane = pitch * P1;
  for (int q = tid; q < plane * P2; q += SC::THREADS) acc[q] = make_double2(0, 0);
  // this lane's taps: offset in the tile and in the products, plane of the warp
  int lofs[STEPS], ixy[STEPS], kp[STEPS];
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int t = lane + 32 * s;
    kp[s] = t / TAPS;
    ixy[s] = t - kp[s] * TAPS;
    lofs[s] = 4 * kp[s] * plane + (ixy[s] / L) * pitch + ixy[s] % L;
  }
  __syncthreads();
  for (int b = task.y; b < task.z; b += NB) {
    const int n = min(NB, task.z - b);
    // window values: item (node, dimension, column)
    for (int q = tid; q < n * 3 * L; q += SC::THREADS) {
      if constexpr (TABLE) {
        s_w[q] = __ldg(Nd.wtab + int64_t(b) * (3 * L) + q);
      } else {
        const int s = q / (3 * L), r = q - s * (3 * L), d = r / L;
        const double t = __ldg(Nd.frac4 + 4 * int64_t(b + s) + d) - 0.5;
        const double* c = G.coeffs + (r - d * L) * (L + 1);
        double w = __ldg(c + L);
#pragma unroll
        for (int i = L - 1; i >= 0; --i) w = fma(w, t, __ldg(c + i));
        s_w[q] = w;
      }
    }
    // records: thread (node, warp)
    if (tid < n * 4) {
      const int s = tid >> 2, w = tid & 3;
      const int4 nd = __ldg(Nd.node4 + b + s);
      const int z0 = nd.z - o2, i0 = (w - z0) & 3;  // the warp's first window plane
      s_rec[tid] = make_int2((z0 + i0) * plane + (nd.y - o1) * pitch + (nd.x - o0), (L - i0 + 3) >> 2);
    }
    __syncthreads();
    for (int q = tid; q < n * TAPS; q += SC::THREADS) {
      const int s = q / TAPS, u = q - s * TAPS, iy = u / L;
      s_xy[q] = s_w[s * 3 * L + u - iy * L] * s_w[s * 3 * L + L + iy];
    }
    for (int q = tid; q < n * L; q += SC::THREADS) {
      const int s = q / L, i = q - s * L;
      const int4 nd = __ldg(Nd.node4 + b + s);
      const double2 c = __ldg(fhat + nd.w);
      const double w = s_w[s * 3 * L + 2 * L + i];
      s_cz[(s * 4 + ((nd.z - o2 + i) & 3)) * KS + (i >> 2)] = make_double2(c.x * w, c.y * w);
    }
    __syncthreads();
    for (int s = 0; s < n; ++s) {
      const int2 rec = s_rec[s * 4 + warp];
      const int taps = rec.y * TAPS;  // of this warp's planes
      double2* p = acc + rec.x;
      const double* xy = s_xy + s * TAPS;
      const double2* cz = s_cz + (s * 4 + warp) * KS;
      auto run = [&](auto steps) {
        constexpr int NS = decltype(steps)::value;
        double2 a[NS];
        double w[NS];
        double2 v[NS];
#pragma unroll
        for (int q = 0; q < NS; ++q)
          if (q + 1 < NS || lane + 32 * q < taps) {
            a[q] = p[lofs[q]];
            w[q] = xy[ixy[q]];
            v[q] = cz[kp[q]];
          }
#pragma unroll
        for (int q = 0; q < NS; ++q)
          if (q + 1 < NS || lane + 32 * q < taps) {
            a[q].x = fma(v[q].x, w[q], a[q].x);
            a[q].y = fma(v[q].y, w[q], a[q].y);
            p[lofs[q]] = a[q];
          }
      };
      if (L % 4 == 0 || rec.y == KS) run(std::integral_constant<int, STEPS>{});
      else run(std::integral_constant<int, SC::STEPS1 < 1 ? 1 : SC::STEPS1>{});
      __syncwarp();  // another lane may read these points for the next node
    }
    __syncthreads();
  }
  flush_tile<3, double, false, SC::NW>(G, acc, g, o0, o1, o2, P0, P1, P2, pitch);
}

}  // namespace
}  // namespace nfft
