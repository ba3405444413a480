// 3-D FP32 spreading by plane owners, for any window width L = 2m and tile
// shapes fixed at compile time (tile3.cuh).
//
// NW (two or four) warps share the padded tile; warp w owns its z planes = w
// mod NW, so every point has one writer and the accumulation is a plain
// read-modify-write.  A node has ceil(L / NW) or floor(L / NW) planes per warp, each a
// flat list of L x L taps t = lane + 32 step (tap t: column t mod L of row t div L),
// free of bank conflicts because the row pitch is L mod 16.  The x-y weight
// products of a node are read once per warp and used for all of its planes.
//
// Staging (16 nodes at a time, 2 NW threads per node, loads one batch ahead
// in registers): thread j of a node writes rows j, j + 2 NW, .. of the products
// and the planes' records {offset of the warp's first tap, planes, value x z
// window values of the planes}.  The tile is cleared by one bulk copy of
// zeros and, where it does not wrap around the grid, added to it by one bulk
// tensor reduction (cp.reduce.async.bulk.tensor ... .add) issued by one thread;
// wrapping tiles and grids without a tensor map use the per-point flush of
// spread_body.cuh.
//
// Bound: shared-memory wavefronts, of which a node's taps take 64 (L = 8) or 140 (L =
// 10).  L = 8: 89 per node with two warps at 86 % of one per clock and SM, 94 at 89 %
// with four (more warps read the products and records again, but fewer do not
// hide the latencies as well), 107 with eight; 256^3 radial set (4.2e6 nodes) 1.58
// (eight) -> 1.49 (four) -> 1.46 ms (two).
// L = 10: 195 (140 + 16 + 8 and the staging) with four warps against ~410 of the generic
// kernel of spread_body.cuh; 300,001 uniform nodes, 202 x 174 x 150 grid 393 -> 246 us.
#pragma once

#include "spread_body.cuh"
#include "tile3.cuh"

namespace nfft {
namespace {

template <int BX, int BY, int BZ, int L, int NW_> struct Plane3 {
  using TC = Tile3<BX, BY, BZ, L>;
  static constexpr int NW = NW_, THREADS = NW * 32;
  static constexpr int NB = 16;                     // nodes per staged batch
  static constexpr int TPN = THREADS / NB;          // threads that stage a node
  static constexpr int RPT = (L + TPN - 1) / TPN;   // window rows and planes of each
  static constexpr int TAPS = L * L;
  static constexpr int NSTEP = (TAPS + 31) / 32;
  static constexpr int KS = (L + NW - 1) / NW;      // planes of a node per warp (most)
  static constexpr int RW = ((1 + KS) * 8 + 15) / 16 * 2;  // record: float2 slots (16-byte multiple)
  // strides that keep the staging stores of neighbouring nodes in distinct banks
  static constexpr int RECS = NW * RW + 2;          // float2 slots of a node's records
  static constexpr int XYS = L % 4 == 0 ? TAPS : (TAPS + 15) / 32 * 32 + 16;  // floats of a node's products
  static constexpr size_t REC_OFF = TC::ACC_BYTES;
  static constexpr size_t XY_OFF = REC_OFF + size_t(NB) * RECS * 8;
  static constexpr size_t BAR_OFF = XY_OFF + size_t(NB) * XYS * 4;
  static constexpr size_t SMEM = BAR_OFF + 16;
  static constexpr int PER_SM = int((227 * 1024) / (SMEM + 1024)) < 1 ? 1 : int((227 * 1024) / (SMEM + 1024));
};

// The polynomial window's coefficients by value (uniform reads hit the constant bank).
template <int L, bool TABLE> struct Plane3Poly {
  float c[TABLE ? 1 : L * (L + 1)];
};

template <int L> __device__ __forceinline__ float plane3_horner(const float* c, float t) {
  float v = c[L];
#pragma unroll
  for (int i = L - 1; i >= 0; --i) v = fmaf(v, t, c[i]);
  return v;
}

template <int BX, int BY, int BZ, int L, int NW, bool TABLE>
__global__ void __launch_bounds__((Plane3<BX, BY, BZ, L, NW>::THREADS), (Plane3<BX, BY, BZ, L, NW>::PER_SM)) spread_plane3_kernel(
    const __grid_constant__ CUtensorMap tmap, int use_tma, Geom<float> G, Nodes<float> Nd,
    const int4* __restrict__ tasks, const float2* __restrict__ fhat, float* __restrict__ g, int64_t fcol, int64_t gcol,
    const float4* __restrict__ zeros, int* status, const __grid_constant__ Plane3Poly<L, TABLE> wp) {
  using TC = Tile3<BX, BY, BZ, L>;
  using PC = Plane3<BX, BY, BZ, L, NW>;
  constexpr int NB = PC::NB, PITCH = TC::PITCH, PLANE = TC::PLANE, KS = PC::KS, NSTEP = PC::NSTEP, RW = PC::RW;
  constexpr int TPN = PC::TPN, RPT = PC::RPT;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  fhat += blockIdx.y * fcol;  // column of a multi-column launch
  g += blockIdx.y * gcol;
  float2* acc = reinterpret_cast<float2*>(smem_raw);
  float2* s_rec = reinterpret_cast<float2*>(smem_raw + PC::REC_OFF);  // [NB][RECS]: 4 records
  float* s_xy = reinterpret_cast<float*>(smem_raw + PC::XY_OFF);      // [NB][XYS]
  const unsigned acc_s = static_cast<unsigned>(__cvta_generic_to_shared(acc));
  const unsigned bar_s = static_cast<unsigned>(__cvta_generic_to_shared(smem_raw + PC::BAR_OFF));
  const int4 task = tasks[blockIdx.x];
  const int tc0 = task.x % G.ntiles[0];
  const int tc1 = (task.x / G.ntiles[0]) % G.ntiles[1];
  const int tc2 = task.x / (G.ntiles[0] * G.ntiles[1]);
  const int o0 = tc0 * BX, o1 = tc1 * BY, o2 = tc2 * BZ;
  if (zeros) {
    if (threadIdx.x == 0) {
      mbar_init(bar_s, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(bar_s, unsigned(TC::NACC) * 8u);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       acc_s),
                   "l"(zeros), "r"(unsigned(TC::NACC) * 8u), "r"(bar_s)
                   : "memory");
    }
  } else {
    float4* a4 = reinterpret_cast<float4*>(acc);
    for (int q = threadIdx.x; q < TC::NACC / 2; q += PC::THREADS) a4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  bool zeroed = zeros == nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = threadIdx.x / TPN, j = threadIdx.x % TPN;  // staged node, its rows / planes j, j + TPN, ..

  int4 r_nd = make_int4(0, 0, 0, 0);
  float2 r_c = make_float2(0.f, 0.f);
  float r_x[L], r_y[RPT], r_z[RPT];
  float4 r_f = make_float4(0.f, 0.f, 0.f, 0.f);
  float cj[RPT][TABLE ? 1 : L + 1];  // Horner: coefficients of this thread's columns
#pragma unroll
  for (int i = 0; i < L; ++i) r_x[i] = 0.f;
#pragma unroll
  for (int h = 0; h < RPT; ++h) {
    r_y[h] = r_z[h] = 0.f;
    if constexpr (!TABLE) {
#pragma unroll
      for (int i = 0; i <= L; ++i) cj[h][i] = j + TPN * h < L ? __ldg(G.coeffs + (j + TPN * h) * (L + 1) + i) : 0.f;
    }
  }
  // the node's record two batches ahead (its index addresses the value), the
  // value and the window values one batch ahead
  int4 r_next = make_int4(0, 0, 0, 0);
  auto prefetch_nd = [&](int b) {
    if (b + s < task.z) r_next = __ldg(Nd.node4 + b + s);
  };
  auto prefetch = [&](int b) {
    const int i = b + s;
    if (i < task.z) {
      r_nd = r_next;
      r_c = __ldg(fhat + r_nd.w);
      if constexpr (TABLE) {
        const float* wt = Nd.wtab + int64_t(i) * (3 * L);
#pragma unroll
        for (int q = 0; q < L; q += 2) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(wt + q));
          r_x[q] = v.x;
          r_x[q + 1] = v.y;
        }
#pragma unroll
        for (int h = 0; h < RPT; ++h)
          if (j + TPN * h < L) {
            r_y[h] = __ldg(wt + L + j + TPN * h);
            r_z[h] = __ldg(wt + 2 * L + j + TPN * h);
          }
      } else {
        r_f = __ldg(reinterpret_cast<const float4*>(Nd.frac4) + i);
      }
    }
  };
  prefetch_nd(task.y);
  prefetch(task.y);
  prefetch_nd(task.y + NB);

  int lofs[NSTEP];  // this lane's taps in a plane
  bool act[NSTEP];
#pragma unroll
  for (int q = 0; q < NSTEP; ++q) {
    const int t = lane + 32 * q;
    act[q] = PC::TAPS % 32 == 0 || t < PC::TAPS;
    lofs[q] = act[q] ? (t / L) * PITCH + t % L : 0;
  }
  __syncthreads();

  for (int b = task.y; b < task.z; b += NB) {
    const int n = min(NB, task.z - b);
    if (s < n) {
      if constexpr (!TABLE) {  // evalpoly(frac - 1/2, coefficients of column l)
        const float tx = r_f.x - 0.5f, ty = r_f.y - 0.5f, tz = r_f.z - 0.5f;
#pragma unroll
        for (int l = 0; l < L; ++l) r_x[l] = plane3_horner<L>(wp.c + l * (L + 1), tx);
#pragma unroll
        for (int h = 0; h < RPT; ++h) {
          r_y[h] = plane3_horner<L>(cj[h], ty);
          r_z[h] = plane3_horner<L>(cj[h], tz);
        }
      }
      const int z0 = r_nd.z - o2;
      const int oxy = (r_nd.y - o1) * PITCH + (r_nd.x - o0 + TC::LEAD);
#pragma unroll
      for (int h = 0; h < RPT; ++h) {
        const int i = j + TPN * h;  // window row and plane
        if (L % TPN != 0 && i >= L) continue;
        float* row = s_xy + s * PC::XYS + i * L;
        if constexpr (L % 4 == 0) {
          // (L = 8: the two halves in an order that keeps the eight rows of a
          // 128-bit store phase, of one or two nodes, on distinct banks)
          const int swap = L != 8 ? 0 : TPN == 8 ? j >> 2 : s & 1;
#pragma unroll
          for (int q = 0; q < L; q += 4) {
            float4 v = make_float4(r_x[q] * r_y[h], r_x[q + 1] * r_y[h], r_x[q + 2] * r_y[h], r_x[q + 3] * r_y[h]);
            if (L == 8 && swap) v = make_float4(r_x[(q + 4) % L] * r_y[h], r_x[(q + 5) % L] * r_y[h],
                                                r_x[(q + 6) % L] * r_y[h], r_x[(q + 7) % L] * r_y[h]);
            *reinterpret_cast<float4*>(row + (q ^ (4 * swap))) = v;
          }
        } else {
#pragma unroll
          for (int q = 0; q < L; q += 2)
            *reinterpret_cast<float2*>(row + q) = make_float2(r_x[q] * r_y[h], r_x[q + 1] * r_y[h]);
        }
        // window plane i is tile plane z0 + i, owned by warp (z0 + i) mod NW
        // as its plane number i / NW
        float2* rec = s_rec + s * PC::RECS + ((z0 + i) % NW) * RW;
        rec[1 + i / NW] = make_float2(r_c.x * r_z[h], r_c.y * r_z[h]);
        if (i < NW)
          rec[0] = make_float2(__int_as_float((z0 + i) * PLANE + oxy), __int_as_float((L - i + NW - 1) / NW));
      }
    }
    __syncthreads();
    prefetch(b + NB);
    prefetch_nd(b + 2 * NB);
    if (!zeroed) {  // (bounded: on timeout the CTA raises its status bit and adds nothing)
      zeroed = __syncthreads_and(mbar_wait_bounded(bar_s, 0));
      if (!zeroed) break;
    }
    // taps: the next node's record and products are loaded during this node's
    float2 rt[1 + KS];
    float w[NSTEP];
    auto fetch = [&](int q) {
      const float4* r4 = reinterpret_cast<const float4*>(s_rec + q * PC::RECS + warp * RW);
#pragma unroll
      for (int i = 0; i < (1 + KS) / 2; ++i) {
        const float4 v = r4[i];
        rt[2 * i] = make_float2(v.x, v.y);
        rt[2 * i + 1] = make_float2(v.z, v.w);
      }
      if constexpr ((1 + KS) % 2 != 0) rt[KS] = *reinterpret_cast<const float2*>(r4 + KS / 2);
      const float* xy = s_xy + q * PC::XYS;
#pragma unroll
      for (int i = 0; i < NSTEP; ++i) w[i] = xy[act[i] ? lane + 32 * i : PC::TAPS - 1];
    };
    fetch(0);
    for (int q = 0; q < n; ++q) {
      float2* p = acc + __float_as_int(rt[0].x);
      const bool last = L % NW == 0 || __float_as_int(rt[0].y) == KS;  // this warp has KS planes of the node
      float2 cz[KS];
      float wc[NSTEP];
#pragma unroll
      for (int k = 0; k < KS; ++k) cz[k] = rt[1 + k];
#pragma unroll
      for (int i = 0; i < NSTEP; ++i) wc[i] = w[i];
      float2 a[KS][NSTEP];
#pragma unroll
      for (int k = 0; k < KS; ++k)
        if (k + 1 < KS || last) {
#pragma unroll
          for (int i = 0; i < NSTEP; ++i)
            if (act[i]) a[k][i] = p[NW * k * PLANE + lofs[i]];
        }
      fetch(q + 1 < n ? q + 1 : q);
#pragma unroll
      for (int k = 0; k < KS; ++k)
        if (k + 1 < KS || last) {
#pragma unroll
          for (int i = 0; i < NSTEP; ++i)
            if (act[i]) {
              a[k][i].x = fmaf(cz[k].x, wc[i], a[k][i].x);
              a[k][i].y = fmaf(cz[k].y, wc[i], a[k][i].y);
              p[NW * k * PLANE + lofs[i]] = a[k][i];
            }
        }
      __syncwarp();  // another lane may read these points for the next node
    }
    __syncthreads();
  }
  // a task without nodes (or a timed-out wait) still waits for its zero
  // fill, so that no copy into shared memory outlives the CTA
  if (!zeroed) zeroed = mbar_wait_bounded(bar_s, 0);
  // the tile's shared-memory writes, made visible to the bulk (async) copy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (!__syncthreads_and(zeroed)) {
    if (threadIdx.x == 0) atomicOr(status, 1);
    return;
  }
  const int q0 = wrap_once(o0 + G.sh[0], G.Nt[0]), q1 = wrap_once(o1 + G.sh[1], G.Nt[1]);
  const int q2 = wrap_once(o2 + G.sh[2], G.Nt[2]);
  if (use_tma && tile3_interior<BX, BY, BZ, L>(G, q0, q1, q2) && (acc_s & 127u) == 0) {
    if (threadIdx.x == 0) {
      // x in floats: a multiple of 4 (16 bytes)
      const int x = 2 * (q0 - TC::XOFF), y = q1 - (L / 2 - 1), z = q2 - (L / 2 - 1);
      asm volatile(
          "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
          ::"l"(reinterpret_cast<uint64_t>(&tmap)), "r"(x), "r"(y), "r"(z), "r"(acc_s)
          : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tile has been read before exit
    }
    return;
  }
  flush_tile<3, float, false, NW>(G, acc + TC::LEAD, g, o0, o1, o2, BX + L - 1, TC::P1, TC::P2, PITCH);
}

}  // namespace
}  // namespace nfft
