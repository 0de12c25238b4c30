// The transform along v of the mixed form, pruned on both sides: only the
// occupied v columns |v| <= Lv of a band row hold data (they are all that the
// band grid stores, in the order v = -Lv ... Lv), and only the ny image columns
// are wanted.  As for the u transform, nv = K M with M = 2^m >= 2 Lv + 1, and a
// row is K twisted M-point FFTs; the output of pass k2 is one contiguous
// segment of the transformed row, entry mm being image column
// j = K (mm + hm0) + k2 + ny/2.
//
// Bound by latency at 16 warps an SM, like the u transforms: issue slots are
// busy 58-59 % of the time, the shared-memory pipe 58-62 %, DRAM 32-34 %; its
// traffic is the rows in and the segments out.  cuFFT transformed whole rows of nv points, three quarters of
// them zeros, and wrote columns that no image pixel uses.  4096^2 image, 1683
// rows x 14 planes, 1683 of 6144 columns occupied: 2.3 GB in 0.49 ms, now 1.1 GB
// in 0.35 ms (forward 0.39); 8192^2, 6.8k rows x 13 planes (14000 points, now
// 2 x 8192, k_vrow_bwd_quad): 8.1 ms, now 5.9 (forward 6.5), and the band grid
// is cleared in 1.0 instead of 2.7 ms.
#pragma once

#include "wsg_device.cuh"

namespace wsg {

struct RowArgs {
  void *band;        // [rows][P][nvs] complex: occupied v columns, v = -Lv first
  void *hv;          // [rows][P][ncol] complex: K segments of hseg
  long long nrow;    // rows x npl
  int P, npl;        // planes in the layout, planes of this pass
  int nvs, Lv, ncol, K, hseg, hm0, ny;
  const void *twM, *twB, *twQ;   // as ColArgs
};

template <int M>
struct RowCfg {
  using C = ColCfg<float, M>;
  static constexpr int TPF = C::TPF, NB = C::NB, THREADS = C::THREADS;
  static constexpr size_t smem(int K, bool full) {
    return (size_t(NB) * FftBuf<M>::value + M + (full ? size_t(K - 1) * M : size_t(K) * (TPF + 32))) *
           sizeof(float2);
  }
};

// The CTA's tables in shared memory: stage twiddles [M], then the twist factors
// [K - 1][M] (FULL) or twist bases [K][TPF] and factors [K][16][2].
template <int M, bool FULL>
struct RowTables {
  const float2 *tw, *twB, *twQ;
  // the twist factor of slot t + TPF q in pass k2 > 0 (base: bases()[k2][t])
  __device__ __forceinline__ float2 base(int k2, int t) const {
    return FULL ? float2() : twB[k2 * (M / 16) + t];
  }
  __device__ __forceinline__ float2 twist(int k2, int t, int q, float2 base) const {
    if constexpr (FULL) return twB[(k2 - 1) * M + t + (M / 16) * q];
    return cmul(twQ[(k2 * 16 + q) * 2 + (q >= 8)], base);
  }
  __device__ __forceinline__ RowTables(float2 *dst, const RowArgs &a) {
    using Cfg = RowCfg<M>;
    fill_table<float2, M, Cfg::THREADS>(dst, reinterpret_cast<const float2 *>(a.twM));
    tw = dst;
    twB = twQ = dst + M;
    if constexpr (FULL) {
      fill_twist<float2, M, Cfg::THREADS>(dst + M, reinterpret_cast<const float2 *>(a.twB),
                                          reinterpret_cast<const float2 *>(a.twQ), a.K, false);
      return;
    }
    float2 *b = dst + M, *q = b + a.K * Cfg::TPF;
    for (int i = threadIdx.x; i < a.K * Cfg::TPF; i += Cfg::THREADS)
      b[i] = reinterpret_cast<const float2 *>(a.twB)[i];
    for (int i = threadIdx.x; i < a.K * 32; i += Cfg::THREADS)
      q[i] = reinterpret_cast<const float2 *>(a.twQ)[i];
    twQ = q;
  }
};

// Band column of slot b = t + TPF q (q a constant: the lower half of the slots
// are v >= 0, the upper half v < 0), or -1 for an empty slot.
template <int M>
__device__ __forceinline__ int row_col(const RowArgs &a, int b, int q) {
  if (q < 8) return b <= a.Lv ? b + a.Lv : -1;
  return b >= M - a.Lv ? b - M + a.Lv : -1;
}

// Band rows -> transformed rows, backward (+).
template <int LOGM, bool FULL>
__global__ void __launch_bounds__(RowCfg<(1 << LOGM)>::THREADS, RowCfg<(1 << LOGM)>::THREADS <= 256 ? 2 : 1)
k_vrow_bwd(RowArgs a) {
  constexpr int M = 1 << LOGM;
  using Cfg = RowCfg<M>;
  constexpr int TPF = Cfg::TPF, NB = Cfg::NB, BL = FftBuf<M>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2 *bufall = reinterpret_cast<float2 *>(smem_raw);
  const int grp = threadIdx.x / TPF, t = threadIdx.x - grp * TPF;
  float2 *A = bufall + grp * BL;
  const RowTables<M, FULL> tb(bufall + NB * BL, a);
  __syncthreads();
  const GroupSync<TPF, Cfg::THREADS> sync{grp};
  for (long long item = (long long)blockIdx.x * NB; item < a.nrow; item += (long long)gridDim.x * NB) {
    const bool rv = item + grp < a.nrow;
    const long long row = rv ? item + grp : a.nrow - 1;
    const long long r = row / a.npl;
    const size_t at = size_t(r) * a.P + size_t(row - r * a.npl);
    const float2 *in = reinterpret_cast<const float2 *>(a.band) + at * a.nvs;
    float2 *out = reinterpret_cast<float2 *>(a.hv) + at * a.ncol;
    float2 g[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int c = row_col<M>(a, t + TPF * q, q);
      g[q] = c >= 0 ? __ldcs(in + c) : make_float2(0.0f, 0.0f);
    }
    for (int k2 = 0; k2 < a.K; ++k2) {
      float2 v[16];
      if (k2 == 0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = g[q];
      } else {
        const float2 base = tb.base(k2, t);
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = cmul(g[q], tb.twist(k2, t, q, base));
      }
      float2 o[16];
      col_fft_inplace<float2, M, TPF, +1>(v, A, tb.tw, t, o, sync);
      if (rv) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int mq = t + TPF * (q < 8 ? q : q - 16);
          const int j = a.K * mq + k2 + a.ny / 2;
          if (unsigned(j) < unsigned(a.ny)) out[k2 * a.hseg + (mq - a.hm0)] = o[q];
        }
      }
    }
  }
}

// Transformed rows -> band rows, forward (-): the transpose.
template <int LOGM, bool FULL>
__global__ void __launch_bounds__(RowCfg<(1 << LOGM)>::THREADS, RowCfg<(1 << LOGM)>::THREADS <= 256 ? 2 : 1)
k_vrow_fwd(RowArgs a) {
  constexpr int M = 1 << LOGM;
  using Cfg = RowCfg<M>;
  constexpr int TPF = Cfg::TPF, NB = Cfg::NB, BL = FftBuf<M>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2 *bufall = reinterpret_cast<float2 *>(smem_raw);
  const int grp = threadIdx.x / TPF, t = threadIdx.x - grp * TPF;
  float2 *A = bufall + grp * BL;
  const RowTables<M, FULL> tb(bufall + NB * BL, a);
  __syncthreads();
  const GroupSync<TPF, Cfg::THREADS> sync{grp};
  for (long long item = (long long)blockIdx.x * NB; item < a.nrow; item += (long long)gridDim.x * NB) {
    const bool rv = item + grp < a.nrow;
    const long long row = rv ? item + grp : a.nrow - 1;
    const long long r = row / a.npl;
    const size_t at = size_t(r) * a.P + size_t(row - r * a.npl);
    const float2 *in = reinterpret_cast<const float2 *>(a.hv) + at * a.ncol;
    float2 *out = reinterpret_cast<float2 *>(a.band) + at * a.nvs;
    float2 acc[16];
    for (int k2 = 0; k2 < a.K; ++k2) {
      float2 v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int mq = t + TPF * (q < 8 ? q : q - 16);
        const int j = a.K * mq + k2 + a.ny / 2;
        v[q] = unsigned(j) < unsigned(a.ny) ? __ldcs(in + (k2 * a.hseg + (mq - a.hm0)))
                                            : make_float2(0.0f, 0.0f);
      }
      float2 o[16];
      col_fft_inplace<float2, M, TPF, -1>(v, A, tb.tw, t, o, sync);
      if (k2 == 0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) acc[q] = o[q];
      } else {
        const float2 base = tb.base(k2, t);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          float2 w = tb.twist(k2, t, q, base);
          w.y = -w.y;
          const float2 x = cmul(o[q], w);
          acc[q].x += x.x;
          acc[q].y += x.y;
        }
      }
    }
    if (rv) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int c = row_col<M>(a, t + TPF * q, q);
        if (c >= 0) out[c] = acc[q];
      }
    }
  }
}

}  // namespace wsg
