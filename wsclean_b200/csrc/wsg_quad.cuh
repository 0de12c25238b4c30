// 8192-point transforms in mixed precision, each as four of 2048 points.
//
// An 8192-point transform needs 512 threads of 128 registers, which is a whole
// SM: with the plain column and row kernels nothing ran beside it while it
// waited for its loads or at its ten barriers a pass.  Here the CTA's four
// groups of 128 threads each transform one residue class b = r (mod 4) of the
// inputs with barriers of their own, a last radix-4 stage joins the four
//     X[p + 2048 s] = sum_r i^(rs) w^(pr) F_r[p],   w = exp(2 pi i / 8192)
// and the next column or row is copied in meanwhile (the transposed direction
// runs the same steps backwards).  Twisted passes are as in the other kernels:
// nu = K 8192, pass k2 gives the outputs K m + k2.
//
// Bound by latency at 16 warps an SM: issue and the shared-memory pipe are busy a
// third and a half of the time, DRAM less; the column loads (16 bytes of every
// band row, rows 850 KB apart) cost the u transform some 1.5 ms of its 10.7.
// 8192^2 image, 6.8k rows, 13 planes, K = 2: u transform 13.4 -> 10.7 ms
// (transposed 11.1 -> 9.2), v transform 7.0 -> 5.9 (7.3 -> 6.5).
//
// Shared memory: four padded buffers of 2048 points, the 2048-point stage
// table, w^k for k < 2048 (the rest by quarter turns), the twist tables of the
// passes after the first and the staged input.
#pragma once

#include "wsg_rows.cuh"

namespace wsg {

struct Quad {
  static constexpr int M = 8192, S = 2048, THREADS = 512, TPF = 128;
  // (4 more than the padded length: the four buffers' banks are 8 words apart,
  // so consecutive points b, buffer b & 3, place b >> 2, do not conflict)
  static constexpr int BS = FftBuf<S>::value + 4;
  static constexpr int BUF = 4 * BS;  // entries
  // table entries: 2048-point stages, w, then per pass k2 > 0 the twist bases [512]
  // and factors [16][2]
  __host__ __device__ static constexpr int tab(int K) { return 2 * S + (K - 1) * (THREADS + 32); }

  float2 *buf, *A;  // the four buffers, the group's own
  const float2 *tw, *w1, *twist;
  int tid, grp, t;
  GroupSync<TPF, THREADS> sync;

  __device__ __forceinline__ static int at(int b) { return (b & 3) * BS + fpad(b >> 2); }

  // buffers and tables in mem (BUF + tab(K) entries); the caller's next CTA
  // barrier completes the tables
  template <typename Args>
  __device__ __forceinline__ Quad(float2 *mem, const Args &a)
      : buf(mem), tid(threadIdx.x), grp(threadIdx.x / TPF), t(threadIdx.x % TPF), sync{grp} {
    A = buf + grp * BS;
    float2 *d = mem + BUF;
    const float2 *src = reinterpret_cast<const float2 *>(a.twM);
    // the 8192-point table's stages have strides 16, 256 (both radix 16) and
    // 4096 (radix 2); 2048 points need strides 16 (the same) and 256 (radix 8)
    constexpr int O1 = TwOffset<256>::value, O2 = TwOffset<4096>::value;
    for (int i = tid; i < O1; i += THREADS) d[i] = src[i];
    for (int i = tid; i < 7 * 256; i += THREADS)
      d[O1 + i] = src[O1 + (2 * (1 + i / 256) - 1) * 256 + i % 256];
    for (int i = tid; i < S; i += THREADS) d[S + i] = src[O2 + i];
    tw = d;
    w1 = d + S;
    float2 *e = d + 2 * S;
    for (int k2 = 1; k2 < a.K; ++k2, e += THREADS + 32) {
      e[tid] = reinterpret_cast<const float2 *>(a.twB)[k2 * THREADS + tid];
      if (tid < 32) e[THREADS + tid] = reinterpret_cast<const float2 *>(a.twQ)[k2 * 32 + tid];
    }
    twist = d + 2 * S;
  }
  // Twist factor of input b = 4 (t + 128 q) + grp in pass k2 > 0 (slot 4 t + grp of
  // the tables' 512 and their factor q).
  __device__ __forceinline__ float2 turn(int k2, int q, bool full) const {
    const float2 *e = twist + (k2 - 1) * (THREADS + 32);
    return cmul(e[THREADS + 2 * q + (q >= 8 && !full)], e[4 * t + grp]);
  }
  // w^k, 0 <= k < 8192
  __device__ __forceinline__ float2 w(int k) const {
    float2 x = w1[k & (S - 1)];
    if (k & S) x = make_float2(-x.y, x.x);
    if (k & (2 * S)) x = make_float2(-x.x, -x.y);
    return x;
  }
  // signed index of output p + 2048 s
  __device__ __forceinline__ static int freq(int p, int s) { return p + S * (s < 2 ? s : s - 4); }

  // The group's inputs g[q] = x[4 (t + 128 q) + grp] -> emit(k2, p, s, X[p + 2048 s])
  // of the K twisted passes.  Ends with a CTA barrier.
  template <typename Emit>
  __device__ __forceinline__ void bwd(const float2 (&g)[16], int K, bool full, Emit emit) const {
    for (int k2 = 0; k2 < K; ++k2) {
      float2 v[16], o[16];
      if (k2 == 0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = g[q];
      } else {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = cmul(g[q], turn(k2, q, full));
      }
      col_fft_inplace<float2, S, TPF, +1>(v, A, tw, t, o, sync);
      sync();  // the last stage's reads are done
#pragma unroll
      for (int q = 0; q < 16; ++q) A[fpad(t + TPF * q)] = o[q];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = tid + THREADS * j;
        float2 x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = buf[r * BS + fpad(p)];
#pragma unroll
        for (int r = 1; r < 4; ++r) x[r] = cmul(x[r], w(r * p));
        dft_reg<4>(x, +1);
#pragma unroll
        for (int s = 0; s < 4; ++s) emit(k2, p, s, x[s]);
      }
      __syncthreads();  // the buffers are free
    }
  }

  // The transpose: load(k2, p, s) gives X[p + 2048 s] of pass k2, the sum over the
  // passes is left in acc[q] = x[4 (t + 128 q) + grp].  The buffers are free at
  // the start and, after a CTA barrier, at the end; loaded(k2) runs when
  // every thread has made its loads of pass k2.
  template <typename Load, typename Loaded>
  __device__ __forceinline__ void fwd(float2 (&acc)[16], int K, bool full, Load load,
                                      Loaded loaded) const {
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = make_float2(0.0f, 0.0f);
    for (int k2 = 0; k2 < K; ++k2) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = tid + THREADS * j;
        float2 x[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) x[s] = load(k2, p, s);
        dft_reg<4>(x, -1);
#pragma unroll
        for (int r = 1; r < 4; ++r) {
          float2 c = w(r * p);
          c.y = -c.y;
          x[r] = cmul(x[r], c);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) buf[r * BS + fpad(p)] = x[r];
      }
      __syncthreads();
      loaded(k2);
      float2 v[16], o[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = A[fpad(t + TPF * q)];
      col_fft_inplace<float2, S, TPF, -1>(v, A, tw, t, o, sync);
      if (k2 == 0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) acc[q] = o[q];
      } else {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          float2 c = turn(k2, q, full);
          c.y = -c.y;
          const float2 y = cmul(o[q], c);
          acc[q].x += y.x;
          acc[q].y += y.y;
        }
      }
      __syncthreads();  // the buffers are free
    }
  }
};

// Shared memory of the u transforms: buffers and tables, then for bwd the
// staged columns (TMA), for fwd the staged H segment and the first column's
// result.
struct QuadCol {
  using T = TmaCfg<float, Quad::M, 2>;
  static size_t bwd_bytes(int L, bool full, int K) {
    return 128 + T::stage_bytes(L, full) + size_t(Quad::BUF + Quad::tab(K)) * sizeof(float2);
  }
  static size_t fwd_bytes(int hseg, int K) {
    return 128 + (size_t(2 * Quad::BUF + Quad::tab(K)) + hseg) * sizeof(float2);
  }
};

// Band columns -> H image rows, backward (+), for pairs of adjacent columns (one
// CTA an SM, looping over (plane, pair)): the pair's rows are staged by the
// tensor memory accelerator while the pair before is transformed.
static __global__ void __launch_bounds__(Quad::THREADS, 1)
k_ucol_bwd_quad(ColArgs a, const __grid_constant__ CUtensorMap tmap, int npl, int *err) {
  using T = QuadCol::T;
  constexpr int M = Quad::M, THREADS = Quad::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t mis = smem_u32(smem_raw) & 127u;
  float2 *stage = reinterpret_cast<float2 *>(smem_raw + (mis ? 128u - mis : 0u));  // [rows][2]
  const Quad Q(stage + size_t(T::rows(a.L, a.band_full)) * 2, a);
  __shared__ __align__(8) uint64_t bar;
  const int npairs = (a.ny + 1) / 2, nitems = npairs * npl;
  const int reg2 = tma_boxes1(a, M, T::BR) * T::BR;
  int item = blockIdx.x;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (item < nitems)
      tma_issue_item<float, M, 2>(a, &tmap, stage, &bar, item / npairs, (item % npairs) * 2);
  }
  __syncthreads();  // the barrier and the tables are in place
  for (uint32_t parity = 0; item < nitems; item += gridDim.x, parity ^= 1u) {
    const int lp = item / npairs, j0 = (item % npairs) * 2;
    // the copy did not complete for some thread: all report and stop
    if (__syncthreads_or(!mbar_wait(&bar, parity))) {
      if (threadIdx.x == 0) atomicOr(err, 2);
      mbar_wait(&bar, parity);
      return;
    }
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      // the column from the staged rows to the groups, through their buffers
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int b = Q.tid + THREADS * q;
        float2 x = make_float2(0.0f, 0.0f);
        if (a.band_full || b <= a.L)
          x = stage[2 * b + c];
        else if (b >= M - a.L)
          x = stage[2 * (reg2 + b - (M - a.L)) + c];
        Q.buf[Quad::at(b)] = x;
      }
      __syncthreads();
      const int next = item + gridDim.x;
      if (c == 1 && threadIdx.x == 0 && next < nitems) {
        // order the reads above (generic proxy) before the copy engine's
        // writes to the same buffer (async proxy)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tma_issue_item<float, M, 2>(a, &tmap, stage, &bar, next / npairs, (next % npairs) * 2);
      }
      float2 g[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) g[q] = Q.A[fpad(Q.t + Quad::TPF * q)];
      const bool jv = j0 + c < a.ny;
      float2 *rowp = reinterpret_cast<float2 *>(a.H) +
                     (size_t(lp) * a.ny + (jv ? j0 + c : 0)) * (size_t(a.K) * a.hseg);
      Q.bwd(g, a.K, a.band_full, [&](int k2, int p, int s, float2 x) {
        const int m = Quad::freq(p, s), i = a.K * m + k2 + a.nx / 2;
        if (jv && unsigned(i) < unsigned(a.nx)) rowp[k2 * a.hseg + (m - a.hm0)] = x;
      });
    }
  }
}

// H image rows -> band columns, forward (-): the transpose, for pairs of adjacent
// columns, stored together (16 bytes a band row).  Each pass's segment of an
// H row is staged by a bulk copy while the pass before is transformed.
static __global__ void __launch_bounds__(Quad::THREADS, 1)
k_ucol_fwd_quad(ColArgs a, int npl, int *err) {
  constexpr int M = Quad::M, THREADS = Quad::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t mis = smem_u32(smem_raw) & 127u;
  float2 *stage = reinterpret_cast<float2 *>(smem_raw + (mis ? 128u - mis : 0u));  // [hseg]
  float2 *hold = stage + a.hseg;  // the pair's first column, as the buffers
  const Quad Q(hold + Quad::BUF, a);
  __shared__ __align__(8) uint64_t bar;
  const int npairs = (a.ny + 1) / 2, nitems = npairs * npl;
  auto issue = [&](int item, int c, int k2) {
    const int lp = item / npairs, j = (item % npairs) * 2 + c;
    const uint32_t bytes = uint32_t(a.hseg) * uint32_t(sizeof(float2));
    mbar_expect_tx(&bar, bytes);
    bulk_load(stage,
              reinterpret_cast<const float2 *>(a.H) +
                  ((size_t(lp) * a.ny + j) * a.K + k2) * size_t(a.hseg),
              bytes, &bar);
  };
  int item = blockIdx.x;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (item < nitems) issue(item, 0, 0);
  }
  __syncthreads();  // the barrier and the tables are in place
  uint32_t parity = 0, open = 0;  // (open: the phase thread 0's last copy completes)
  bool ok = true;
  for (; item < nitems; item += gridDim.x) {
    const int lp = item / npairs, j0 = (item % npairs) * 2;
    const int nc = min(2, a.ny - j0);
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
      float2 acc[16];
      int waited = -1;
      Q.fwd(
          acc, a.K, a.band_full,
          [&](int k2, int p, int s) {
            if (waited != k2) {  // once a pass, at its first load
              waited = k2;
              ok = ok && mbar_wait(&bar, parity);
              open = ok ? parity ^ 1u : open;
              parity ^= 1u;
            }
            const int m = Quad::freq(p, s), i = a.K * m + k2 + a.nx / 2;
            return unsigned(i) < unsigned(a.nx) ? stage[m - a.hm0] : make_float2(0.0f, 0.0f);
          },
          [&](int k2) {
            if (threadIdx.x != 0 || !ok) return;
            int ni = item, cn = c, kn = k2 + 1;
            if (kn == a.K) {
              kn = 0;
              if (++cn == nc) {
                cn = 0;
                ni += gridDim.x;
              }
            }
            if (ni < nitems) {
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              issue(ni, cn, kn);
            }
          });
      float2 *dst = (c == nc - 1 ? Q.buf : hold) + Q.grp * Quad::BS;
#pragma unroll
      for (int q = 0; q < 16; ++q) dst[fpad(Q.t + Quad::TPF * q)] = acc[q];
    }
    // a copy did not complete for some thread: all report and stop
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(err, 2);
      mbar_wait(&bar, open);
      return;
    }
    int jx = j0 + a.joff;
    jx -= (jx >= a.nv) ? a.nv : 0;
    float2 *col = reinterpret_cast<float2 *>(a.band) + size_t(lp) * a.nv + jx;
#pragma unroll 4
    for (int q = 0; q < 16; ++q) {
      const int b = Q.tid + THREADS * q;
      const int u = slot_u(a, b, M);
      if (u >= (1 << 29)) continue;
      float2 *dst = col + size_t(slot_bi(a, u)) * a.P * a.nv;
      const float2 y = Q.buf[Quad::at(b)];
      if (nc == 2) {
        const float2 x = hold[Quad::at(b)];
        *reinterpret_cast<float4 *>(dst) = make_float4(x.x, x.y, y.x, y.y);
      } else {
        *dst = y;
      }
    }
    __syncthreads();  // the buffers are free
  }
}

__device__ __forceinline__ void copy8(float2 *dst, const float2 *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)),
               "l"(__cvta_generic_to_global(src))
               : "memory");
}

struct QuadRow {
  static size_t bwd_bytes(int K) { return size_t(2 * Quad::BUF + Quad::tab(K)) * sizeof(float2); }
  static size_t fwd_bytes(int ncol, int K) {
    return (size_t(Quad::BUF + Quad::tab(K)) + ncol) * sizeof(float2);
  }
};

// Band rows -> transformed rows, backward (+), one row at a time (k_vrow_bwd):
// the next row is copied in, laid out as the buffers, under the transform.
static __global__ void __launch_bounds__(Quad::THREADS, 1) k_vrow_bwd_quad(RowArgs a) {
  constexpr int M = Quad::M, THREADS = Quad::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2 *stage = reinterpret_cast<float2 *>(smem_raw);
  const Quad Q(stage + Quad::BUF, a);
  auto row_at = [&](long long row) {
    const long long r = row / a.npl;
    return size_t(r) * a.P + size_t(row - r * a.npl);
  };
  auto issue = [&](long long row) {
    const float2 *in = reinterpret_cast<const float2 *>(a.band) + row_at(row) * a.nvs;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int b = Q.tid + THREADS * q, c = row_col<M>(a, b, q);
      if (c >= 0) copy8(&stage[Quad::at(b)], in + c);
    }
  };
  // (the empty slots are the same in every row)
  for (int i = threadIdx.x; i < Quad::BUF; i += THREADS) stage[i] = make_float2(0.0f, 0.0f);
  __syncthreads();
  long long row = blockIdx.x;
  if (row < a.nrow) issue(row);
  for (; row < a.nrow; row += gridDim.x) {
    copies_done();
    __syncthreads();
    float2 g[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) g[q] = stage[Q.grp * Quad::BS + fpad(Q.t + Quad::TPF * q)];
    __syncthreads();
    if (row + gridDim.x < a.nrow) issue(row + gridDim.x);
    float2 *out = reinterpret_cast<float2 *>(a.hv) + row_at(row) * a.ncol;
    Q.bwd(g, a.K, false, [&](int k2, int p, int s, float2 x) {
      const int m = Quad::freq(p, s), j = a.K * m + k2 + a.ny / 2;
      if (unsigned(j) < unsigned(a.ny)) out[k2 * a.hseg + (m - a.hm0)] = x;
    });
  }
}

// Transformed rows -> band rows, forward (-): the transpose.
static __global__ void __launch_bounds__(Quad::THREADS, 1) k_vrow_fwd_quad(RowArgs a) {
  constexpr int M = Quad::M, THREADS = Quad::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Quad Q(reinterpret_cast<float2 *>(smem_raw), a);
  float2 *stage = reinterpret_cast<float2 *>(smem_raw) + Quad::BUF + Quad::tab(a.K);  // [ncol]
  auto row_at = [&](long long row) {
    const long long r = row / a.npl;
    return size_t(r) * a.P + size_t(row - r * a.npl);
  };
  auto issue = [&](long long row) {
    const float2 *in = reinterpret_cast<const float2 *>(a.hv) + row_at(row) * a.ncol;
    for (int i = threadIdx.x; i < a.ncol; i += THREADS) copy8(stage + i, in + i);
  };
  long long row = blockIdx.x;
  if (row < a.nrow) issue(row);
  for (; row < a.nrow; row += gridDim.x) {
    copies_done();
    __syncthreads();
    float2 acc[16];
    Q.fwd(
        acc, a.K, false,
        [&](int k2, int p, int s) {
          const int m = Quad::freq(p, s), j = a.K * m + k2 + a.ny / 2;
          return unsigned(j) < unsigned(a.ny) ? stage[k2 * a.hseg + (m - a.hm0)]
                                              : make_float2(0.0f, 0.0f);
        },
        [&](int k2) {
          if (k2 == a.K - 1 && row + gridDim.x < a.nrow) issue(row + gridDim.x);
        });
#pragma unroll
    for (int q = 0; q < 16; ++q) Q.A[fpad(Q.t + Quad::TPF * q)] = acc[q];
    __syncthreads();
    float2 *out = reinterpret_cast<float2 *>(a.band) + row_at(row) * a.nvs;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int b = Q.tid + THREADS * q, c = row_col<M>(a, b, q);
      if (c >= 0) out[c] = Q.buf[Quad::at(b)];
    }
    __syncthreads();  // the buffers are free
  }
}

}  // namespace wsg
