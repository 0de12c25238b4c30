// Spreading and interpolation in FP32 (the mixed form).
//
// A CTA of 8 warps owns a chunk: records of one (tile, first plane) bin,
// sorted by footprint origin, each warp a contiguous slice of them.  A warp
// stages 32 records at a time (lane l evaluates record l's 3W kernel values)
// and then works record by record: lane q owns the (plane, u-row) pairs
// q + 32 k of the footprint and their W cells along v, which stay in registers
// while the origin repeats.
//
// What bounds it: latency at 16 warps an SM (fixed-latency waits first), with issue
// slots 59-64% and the shared-memory pipe 44-51% busy; DRAM is at 5-6%.  So
//  * cells are kept as pairs along v, real and imaginary parts apart: the
//    kernel values along v are pairs as loaded, and one two-lane multiply-add
//    serves two cells with no register moves (pairs of (re, im) needed every
//    kernel value twice);
//  * mirrored kernel pieces share one even/odd polynomial (half the work);
//  * where the origin changes is one ballot a batch, not a test a record, and
//    a run's first record sets the cells instead of adding to cleared ones;
//  * cells are added to the tile by two exchanges (wsg_tile.cuh); shared FP32
//    additions are compare-and-swap loops, ~10 instructions a value;
//  * tile lines are found one a lane (wsg_tile.cuh), and the loads that open a
//    chunk are issued during the one before.
// Two CTAs an SM, 128 registers a thread: 3 x 8 and 2 x 12 warps an SM (80
// registers) spill and were 5-10% slower; two tiles an SM also leave room for
// 24 x 24 cells (20 x 20: 6% slower).  8.1M visibilities at 4096^2, W = 8:
// spread 1.595 -> 1.046 ms, interpolation 1.310 -> 1.236 ms; 3.3M at 2048^2,
// W = 7: 0.720 -> 0.562, 0.611 -> 0.606 ms.
#pragma once

#include "wsg_tile.cuh"

namespace wsg {

constexpr int kWarps32 = kGrid32Warps;

template <int W>
struct Cfg32 {
  static constexpr int PPL = W * W > 32 ? 2 : 1;  // (plane, u-row) pairs a lane
  static constexpr bool SAME_U = 32 % W == 0;     // a lane's pairs are of one u-row
  static constexpr int VP = (W + 1) / 2;          // cell pairs along v
  static constexpr int W4 = (W + 3) & ~3;
  // a staged record: [v: W4, zero past W][w: W4][u: W4][V: 2], stride 4 mod 8
  // floats (16-byte stores of 8 lanes fall on different banks)
  static constexpr int SW = W4, SU = 2 * W4, SV = 3 * W4;
  static constexpr int ST = grid32_stride(W);
  // (the interpolation's rows also hold 16 complex sums)
  static constexpr int IST = 36;
  static_assert(W <= 8 && ST >= SV + 2 && ST % 8 == 4, "staged record layout");
};

// All 3W values of a record into its staged row (axis a at a W4; v first).
template <int W>
__device__ __forceinline__ void eval32(const DevKernel<float> &kc, float x, float (&out)[(W + 3) & ~3]) {
  constexpr int DEG = KDeg<W>::value, H = (W + 1) / 2;
  constexpr int DE = DEG & ~1, DO = (DEG - 1) | 1;
  const float y = x * x;
#pragma unroll
  for (int i = W; i < ((W + 3) & ~3); ++i) out[i] = 0.0f;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    float e = kc.c[DE][k], o = kc.c[DO][k];
#pragma unroll
    for (int j = DE - 2; j >= 0; j -= 2) e = fmaf(e, y, kc.c[j][k]);
#pragma unroll
    for (int j = DO - 2; j >= 1; j -= 2) o = fmaf(o, y, kc.c[j][k]);
    out[k] = fmaf(o, x, e);
    if (2 * k + 1 != W) out[W - 1 - k] = fmaf(-o, x, e);
  }
}

template <int N>
__device__ __forceinline__ void store_row(float *p, const float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 4)
    *reinterpret_cast<float4 *>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

template <int W>
__device__ __forceinline__ void stage32(const DevKernel<float> &kc, const RecF &r, int do_w,
                                        float *row) {
  using K = Cfg32<W>;
  float v[K::W4];
  eval32<W>(kc, r.xv, v);
  store_row(row, v);
  eval32<W>(kc, r.xu, v);
  store_row(row + K::SU, v);
  if (do_w) {
    eval32<W>(kc, r.xw, v);
  } else {
#pragma unroll
    for (int i = 0; i < K::W4; ++i) v[i] = i == 0 ? 1.0f : 0.0f;
  }
  store_row(row + K::SW, v);
}

// The cell pairs' kernel values along v of a staged row.
template <int W>
__device__ __forceinline__ void load_v(const float *row, float2 (&kv)[Cfg32<W>::VP]) {
#pragma unroll
  for (int i = 0; i < Cfg32<W>::VP; i += 2) {
    const float4 x = *reinterpret_cast<const float4 *>(row + 2 * i);
    kv[i] = make_float2(x.x, x.y);
    if (i + 1 < Cfg32<W>::VP) kv[i + 1] = make_float2(x.z, x.w);
  }
}

__device__ __forceinline__ uint32_t origin32(const RecF &rr, int tu, int tv, int mp, int T, int *err) {
  const int lu = int(rr.iuv >> 16) - tu * T, lv = int(rr.iuv & 0xffffu) - tv * T;
  if (lu < 0 || lu >= T || lv < 0 || lv >= T || int(rr.mp) != mp) {
    atomicOr(err, 1);
    return kSkip;
  }
  return (uint32_t(lu) << 16) | uint32_t(lv);
}

// The visibility a record spreads: its own, or (plan execution) the gathered
// one times the record's static factor.
__device__ __forceinline__ float2 spread_value(const RecF &rr, const GridArgs &a) {
  if (!a.vis_in) return make_float2(rr.vr, rr.vi);
  const uint32_t id = rr.idx & 0x7fffffffu;
  float xr, xi;
  if (a.vis_in_double) {
    const double2 x = reinterpret_cast<const double2 *>(a.vis_in)[id];
    xr = float(x.x);
    xi = float(x.y);
  } else {
    const float2 x = reinterpret_cast<const float2 *>(a.vis_in)[id];
    xr = x.x;
    xi = x.y;
  }
  const float vr = xr * rr.vr + xi * rr.vi, vi = xi * rr.vr - xr * rr.vi;
  return make_float2(vr, (rr.idx & 0x80000000u) ? -vi : vi);
}

__device__ __forceinline__ RecF load32(const RecF *recs, int s, bool valid) {
  RecF r{};
  if (valid) r = recs[s];
  return r;
}

// Tile strides in cells: odd row stride, plane stride 8 mod 16, so that a
// footprint's 8 rows x 2 planes (a half warp's 8-byte cells) fall on different
// banks.
__device__ __forceinline__ int plane32(int S, int RS) {
  const int n = S * RS;
  return n + (((8 - n % 16) + 16) % 16);
}

// ------------------------------------------------------------- k_spread32
template <int W>
__global__ void __launch_bounds__(kWarps32 * 32, 2)
k_spread32(GridArgs a, DevGeom g, DevKernel<float> kc) {
  using K = Cfg32<W>;
  constexpr int NWARP = kWarps32, PPL = K::PPL, VP = K::VP, ST = K::ST;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ChunkState css[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = g.T + W - 1, RS = S | 1, PS = plane32(S, RS);
  float2 *tile = reinterpret_cast<float2 *>(smem_raw);
  float *st = reinterpret_cast<float *>(tile + W * PS) + warp * 32 * ST;
  const RecF *recs = reinterpret_cast<const RecF *>(a.rec);

  for (int i = tid; i < W * PS; i += NWARP * 32) tile[i] = make_float2(0.0f, 0.0f);
  // the lane's staged-row indices and tile offsets
  int kwi[PPL], kui[PPL], coff[PPL];
  auto ok = [&](int k) { return 32 * (k + 1) <= W * W || lane + 32 * k < W * W; };
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    const int q = lane + 32 * k, p = q / W, c = q - p * W;
    kwi[k] = K::SW + (ok(k) ? p : 0);
    kui[k] = K::SU + (ok(k) ? c : 0);
    coff[k] = p * PS + c * RS;
  }
  int b = 0;
  if (tid == 0) first_chunks(css, a, g);
  __syncthreads();
  // the warp's slice [j0, j1) of chunk c, and its lane's first record
  int j0 = 0, j1 = 0;
  ChunkBin bin{};
  RecF rr{};
  auto open = [&](const ChunkState &c) {
    if (c.chunk < 0) return;
    j0 = c.s0 + (c.s1 - c.s0) * warp / NWARP;
    j1 = c.s0 + (c.s1 - c.s0) * (warp + 1) / NWARP;
    rr = load32(recs, j0 + lane, j0 + lane < j1);
    bin = chunk_bin<W>(c, recs, g.T);
  };
  open(css[0]);
  for (;; b = b == 2 ? 0 : b + 1) {
    __syncthreads();  // the tile is clean
    ChunkState &cs = css[b];
    if (cs.chunk < 0) break;
    ChunkFetch fetch;
    if (tid == 0) fetch.begin(a);
    const int tu = bin.tu, tv = bin.tv, mp = bin.mp;
    const bool pass = bin.pass;
    if (pass && j0 < j1) {
      float2 re[PPL][VP], im[PPL][VP];
#pragma unroll
      for (int k = 0; k < PPL; ++k)
#pragma unroll
        for (int c = 0; c < VP; ++c) re[k][c] = im[k][c] = make_float2(0.0f, 0.0f);
      uint32_t cur = kNone;
      int b0 = 1 << 30, b1 = -1, b2 = 1 << 30, b3 = -1;

      auto commit = [&]() {
        if (cur < kSkip) {
          float2 *const o = tile + (int(cur >> 16) * RS + int(cur & 0xffffu));
#pragma unroll
          for (int k = 0; k < PPL; ++k) {
            if (ok(k)) {
              float2 *const t = o + coff[k];
              float2 x[W], got[W];
              bool left = false;
#pragma unroll
              for (int c = 0; c < W; ++c) {
                const float2 pr = re[k][c / 2], pi = im[k][c / 2];
                x[c] = c % 2 ? make_float2(pr.y, pi.y) : make_float2(pr.x, pi.x);
              }
#pragma unroll
              for (int c = 0; c < W; ++c) got[c] = take_cell(t + c);
#pragma unroll
              for (int c = 0; c < W; ++c) {
                x[c] = put_cell(t + c, make_float2(got[c].x + x[c].x, got[c].y + x[c].y));
                left |= cell_set(x[c]);
              }
              while (left) {  // what concurrent adds left is added in turn
                left = false;
#pragma unroll
                for (int c = 0; c < W; ++c)
                  if (cell_set(x[c])) {
                    const float2 y = take_cell(t + c);
                    x[c] = put_cell(t + c, make_float2(y.x + x[c].x, y.y + x[c].y));
                    left |= cell_set(x[c]);
                  }
              }
            }
          }
        }
      };

      for (int s = j0; s < j1; s += 32) {
        const int nb = min(32, j1 - s);
        uint32_t my = kSkip;
        if (lane < nb) {
          float *row = st + lane * ST;
          my = origin32(rr, tu, tv, mp, g.T, a.err);
          if (my != kSkip) {
            b0 = min(b0, int(my >> 16)); b1 = max(b1, int(my >> 16));
            b2 = min(b2, int(my & 0xffffu)); b3 = max(b3, int(my & 0xffffu));
          }
          *reinterpret_cast<float2 *>(row + K::SV) = spread_value(rr, a);
          stage32<W>(kc, rr, g.do_w, row);
        }
        rr = load32(recs, s + 32 + lane, s + 32 + lane < j1);
        __syncwarp();
        uint32_t prev = __shfl_up_sync(0xffffffffu, my, 1);
        if (lane == 0) prev = cur;
        const unsigned chg = __ballot_sync(0xffffffffu, lane < nb && my != prev);
        list_origins(cs, my, lane < nb, cur, lane);
        for (int j = 0; j < nb;) {
          const bool first = (chg >> j) & 1u;
          if (first) {
            commit();
            cur = __shfl_sync(0xffffffffu, my, j);
          }
          const unsigned rest = j < 31 ? chg >> (j + 1) : 0u;
          const int je = rest ? min(nb, j + __ffs(rest)) : nb;
          auto add = [&](int jj, bool fresh) {
            const float *row = st + jj * ST;
            float2 kv[VP];
            load_v<W>(row, kv);
            float2 V = *reinterpret_cast<const float2 *>(row + K::SV);
            if constexpr (K::SAME_U) V = __fmul2_rn(V, make_float2(row[kui[0]], row[kui[0]]));
#pragma unroll
            for (int k = 0; k < PPL; ++k) {
              float f = row[kwi[k]];
              if constexpr (!K::SAME_U) f *= row[kui[k]];
              const float ar = V.x * f, ai = V.y * f;
              const float2 ar2 = make_float2(ar, ar), ai2 = make_float2(ai, ai);
#pragma unroll
              for (int c = 0; c < VP; ++c) {
                re[k][c] = fresh ? __fmul2_rn(ar2, kv[c]) : __ffma2_rn(ar2, kv[c], re[k][c]);
                im[k][c] = fresh ? __fmul2_rn(ai2, kv[c]) : __ffma2_rn(ai2, kv[c], im[k][c]);
              }
            }
          };
          // (a run's first record sets the cells: no clearing)
          if (first) add(j++, true);
#pragma unroll 2
          for (; j < je; ++j) add(j, false);
        }
        __syncwarp();
      }
      commit();
      merge_box(cs, b0, b1, b2, b3, lane);
    }
    __syncthreads();
    if (tid == 0) fetch.starts(a);
    open(css[b == 2 ? 0 : b + 1]);
    if (pass) {
      const TileLines tln = tile_lines<W>(cs.bb, cs.norig, cs.orig, lane, NWARP);
      tile_flush<W, float2>(tile, RS, PS, tln, cs.job, mp, tu * g.T - g.nsafe, tv * g.T - g.nsafe,
                            warp, lane, NWARP);
    }
    if (tid == 0) fetch.store(css[b == 0 ? 2 : b - 1], a, g);
  }
}

// ------------------------------------------------------------- k_interp32
//
// The transpose: the chunk's tile region is copied from the band grid, and
// each lane dots its cells with a record's kernel values.  The lanes' parts
// are added in pairs by one shuffle and left in the record's staged row, which
// is read by then; after the batch each lane adds up its own record's sixteen
// (about 5 instructions a record, against 10 for shuffle reductions of four
// records at a time).
template <int W>
__global__ void __launch_bounds__(kWarps32 * 32, 2)
k_interp32(GridArgs a, DevGeom g, DevKernel<float> kc) {
  using K = Cfg32<W>;
  constexpr int NWARP = kWarps32, PPL = K::PPL, VP = K::VP, ST = K::IST;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ChunkState css[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = g.T + W - 1, RS = S | 1, PS = plane32(S, RS);
  float2 *tile = reinterpret_cast<float2 *>(smem_raw);
  float *st = reinterpret_cast<float *>(tile + W * PS) + warp * 32 * ST;
  const RecF *recs = reinterpret_cast<const RecF *>(a.rec);
  const bool direct = a.last_pass && a.first_pass;

  int kwi[PPL], kui[PPL], coff[PPL];
  auto ok = [&](int k) { return 32 * (k + 1) <= W * W || lane + 32 * k < W * W; };
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    const int q = lane + 32 * k, p = q / W, c = q - p * W;
    kwi[k] = K::SW + (ok(k) ? p : 0);
    kui[k] = K::SU + (ok(k) ? c : 0);
    coff[k] = p * PS + c * RS;
  }
  int b = 0;
  if (tid == 0) first_chunks(css, a, g);
  __syncthreads();
  // a chunk's bin, and its origins if it has planes in this pass
  auto open = [&](ChunkState &c) {
    ChunkBin n{};
    if (c.chunk >= 0) {
      n = chunk_bin<W>(c, recs, g.T);
      if (n.pass) scan_origins(c, recs, c.s0, c.s1, n.tu, n.tv, g.T, tid, NWARP * 32);
    }
    return n;
  };
  ChunkBin bin = open(css[0]);
  for (;; b = b == 2 ? 0 : b + 1) {
    __syncthreads();  // the chunk's origins are known, the tile is free
    ChunkState &cs = css[b];
    if (cs.chunk < 0) break;
    ChunkFetch fetch;
    if (tid == 0) fetch.begin(a);
    const int tu = bin.tu, tv = bin.tv, mp = bin.mp;
    const bool pass = bin.pass;  // (else nothing in this pass)
    const int j0 = cs.s0 + (cs.s1 - cs.s0) * warp / NWARP;
    const int j1 = cs.s0 + (cs.s1 - cs.s0) * (warp + 1) / NWARP;
    if (pass) {
      const TileLines tln = tile_lines<W>(cs.bb, cs.norig, cs.orig, lane, NWARP);
      tile_stage<W, float2>(tile, RS, PS, tln, cs.job, mp, tu * g.T - g.nsafe, tv * g.T - g.nsafe,
                            warp, lane, NWARP);
    }
    // under the copies: the lane's first record, the next chunk's origins
    RecF rr = load32(recs, j0 + lane, j0 + lane < j1);
    bin = open(css[b == 2 ? 0 : b + 1]);
    if (tid == 0) fetch.starts(a);
    copies_done();
    __syncthreads();
    if (tid == 0) fetch.store(css[b == 0 ? 2 : b - 1], a, g);
    if (!pass) continue;

    float2 re[PPL][VP], im[PPL][VP];  // the lane's cells at the current origin
#pragma unroll
    for (int k = 0; k < PPL; ++k)
#pragma unroll
      for (int c = 0; c < VP; ++c) re[k][c] = im[k][c] = make_float2(0.0f, 0.0f);
    uint32_t cur = kNone;
    for (int s = j0; s < j1; s += 32) {
      const int nb = min(32, j1 - s);
      uint32_t my = kSkip;
      if (lane < nb) {
        my = origin32(rr, tu, tv, mp, g.T, a.err);
        stage32<W>(kc, rr, g.do_w, st + lane * ST);
      }
      const float2 fac = make_float2(rr.vr, rr.vi);
      const uint32_t idx = rr.idx;
      rr = load32(recs, s + 32 + lane, s + 32 + lane < j1);
      __syncwarp();
      uint32_t prev = __shfl_up_sync(0xffffffffu, my, 1);
      if (lane == 0) prev = cur;
      const unsigned chg = __ballot_sync(0xffffffffu, lane < nb && my != prev);
      for (int j = 0; j < nb;) {
        if ((chg >> j) & 1u) {
          cur = __shfl_sync(0xffffffffu, my, j);
          if (cur != kSkip) {
            const float2 *const o = tile + (int(cur >> 16) * RS + int(cur & 0xffffu));
#pragma unroll
            for (int k = 0; k < PPL; ++k) {
              const float2 *const t = o + (ok(k) ? coff[k] : 0);
#pragma unroll
              for (int c = 0; c < VP; ++c) {
                const float2 x = t[2 * c];
                const float2 y = 2 * c + 1 < W ? t[2 * c + 1] : make_float2(0.0f, 0.0f);
                re[k][c] = make_float2(x.x, y.x);
                im[k][c] = make_float2(x.y, y.y);
              }
            }
          }
        }
        const unsigned rest = j < 31 ? chg >> (j + 1) : 0u;
        const int je = rest ? min(nb, j + __ffs(rest)) : nb;
#pragma unroll 2
        for (; j < je; ++j) {
          float *const row = st + j * ST;
          float2 kv[VP];
          load_v<W>(row, kv);
          float2 sr, si;
#pragma unroll
          for (int k = 0; k < PPL; ++k) {
            float f = row[kwi[k]];
            if constexpr (!K::SAME_U) f *= row[kui[k]];
            if (!ok(k)) f = 0.0f;
            float2 tr = __fmul2_rn(re[k][0], kv[0]), ti = __fmul2_rn(im[k][0], kv[0]);
#pragma unroll
            for (int c = 1; c < VP; ++c) {
              tr = __ffma2_rn(re[k][c], kv[c], tr);
              ti = __ffma2_rn(im[k][c], kv[c], ti);
            }
            const float2 f2 = make_float2(f, f);
            sr = k == 0 ? __fmul2_rn(tr, f2) : __ffma2_rn(tr, f2, sr);
            si = k == 0 ? __fmul2_rn(ti, f2) : __ffma2_rn(ti, f2, si);
          }
          float2 x = make_float2(sr.x + sr.y, si.x + si.y);
          if constexpr (K::SAME_U) {
            const float ku = row[kui[0]];
            x = make_float2(x.x * ku, x.y * ku);
          }
          const float2 y = make_float2(__shfl_xor_sync(0xffffffffu, x.x, 16),
                                       __shfl_xor_sync(0xffffffffu, x.y, 16));
          // (the record's row has been read by every lane: it holds its sums)
          x = cadd(x, y);
          if (lane < 16) reinterpret_cast<float2 *>(row)[lane] = x;
        }
      }
      __syncwarp();
      // every lane adds up and finishes its own record
      if (lane < nb && my != kSkip) {
        const float4 *const row = reinterpret_cast<const float4 *>(st + lane * ST);
        float2 own = make_float2(0.0f, 0.0f), odd = own;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 x = row[i];
          own = cadd(own, make_float2(x.x, x.y));
          odd = cadd(odd, make_float2(x.z, x.w));
        }
        own = cadd(own, odd);
        if (direct) {
          const float si = (idx & 0x80000000u) ? -own.y : own.y;
          const double orr = double(fac.x) * double(own.x) - double(fac.y) * double(si);
          const double oi = double(fac.x) * double(si) + double(fac.y) * double(own.x);
          store_vis(a.vis_out, a.vis_double, a.vis_accumulate, idx & 0x7fffffffu, orr, oi);
        } else {  // the record's one writer in this pass
          float2 *p = reinterpret_cast<float2 *>(a.acc) + s + lane;
          p->x += own.x;
          p->y += own.y;
        }
      }
      __syncwarp();
    }
  }
}

}  // namespace wsg
