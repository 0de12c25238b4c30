// Spreading and interpolation in FP64 on the FP64 matrix units.
//
// Records of a chunk are sorted by footprint origin, and all records of one
// origin spread into the same W x W x W cells, so a run of them is a matrix
// product.  With rows (p, c) -- plane p, c = real or imaginary part -- and
// columns (u, v):
//     spread   C[(p,c), (u,v)] += sum_r (V_c w_p)[r] (u_u v_v)[r]
//     interp   D[(p,c), r]      = sum_(u,v) cell[(p,c), (u,v)] (u_u v_v)[r],
//              out_c[r]         = sum_p w_p[r] D[(p,c), r]
// (w, u, v: the record's kernel values).  Both are chains of
// mma.m8n8k4.f64, which is the widest FP64 instruction there is (tcgen05 has
// no FP64 form) and runs at the rate of the FP64 pipe: 256 multiply-adds in
// one instruction, 18.5 T/s measured against 18.2 for scalar FMAs, reached
// with one warp a scheduler.  The former kernels needed 8 independent scalar
// FMA chains, their shared-memory operands and a shuffle reduction for the
// same work and were bound by latency at one CTA an SM.
// 2.9M visibilities, W = 14 (1024^2, eps 1e-12): spread 4.59 -> 2.35 ms,
// interpolation 5.19 -> 2.37 ms (1.07 ms of it the products).
//
// A CTA's 16 warps work as two teams of 8 on the two halves of a chunk, on one
// tile.  A team's warps share every record: the spread splits the output tiles
// over them, the interpolation the (u, v) sum.  They stage 32 records at a time
// together, double buffered (one team barrier a batch), each warp evaluating a
// fixed share of a record's 3 W kernel values; the records of the batch after
// are loaded meanwhile.  The teams drift apart, so that one's staging and
// commits run under the other's products (one team of 16 warps took 2.5 ms
// where two take 2.4, W = 14).  Up to W = 8 the interpolation instead
// gives a warp whole records of its own slice of the chunk (the 2 x 16 cell
// tiles of W = 8 fit its registers), as summing 8 warps' parts would cost more
// than the products.
#pragma once

#include "wsg_tile.cuh"

namespace wsg {

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

template <int W>
struct Cfg64 {
  static constexpr int MT = (2 * W + 7) / 8;    // row tiles of (p, c)
  static constexpr int N = W * W;
  static constexpr int WARPS = 16, TEAM = 8;    // warps a CTA, a team
  // spread: a team's warps as MG row groups of MTW row tiles by NG column
  // groups (two row groups where there are few column tiles)
  static constexpr int NTALL = (N + 7) / 8;
  static constexpr int MG = (W <= 8 && MT % 2 == 0) ? 2 : 1;
  static constexpr int MTW = MT / MG;
  static constexpr int NG = TEAM / MG;
  static constexpr int NT = (NTALL + NG - 1) / NG;
  // interpolation: (u, v) steps of 4, split over the KG warps of a record
  static constexpr bool SOLO = W <= kSolo64;
  static constexpr int IWARPS = SOLO ? 8 : WARPS;
  static constexpr int KG = SOLO ? 1 : TEAM;
  static constexpr int KTALL = (N + 3) / 4;
  static constexpr int KT = (KTALL + KG - 1) / KG;
  // a staged record: spread [V_c w_p: 8 MT][u: W][v: W], interpolation
  // [w: W][u: W][v: W]; row strides of 4 mod 16 doubles keep the fragment
  // loads (4 records x 4 consecutive values a half warp) free of conflicts
  static constexpr int SU = 8 * MT, SV = SU + W, SST = grid64_spread_stride(W);
  static constexpr int IU = W, IV = 2 * W, IST = grid64_interp_stride(W);
};

// Barrier of one team (0 or 1): named barriers 1 and 2.
__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, 256;" ::"r"(team + 1) : "memory");
}

// Tile strides in complex cells: rows of S cells; the plane stride is 1
// (spread) or 4 (interpolation) mod 8, which keeps a half warp's four rows
// (p, c) on different banks from one another.
__device__ __forceinline__ int plane64(int S, int r) {
  const int n = S * S;
  return n + ((r - n % 8) + 8) % 8;
}

// The 3W kernel values of a record come in mirrored pairs: the kernel is even,
// so pieces k and W-1-k are E(x^2) +- x O(x^2) of one polynomial (make_kernel
// makes the coefficients exactly so), half the multiply-adds and coefficients
// of two separate ones.  Pairs [q0, q0 + NU) (axes u, v, w in turn), up to
// four side by side; q0 is a constant once inlined (constant-bank
// coefficients).  put_value(axis, piece, value) stores one value.
template <int W>
struct Pairs64 {
  static constexpr int H = (W + 1) / 2, ALL = 3 * H;
};
template <int W, int NU, typename Put>
__device__ __forceinline__ void eval64(const DevKernel<double> &kc, const RecD &r, const int q0,
                                       int do_w, Put &&put_value) {
  constexpr int DEG = KDeg<W>::value, H = Pairs64<W>::H;
  constexpr int DE = DEG & ~1, DO = (DEG - 1) | 1;  // highest even and odd powers
  constexpr int G = NU < 4 ? NU : 4;
#pragma unroll
  for (int i0 = 0; i0 < NU; i0 += G) {
    double x[G], y[G], e[G], o[G];
    int axis[G], k[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int q = min(q0 + i0 + i, 3 * H - 1);
      axis[i] = q / H;
      k[i] = q - axis[i] * H;
      x[i] = axis[i] == 0 ? r.xu : (axis[i] == 1 ? r.xv : r.xw);
      y[i] = x[i] * x[i];
      e[i] = kc.c[DE][k[i]];
      o[i] = kc.c[DO][k[i]];
    }
#pragma unroll
    for (int j = DE - 2; j >= 0; j -= 2)
#pragma unroll
      for (int i = 0; i < G; ++i) e[i] = fma(e[i], y[i], kc.c[j][k[i]]);
#pragma unroll
    for (int j = DO - 2; j >= 1; j -= 2)
#pragma unroll
      for (int i = 0; i < G; ++i) o[i] = fma(o[i], y[i], kc.c[j][k[i]]);
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if (i0 + i < NU && q0 + i0 + i < 3 * H) {
        double lo = fma(o[i], x[i], e[i]), hi = fma(-o[i], x[i], e[i]);
        if (axis[i] == 2 && !do_w) {
          lo = k[i] == 0 ? 1.0 : 0.0;
          hi = 0.0;
        }
        put_value(axis[i], k[i], lo);
        if (2 * k[i] + 1 != W) put_value(axis[i], W - 1 - k[i], hi);
      }
    }
  }
}

// A warp's share of the pairs when NW warps split them, by a branch on the
// warp's number (uniform) to code with that share's coefficients.
template <int W, int NW, int I = 0, typename Put>
__device__ __forceinline__ void eval64_share(const DevKernel<double> &kc, const RecD &r, int warp,
                                             int do_w, Put &&put_value) {
  constexpr int NU = (Pairs64<W>::ALL + NW - 1) / NW;
  if constexpr (I * NU < Pairs64<W>::ALL) {
    if (warp == I)
      eval64<W, NU>(kc, r, I * NU, do_w, put_value);
    else
      eval64_share<W, NW, I + 1>(kc, r, warp, do_w, put_value);
  }
}

// Loads the parts of record s that a warp's share of the values needs (axes
// [a0, a1], the visibility with the w axis) and, when meta, the rest.  A
// record is 64 bytes, so each 8 to 16 byte load of 32 records touches 16
// cache lines; zeros when not valid.
template <int W, int NW>
__device__ __forceinline__ RecD load64(const RecD *recs, int s, bool valid, int warp, bool meta) {
  constexpr int NU = (Pairs64<W>::ALL + NW - 1) / NW, H = Pairs64<W>::H;
  const int a0 = warp * NU / H, a1 = min(2, (warp * NU + NU - 1) / H);
  RecD r{};
  if (valid) {
    const RecD *p = recs + s;
    if (a0 == 0) r.xu = p->xu;
    if (a0 <= 1 && a1 >= 1) r.xv = p->xv;
    if (a0 <= 2 && a1 == 2) {
      r.xw = p->xw;
      r.idx = p->idx;
      r.vr = p->vr;
      r.vi = p->vi;
    }
    if (meta) {
      r.iuv = p->iuv;
      r.mp = p->mp;
    }
  }
  return r;
}

// The visibility a record spreads: its own, or (plan execution) the gathered
// one times the record's static factor.
__device__ __forceinline__ double2 spread_value(const RecD &rr, const GridArgs &a) {
  if (!a.vis_in) return make_double2(rr.vr, rr.vi);
  const uint32_t id = rr.idx & 0x7fffffffu;
  double xr, xi;
  if (a.vis_in_double) {
    const double2 x = reinterpret_cast<const double2 *>(a.vis_in)[id];
    xr = x.x;
    xi = x.y;
  } else {
    const float2 x = reinterpret_cast<const float2 *>(a.vis_in)[id];
    xr = x.x;
    xi = x.y;
  }
  const double vr = xr * rr.vr + xi * rr.vi, vi = xi * rr.vr - xr * rr.vi;
  return make_double2(vr, (rr.idx & 0x80000000u) ? -vi : vi);
}

// The packed in-tile origin of a record, or kSkip outside its chunk's tile.
__device__ __forceinline__ uint32_t origin64(const RecD &rr, int tu, int tv, int mp, int T, int *err) {
  const int lu = int(rr.iuv >> 16) - tu * T, lv = int(rr.iuv & 0xffffu) - tv * T;
  if (lu < 0 || lu >= T || lv < 0 || lv >= T || int(rr.mp) != mp) {
    atomicOr(err, 1);
    return kSkip;
  }
  return (uint32_t(lu) << 16) | uint32_t(lv);
}

// ------------------------------------------------------------- k_spread64
template <int W>
__global__ void __launch_bounds__(Cfg64<W>::WARPS * 32, 1)
k_spread64(GridArgs a, DevGeom g, DevKernel<double> kc) {
  using K = Cfg64<W>;
  constexpr int NWARP = K::WARPS, TW = K::TEAM, MT = K::MTW, NT = K::NT, NG = K::NG;
  constexpr int SST = K::SST, SU = K::SU, SV = K::SV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ChunkState cs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int team = warp / TW, tw = warp % TW;  // the warp's team and number in it
  const int S = g.T + W - 1, RS = S, PS = plane64(S, 1);
  double2 *tile = reinterpret_cast<double2 *>(smem_raw);
  double *spare = reinterpret_cast<double *>(tile + size_t(W) * PS);  // one a thread
  double *stg = spare + NWARP * 32 + team * 2 * 32 * SST;             // [2][32][SST] a team
  uint32_t *luvs =
      reinterpret_cast<uint32_t *>(spare + NWARP * 32 + 4 * 32 * SST) + team * 64;  // [2][32]
  const RecD *recs = reinterpret_cast<const RecD *>(a.rec);
  // The warp's place in the team's work.  Place 0 has one column tile more
  // (W = 14: 25 tiles for 8 warps) and no kernel values to evaluate, only the
  // records' origins; the teams' places are rotated so that the two warps with
  // the extra tile are on different schedulers (W = 8, 1.2M visibilities in 5
  // calls: 248 -> 239 us; W = 14: spread the same, interpolation 2.42 -> 2.37 ms).
  const int place = K::MG == 1 ? (tw + team) % TW : tw;
  const int colg = place % NG, rowg = place / NG, share = (place + TW - 1) % TW;

  for (int i = tid; i < W * PS; i += NWARP * 32) tile[i] = make_double2(0.0, 0.0);
  spare[tid] = 0.0;

  // the lane's cells: rows (p, c) of its row tiles, columns of column tiles
  // colg, colg + NG, ...  (an output past the last row or column is added to
  // the thread's spare cell instead: no branches in the commit)
  const int rrow = lane >> 2, kq = lane & 3;
  int bu[NT], bv[NT], noff[NT][2], moff[MT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int t8 = 8 * (colg + NG * j);
    const int nb = min(t8 + rrow, K::N - 1);
    bu[j] = SU + nb / W;
    bv[j] = SV + nb % W;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = t8 + 2 * kq + h;
      noff[j][h] = n < K::N ? 2 * ((n / W) * RS + n % W) : -1;
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int row = 8 * (rowg * MT + i) + rrow;
    moff[i] = row < 2 * W ? 2 * (row >> 1) * PS + (row & 1) : -1;
  }

  // (a chunk of FP64 records takes many times as long as fetching the next one:
  // nothing is kept in registers for that meanwhile)
  for (;;) {
    __syncthreads();  // the tile is clean
    if (tid == 0) fetch_chunk(cs, a, g);
    __syncthreads();
    if (cs.chunk < 0) break;
    const int s0 = cs.s0, s1 = cs.s1;
    const ChunkBin bin = chunk_bin<W>(cs, recs, g.T);
    const int tu = bin.tu, tv = bin.tv, mp = bin.mp;
    if (!bin.pass) continue;

    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    uint32_t cur = kSkip, last = kSkip;
    int b0 = 1 << 30, b1 = -1, b2 = 1 << 30, b3 = -1;

    // adds the accumulated cells of origin cur to the tile
    auto commit = [&]() {
      if (cur != kSkip) {
        double *const t0 = reinterpret_cast<double *>(tile);
        const int o = 2 * (int(cur >> 16) * RS + int(cur & 0xffffu));
        const int sp = int(spare - t0) + tid;
        // a column tile at a time: its exchanges are in flight together
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          if (colg + NG * j < K::NTALL) {
            // (tiles with rows or columns past the last: known when compiled)
            constexpr bool kRows = 8 * K::MT == 2 * W;
            int at[MT][2];
            double got[MT][2];
            bool left = false;
#define EACH                                     \
  _Pragma("unroll") for (int i = 0; i < MT; ++i) \
  _Pragma("unroll") for (int h = 0; h < 2; ++h)
            EACH {
              const bool in = (kRows || (K::MG == 1 && 8 * (i + 1) <= 2 * W) || moff[i] >= 0) &&
                              (8 * NG * (j + 1) <= K::N || noff[j][h] >= 0);
              at[i][h] = in ? o + moff[i] + noff[j][h] : sp;
            }
            EACH got[i][h] = take(t0 + at[i][h]);
            EACH {
              double &x = acc[i][j][h];
              x = put(t0 + at[i][h], got[i][h] + x);
              if (at[i][h] == sp) x = 0.0;
            }
            EACH left |= acc[i][j][h] != 0.0;
            while (left) {  // what concurrent adds left is added in turn
              left = false;
              EACH {
                double &x = acc[i][j][h];
                if (x != 0.0) {
                  double *c = t0 + at[i][h];
                  x = put(c, take(c) + x);
                  left |= x != 0.0;
                }
              }
            }
#undef EACH
          }
        }
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    };

    // stages the warp's share of n records (rr: the lane's) into st
    auto stage = [&](const RecD &rr, int n, double *st, uint32_t *lv) {
      if (lane < n) {
        double *row = st + lane * SST;
        const double2 V = spread_value(rr, a);
        eval64_share<W, TW>(kc, rr, share, g.do_w, [&](int axis, int piece, double val) {
          if (axis == 0) {
            row[SU + piece] = val;
          } else if (axis == 1) {
            row[SV + piece] = val;
          } else {
            row[2 * piece] = val * V.x;
            row[2 * piece + 1] = val * V.y;
          }
        });
      }
      if (share == TW - 1) {  // (the warp with the smallest share of values)
        uint32_t luv = kSkip;
        if (lane < n) {
          luv = origin64(rr, tu, tv, mp, g.T, a.err);
          lv[lane] = luv;
          if (luv != kSkip) {
            b0 = min(b0, int(luv >> 16)); b1 = max(b1, int(luv >> 16));
            b2 = min(b2, int(luv & 0xffffu)); b3 = max(b3, int(luv & 0xffffu));
          }
        }
        list_origins(cs, luv, lane < n, last, lane);
        last = __shfl_sync(0xffffffffu, luv, n - 1);
      }
    };

    // adds n staged records, one run of equal origins after another
    auto consume = [&](int n, const double *st, const uint32_t *lv) {
      const uint32_t my = lane < n ? lv[lane] : kSkip;
      uint32_t prev = __shfl_up_sync(0xffffffffu, my, 1);
      if (lane == 0) prev = cur;
      const unsigned chg = __ballot_sync(0xffffffffu, lane < n && my != prev);
      for (int j = 0; j < n;) {
        if ((chg >> j) & 1u) {
          commit();
          cur = __shfl_sync(0xffffffffu, my, j);
        }
        const unsigned rest = j < 31 ? chg >> (j + 1) : 0u;
        const int j1 = rest ? min(n, j + __ffs(rest)) : n;
        auto step = [&](const double *row, bool in) {
          double av[MT];
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            av[i] = row[8 * (rowg * MT + i) + rrow];
            if (!in) av[i] = 0.0;
          }
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            if (colg + NG * t < K::NTALL) {
              const double bvv = row[bu[t]] * row[bv[t]];
#pragma unroll
              for (int i = 0; i < MT; ++i) dmma(acc[i][t][0], acc[i][t][1], av[i], bvv);
            }
          }
        };
        const double *row = st + (j + kq) * SST;
        for (; j + 4 <= j1; j += 4, row += 4 * SST) step(row, true);
        if (j < j1) step(st + min(j + kq, j1 - 1) * SST, j + kq < j1);
        j = j1;
      }
    };

    const int j0 = s0 + (s1 - s0) * team / 2, j1 = s0 + (s1 - s0) * (team + 1) / 2;
    auto load = [&](int s) { return load64<W, TW>(recs, s, s < j1, share, share == TW - 1); };
    if (j0 < j1) {
      RecD rr = load(j0 + lane);
      stage(rr, min(32, j1 - j0), stg, luvs);
      rr = load(j0 + 32 + lane);
      int b = 0;
      for (int s = j0; s < j1; s += 32, b ^= 1) {
        team_sync(team);  // this batch is staged, the other buffer is free
        if (s + 32 < j1) {
          stage(rr, min(32, j1 - s - 32), stg + (b ^ 1) * 32 * SST, luvs + (b ^ 1) * 32);
          rr = load(s + 64 + lane);
        }
        consume(min(32, j1 - s), stg + b * 32 * SST, luvs + b * 32);
      }
      commit();
      if (share == TW - 1) merge_box(cs, b0, b1, b2, b3, lane);
    }
    __syncthreads();
    const TileLines tln = tile_lines<W>(cs.bb, cs.norig, cs.orig, lane, NWARP);
    tile_flush<W, double2>(tile, RS, PS, tln, cs.job, mp, tu * g.T - g.nsafe, tv * g.T - g.nsafe,
                           warp, lane, NWARP);
  }
}

// ------------------------------------------------------------- k_interp64

// Writes one record's sum: finalised in a single plane pass, else added to
// the per-record accumulator (one writer a record and pass).
__device__ __forceinline__ void finish64(const GridArgs &a, const RecD *recs, int s, double sr,
                                         double si, bool direct) {
  if (direct) {
    const RecD rr = recs[s];
    if (rr.idx & 0x80000000u) si = -si;
    store_vis(a.vis_out, a.vis_double, a.vis_accumulate, rr.idx & 0x7fffffffu,
              rr.vr * sr - rr.vi * si, rr.vr * si + rr.vi * sr);
  } else {
    double2 *p = reinterpret_cast<double2 *>(a.acc) + s;
    p->x += sr;
    p->y += si;
  }
}

template <int W>
__global__ void __launch_bounds__(Cfg64<W>::IWARPS * 32, 1)
k_interp64(GridArgs a, DevGeom g, DevKernel<double> kc) {
  using K = Cfg64<W>;
  constexpr int NWARP = K::IWARPS, MT = K::MT, KT = K::KT, NG = K::KG, TW = K::TEAM;
  constexpr int IST = K::IST, IU = K::IU, IV = K::IV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ChunkState cs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = g.T + W - 1, RS = S, PS = plane64(S, 4);
  double2 *tile = reinterpret_cast<double2 *>(smem_raw);
  const int team = warp / TW, tw = warp % TW;  // the warp's team and number in it
  // staging areas of 32 records (one a warp, or two a team), the warps' sums
  // of a batch [record][c] (one a warp, or two), the records' origins (one set
  // a warp, or three a team)
  constexpr int NST = K::SOLO ? NWARP : 4, NSUM = K::SOLO ? NWARP : 2 * NWARP;
  double *stg = reinterpret_cast<double *>(tile + size_t(W) * PS);
  double *osum = stg + NST * 32 * IST;
  uint32_t *luvs = reinterpret_cast<uint32_t *>(osum + NSUM * 64);
  const RecD *recs = reinterpret_cast<const RecD *>(a.rec);
  const bool direct = a.last_pass && a.first_pass;
  // (places as in the spread: place 0 has one step more and no evaluation)
  const int place = (tw + team) % TW;
  const int grp = K::SOLO ? 0 : place;
  const int share = K::SOLO ? 0 : (place + TW - 1) % TW;

  // the lane's cells: rows (p, c) of row tile i, (u, v) of step t
  const int rrow = lane >> 2, kq = lane & 3;
  int ku[KT], kv[KT], noff[KT];
#pragma unroll
  for (int t = 0; t < KT; ++t) {
    const int n = 4 * (grp + NG * t) + kq;
    const int nn = n < K::N ? n : 0;  // (the cell is taken as zero)
    ku[t] = IU + nn / W;
    kv[t] = IV + nn % W;
    noff[t] = n < K::N ? 2 * ((nn / W) * RS + nn % W) : -1;
  }

  for (;;) {
    __syncthreads();
    if (tid == 0) fetch_chunk(cs, a, g);
    __syncthreads();
    if (cs.chunk < 0) break;
    const int s0 = cs.s0, s1 = cs.s1;
    const ChunkBin bin = chunk_bin<W>(cs, recs, g.T);
    const int tu = bin.tu, tv = bin.tv, mp = bin.mp;
    if (!bin.pass) continue;  // nothing in this pass
    scan_origins(cs, recs, s0, s1, tu, tv, g.T, tid, NWARP * 32);
    __syncthreads();
    {
      const TileLines tln = tile_lines<W>(cs.bb, cs.norig, cs.orig, lane, NWARP);
      tile_stage<W, double2>(tile, RS, PS, tln, cs.job, mp, tu * g.T - g.nsafe, tv * g.T - g.nsafe,
                             warp, lane, NWARP);
    }
    copies_done();
    __syncthreads();

    double cell[MT][KT];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int t = 0; t < KT; ++t) cell[i][t] = 0.0;
    uint32_t cur = kSkip;

    auto stage = [&](const RecD &rr, int n, double *st, uint32_t *lv) {
      if (lane < n) {
        double *row = st + lane * IST;
        if (K::SOLO || share == TW - 1) lv[lane] = origin64(rr, tu, tv, mp, g.T, a.err);
        eval64_share<W, NG>(kc, rr, share, g.do_w, [&](int axis, int piece, double val) {
          row[axis == 0 ? IU + piece : (axis == 1 ? IV + piece : piece)] = val;
        });
      }
    };

    // sums of n staged records into os[record][c], eight of a run at a time
    auto consume = [&](int n, const double *st, const uint32_t *lv, double *os) {
      const uint32_t my = lane < n ? lv[lane] : kSkip;
      uint32_t prev = __shfl_up_sync(0xffffffffu, my, 1);
      if (lane == 0) prev = cur;
      const unsigned chg = __ballot_sync(0xffffffffu, lane < n && my != prev);
      for (int j = 0; j < n;) {
        if ((chg >> j) & 1u) {
          cur = __shfl_sync(0xffffffffu, my, j);
          if (cur != kSkip) {
            const double *o = reinterpret_cast<const double *>(tile) +
                              2 * (int(cur >> 16) * RS + int(cur & 0xffffu));
#pragma unroll
            for (int i = 0; i < MT; ++i) {
              const int row = 8 * i + rrow;
              const double *om = o + 2 * (row >> 1) * PS + (row & 1);
#pragma unroll
              for (int t = 0; t < KT; ++t)
                cell[i][t] = (row < 2 * W && noff[t] >= 0) ? om[noff[t]] : 0.0;
            }
          }
        }
        const unsigned rest = j < 31 ? chg >> (j + 1) : 0u;
        const int j1 = rest ? min(n, j + __ffs(rest)) : n;
        for (; j < j1; j += 8) {
          const double *row = st + min(j + rrow, j1 - 1) * IST;
          double d[MT][2];
#pragma unroll
          for (int i = 0; i < MT; ++i) d[i][0] = d[i][1] = 0.0;
#pragma unroll
          for (int t = 0; t < KT; ++t) {
            if (NG == 1 || grp + NG * t < K::KTALL) {
              const double b = row[ku[t]] * row[kv[t]];
#pragma unroll
              for (int i = 0; i < MT; ++i) dmma(d[i][0], d[i][1], cell[i][t], b);
            }
          }
          // sum over p: rows of one parity, in this lane and in lanes 8, 16 apart
          double sum[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const double *wr = st + min(j + 2 * kq + h, j1 - 1) * IST;
            double x = 0.0;
#pragma unroll
            for (int i = 0; i < MT; ++i) {
              const int p = 4 * i + (rrow >> 1);
              x = fma(d[i][h], wr[min(p, W - 1)], x);  // (rows past the last are zero)
            }
            x += __shfl_xor_sync(0xffffffffu, x, 8);
            x += __shfl_xor_sync(0xffffffffu, x, 16);
            sum[h] = x;
          }
          if (lane < 8) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (j + 2 * kq + h < j1) os[2 * (j + 2 * kq + h) + rrow] = sum[h];
          }
        }
        j = j1;
      }
    };

    const int n = s1 - s0;
    if constexpr (K::SOLO) {
      const int j0 = s0 + (n * warp) / NWARP, j1 = s0 + (n * (warp + 1)) / NWARP;
      double *st = stg + size_t(warp) * 32 * IST;
      double *os = osum + warp * 64;
      uint32_t *lv = luvs + warp * 32;
      auto load = [&](int s) { return load64<W, 1>(recs, s, s < j1, 0, true); };
      RecD rr = load(j0 + lane);
      for (int s = j0; s < j1; s += 32) {
        const int nb = min(32, j1 - s);
        stage(rr, nb, st, lv);
        rr = load(s + 32 + lane);
        __syncwarp();
        consume(nb, st, lv, os);
        __syncwarp();
        if (lane < nb && lv[lane] != kSkip)
          finish64(a, recs, s + lane, os[2 * lane], os[2 * lane + 1], direct);
        __syncwarp();
      }
    } else {
      const int j0 = s0 + n * team / 2, j1 = s0 + n * (team + 1) / 2;
      if (j0 >= j1) continue;
      stg += team * 2 * 32 * IST;
      osum += team * 2 * TW * 64;  // [buffer][warp][record][c]
      luvs += team * 96;
      // batch b's sums are added up and written after the barrier that ends
      // it, by the team's first two warps
      auto finish = [&](int s, int nb, int b, int l) {
        if (tw < 2) {
          const int r = (tw * 32 + lane) >> 1, c = lane & 1;
          double x = 0.0;
          if (r < nb) {
            const double *os = osum + b * TW * 64 + 2 * r + c;
#pragma unroll
            for (int w = 0; w < TW; ++w) x += os[w * 64];
          }
          const double y = __shfl_xor_sync(0xffffffffu, x, 1);
          if (c == 0 && r < nb && luvs[l * 32 + r] != kSkip)
            finish64(a, recs, s + r, x, y, direct);
        }
      };
      // (three sets of origins: those of the batch before are read by the
      // first two warps while the last warp stages the batch after)
      auto load = [&](int s) { return load64<W, TW>(recs, s, s < j1, share, share == TW - 1); };
      RecD rr = load(j0 + lane);
      stage(rr, min(32, j1 - j0), stg, luvs);
      rr = load(j0 + 32 + lane);
      int b = 0, l = 0;
      for (int s = j0; s < j1; s += 32, b ^= 1) {
        team_sync(team);  // this batch is staged; the one before is summed
        const int ln = l == 2 ? 0 : l + 1, lp = l == 0 ? 2 : l - 1;
        if (s > j0) finish(s - 32, 32, b ^ 1, lp);
        if (s + 32 < j1) {
          stage(rr, min(32, j1 - s - 32), stg + (b ^ 1) * 32 * IST, luvs + ln * 32);
          rr = load(s + 64 + lane);
        }
        consume(min(32, j1 - s), stg + b * 32 * IST, luvs + l * 32, osum + (b * TW + tw) * 64);
        l = ln;
      }
      team_sync(team);
      const int nb = (j1 - j0 - 1) % 32 + 1;
      finish(j1 - nb, nb, b ^ 1, l == 0 ? 2 : l - 1);
      stg -= team * 2 * 32 * IST;
      osum -= team * 2 * TW * 64;
      luvs -= team * 96;
    }
  }
}

}  // namespace wsg
