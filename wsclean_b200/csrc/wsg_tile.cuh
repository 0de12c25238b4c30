// The shared-memory tile of a spread / interpolation CTA and its exchange
// with the band grid.  A tile holds W planes of S x S complex cells
// (S = T + W - 1 <= 32), cell (p, ia, ib) at p PS + ia RS + ib.
#pragma once

#include "wsg_internal.h"
// (the device header uses the host declarations above)
#include "wsg_device.cuh"

namespace wsg {

// Adding to a shared-memory cell that other warps may be adding to, without a
// lock or a compare-and-swap loop: take() empties the cell, put() puts the sum
// back and returns what a concurrent add left there in between (zero as a
// rule), which the caller adds in turn.  Of two adds that collide at least one
// is done, so the loop ends.  Exchanges run at the rate of plain loads and
// stores (2.1 cycles a warp for 64 bits on the B200), FP32 and FP64
// shared-memory additions at 6 to 11 cycles a warp.
__device__ __forceinline__ unsigned long long exch64(void *p, unsigned long long v) {
  return atomicExch(reinterpret_cast<unsigned long long *>(p), v);
}
__device__ __forceinline__ double take(double *p) {
  return __longlong_as_double((long long)exch64(p, 0ull));
}
__device__ __forceinline__ double put(double *p, double v) {
  return __longlong_as_double((long long)exch64(p, (unsigned long long)__double_as_longlong(v)));
}

// The cells of a chunk's tile that its records touch, as lines along v: over
// the bounding box of the footprints, or footprint by footprint when few
// origins were used.  A warp takes up to 32 consecutive lines at a time: each
// lane finds one line's grid row, then the warp walks the lines with lanes
// along v (several short lines side by side), so that finding a row costs one
// lane's work instead of a warp's (the flush and the staging of a W = 8 tile
// of 27 x 27 cells took 70 warp instructions a line when every lane did it).
struct TileLines {
  int nline, len, lpi, sub, col, gsz;
  bool by_list, act;
  int lu0, lv0, nbu;
  const uint32_t *orig;
};

template <int W>
__device__ __forceinline__ TileLines tile_lines(const int *bb, int norig, const uint32_t *orig,
                                                int lane, int nwarp) {
  TileLines t;
  t.lu0 = bb[0];
  t.lv0 = bb[2];
  t.nbu = max(bb[1] + W - t.lu0, 0);
  const int nbv = max(bb[3] + W - t.lv0, 0);
  t.by_list = norig <= kMaxOrig && norig * W * W < t.nbu * nbv;
  t.nline = t.by_list ? norig * W * W : W * t.nbu;
  t.len = t.by_list ? W : max(nbv, 1);
  t.lpi = 32 / t.len;
  t.sub = lane / t.len;
  t.col = lane - t.sub * t.len;
  t.act = t.sub < t.lpi;
  t.gsz = min(32, (t.nline + nwarp - 1) / nwarp);
  t.orig = orig;
  return t;
}

// One lane's line: the grid row (null outside the pass or the band), and in
// where the first stored column (upper half; grids are below 65535) and the
// line's tile offset.
template <int W, typename C>
__device__ __forceinline__ C *tile_line(const TileLines &t, const JobRegs &jr, int line, int mp,
                                        int ucorner, int vcorner, int RS, int PS, uint32_t &where) {
  int p, ia, ib;
  if (t.by_list) {
    const int o = line / (W * W), pr = line - o * W * W;
    p = pr / W;
    const uint32_t luv = t.orig[o];
    ia = int(luv >> 16) + (pr - p * W);
    ib = int(luv & 0xffffu);
  } else {
    p = line / t.nbu;
    ia = t.lu0 + (line - p * t.nbu);
    ib = t.lv0;
  }
  where = (uint32_t(jr.first_col(vcorner + ib)) << 16) | uint32_t(p * PS + ia * RS + ib);
  const int plane = mp + p;
  const int bi = jr.band_row(jr.wrap_u(ucorner + ia));
  if (plane < jr.pb0 || plane >= jr.pb1 || bi < 0) return nullptr;
  return reinterpret_cast<C *>(jr.grid) + (size_t(bi) * jr.P + (plane - jr.pb0)) * size_t(jr.nvs);
}

__device__ __forceinline__ void *shfl_ptr(void *p, int src) {
  return reinterpret_cast<void *>(
      __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), src));
}

__device__ __forceinline__ float2 take_cell(float2 *p) {
  const unsigned long long v = exch64(p, 0ull);
  return make_float2(__uint_as_float(uint32_t(v)), __uint_as_float(uint32_t(v >> 32)));
}
// (put's counterpart for a cell, and whether anything came back)
__device__ __forceinline__ float2 put_cell(float2 *p, float2 x) {
  const unsigned long long v =
      exch64(p, (unsigned long long)__float_as_uint(x.x) |
                    ((unsigned long long)__float_as_uint(x.y) << 32));
  return make_float2(__uint_as_float(uint32_t(v)), __uint_as_float(uint32_t(v >> 32)));
}
__device__ __forceinline__ bool cell_set(float2 x) {
  return (__float_as_uint(x.x) | __float_as_uint(x.y)) != 0u;
}
__device__ __forceinline__ double2 take_cell(double2 *p) {
  return make_double2(take(&p->x), take(&p->y));
}
__device__ __forceinline__ void red_cell(float2 *p, float2 v) { atomicAdd(p, v); }
__device__ __forceinline__ void red_cell(double2 *p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// Adds the touched cells of the tile to the band grid and leaves them zero
// (a cell shared by two listed footprints is taken once).
template <int W, typename C>
__device__ __forceinline__ void tile_flush(C *tile, int RS, int PS, const TileLines &t,
                                           const JobGeom &jb, int mp, int ucorner, int vcorner,
                                           int warp, int lane, int nwarp) {
  const JobRegs jr(jb);
  for (int l0 = warp * t.gsz; l0 < t.nline; l0 += nwarp * t.gsz) {
    uint32_t where = 0;
    C *row = nullptr;
    if (lane < t.gsz && l0 + lane < t.nline)
      row = tile_line<W, C>(t, jr, l0 + lane, mp, ucorner, vcorner, RS, PS, where);
    const int n = min(t.gsz, t.nline - l0);
    // iterations whose exchanges are in flight together (the FP64 kernels have
    // no registers to spare)
    constexpr int U = sizeof(C) == 8 ? 4 : 1;
    for (int i0 = 0; i0 < n; i0 += U * t.lpi) {
      C x[U], *dst[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int i = i0 + q * t.lpi, src = min(i + t.sub, 31);
        C *const rp = reinterpret_cast<C *>(shfl_ptr(row, src));
        const uint32_t wh = __shfl_sync(0xffffffffu, where, src);
        dst[q] = nullptr;
        if (t.act && i + t.sub < n) {
          x[q] = take_cell(&tile[(wh & 0xffffu) + t.col]);
          const int v = jr.next_col(int(wh >> 16), t.col);
          if (rp && v >= 0) dst[q] = rp + v;
        }
      }
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (dst[q] && (x[q].x != 0 || x[q].y != 0)) red_cell(dst[q], x[q]);
    }
  }
}

// One cell from global to shared memory without a register in between (zero
// when src is null; size 8 or 16 bytes).
template <typename C>
__device__ __forceinline__ void copy_cell(C *dst, const C *src, const void *any) {
  const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
  const void *p = src ? static_cast<const void *>(src) : any;
  const int n = src ? int(sizeof(C)) : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(__cvta_generic_to_global(p)),
               "n"(sizeof(C)), "r"(n)
               : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Copies the touched cells from the band grid into the tile, asynchronously
// (copies_done and a barrier end it): all of a warp's cells are in flight
// together.
template <int W, typename C>
__device__ __forceinline__ void tile_stage(C *tile, int RS, int PS, const TileLines &t,
                                           const JobGeom &jb, int mp, int ucorner, int vcorner,
                                           int warp, int lane, int nwarp) {
  const JobRegs jr(jb);
  for (int l0 = warp * t.gsz; l0 < t.nline; l0 += nwarp * t.gsz) {
    uint32_t where = 0;
    C *row = nullptr;
    if (lane < t.gsz && l0 + lane < t.nline)
      row = tile_line<W, C>(t, jr, l0 + lane, mp, ucorner, vcorner, RS, PS, where);
    const int n = min(t.gsz, t.nline - l0);
    for (int i = 0; i < n; i += t.lpi) {
      const int src = min(i + t.sub, 31);
      const C *const rp = reinterpret_cast<const C *>(shfl_ptr(row, src));
      const uint32_t wh = __shfl_sync(0xffffffffu, where, src);
      if (t.act && i + t.sub < n) {
        const int v = jr.next_col(int(wh >> 16), t.col);
        copy_cell(&tile[(wh & 0xffffu) + t.col], rp && v >= 0 ? rp + v : nullptr, jr.grid);
      }
    }
  }
}

// The chunk a CTA works on (filled by thread 0).
struct ChunkState {
  int chunk, norig;  // chunk < 0: none left
  int s0, s1;        // its records
  int bb[4];
  uint32_t orig[kMaxOrig];
  JobGeom job;
};

// Thread 0's fetch of the chunk after the CTA's next one (a CTA keeps three:
// the one in hand, the next, whose records are loaded early, and the one being
// fetched), in three parts spread over the work in hand so that none of the
// dependent loads is waited for.
struct ChunkFetch {
  int c, s0, s1;
  __device__ __forceinline__ void begin(const GridArgs &a) { c = atomicAdd(a.counter, 1); }
  __device__ __forceinline__ void starts(const GridArgs &a) {
    const int n = *a.nchunks;
    if (c >= n) {
      c = -1;
      return;
    }
    s0 = a.chunk_start[c];
    s1 = c + 1 < n ? a.chunk_start[c + 1] : a.nvis;
  }
  __device__ __forceinline__ void store(ChunkState &cs, const GridArgs &a, const DevGeom &g) const {
    cs.chunk = c;
    cs.s0 = s0;
    cs.s1 = s1;
    cs.bb[0] = cs.bb[2] = 1 << 30;
    cs.bb[1] = cs.bb[3] = -1;
    cs.norig = 0;
    if (c >= 0) cs.job = load_job(a, g, c);
  }
};
__device__ __forceinline__ void fetch_chunk(ChunkState &cs, const GridArgs &a, const DevGeom &g) {
  ChunkFetch f;
  f.begin(a);
  f.starts(a);
  f.store(cs, a, g);
}
__device__ __forceinline__ void first_chunks(ChunkState *css, const GridArgs &a, const DevGeom &g) {
  fetch_chunk(css[0], a, g);
  fetch_chunk(css[1], a, g);
}
// A chunk's bin: its first record's tile and plane, and whether it has planes
// in this pass.
struct ChunkBin {
  int tu, tv, mp;
  bool pass;
};
template <int W, typename Rec>
__device__ __forceinline__ ChunkBin chunk_bin(const ChunkState &cs, const Rec *recs, int T) {
  const uint32_t iuv = recs[cs.s0].iuv;
  ChunkBin b;
  b.mp = int(recs[cs.s0].mp);
  b.tu = int(iuv >> 16) / T;
  b.tv = int(iuv & 0xffffu) / T;
  b.pass = (b.mp < cs.job.pb1) && (b.mp + W > cs.job.pb0);
  return b;
}

// Lists a staged batch's new footprint origins (one warp): my is the lane's
// packed origin, prev the last one of the batch before.  A repeated origin in
// the list is harmless, its cells being taken once.
__device__ __forceinline__ void list_origins(ChunkState &cs, uint32_t my, bool valid, uint32_t prev,
                                             int lane) {
  uint32_t before = __shfl_up_sync(0xffffffffu, my, 1);
  if (lane == 0) before = prev;
  const unsigned nm = __ballot_sync(0xffffffffu, valid && my != before && my != kSkip);
  if (!nm) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(&cs.norig, __popc(nm));
  base = __shfl_sync(0xffffffffu, base, 0);
  const int k = base + __popc(nm & ((1u << lane) - 1u));
  if (((nm >> lane) & 1u) && k < kMaxOrig) cs.orig[k] = my;
}

// Bounding box of the lanes' origins into the chunk's (one warp).
__device__ __forceinline__ void merge_box(ChunkState &cs, int b0, int b1, int b2, int b3, int lane) {
  b0 = __reduce_min_sync(0xffffffffu, b0);
  b1 = __reduce_max_sync(0xffffffffu, b1);
  b2 = __reduce_min_sync(0xffffffffu, b2);
  b3 = __reduce_max_sync(0xffffffffu, b3);
  if (lane == 0 && b1 >= 0) {
    atomicMin(&cs.bb[0], b0);
    atomicMax(&cs.bb[1], b1);
    atomicMin(&cs.bb[2], b2);
    atomicMax(&cs.bb[3], b3);
  }
}

// Bounding box and distinct origins of a chunk's records [s0, s1), by all
// warps (before an interpolation stages its tile).
template <typename Rec>
__device__ __forceinline__ void scan_origins(ChunkState &cs, const Rec *recs, int s0, int s1, int tu,
                                             int tv, int T, int tid, int nthr) {
  const int lane = tid & 31;
  int b0 = 1 << 30, b1 = -1, b2 = 1 << 30, b3 = -1;
  for (int s = s0 + tid - lane; s < s1; s += nthr) {
    uint32_t luv = kSkip;
    if (s + lane < s1) {
      const uint32_t iuv = recs[s + lane].iuv;
      const int lu = int(iuv >> 16) - tu * T, lv = int(iuv & 0xffffu) - tv * T;
      if (lu >= 0 && lu < T && lv >= 0 && lv < T) {
        luv = (uint32_t(lu) << 16) | uint32_t(lv);
        b0 = min(b0, lu); b1 = max(b1, lu);
        b2 = min(b2, lv); b3 = max(b3, lv);
      }
    }
    list_origins(cs, luv, true, kSkip, lane);
  }
  merge_box(cs, b0, b1, b2, b3, lane);
}

}  // namespace wsg
