// Launchers of the spread / interpolation kernels (dispatched over the
// support W), the pruned u transforms (over log2 M, with their staged
// forms) and the w-screens: the one translation unit that compiles them.

#include "wsg_grid32.cuh"
#include "wsg_grid64.cuh"
#include "wsg_host.cuh"
#include "wsg_quad.cuh"

namespace wsg {

namespace {

// Resident CTAs an SM, cached: the query is a driver call, and plans enqueue
// launches while a stream is being captured into a graph.
int resident_ctas(const void *fn, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, size_t, int>, int> memo;
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  const auto key = std::make_tuple(fn, smem, dev);
  std::lock_guard<std::mutex> lk(mu);
  auto it = memo.find(key);
  if (it != memo.end()) return it->second;
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem);
  return memo[key] = std::max(nb, 1);
}

// Spread / interpolation kernels, dispatched over the support W: one
// persistent launch of as many CTAs as are resident.
template <typename R>
struct GridKernels {
  template <int W>
  static void run(bool spread, int nsm, cudaStream_t st, const GridArgs &a, const DevGeom &g,
                  const DevKernel<R> &kc) {
    using Fn = void (*)(GridArgs, DevGeom, DevKernel<R>);
    Fn fn;
    int threads;
    if constexpr (sizeof(R) == 8) {
      fn = spread ? k_spread64<W> : k_interp64<W>;
      threads = 32 * (spread ? Cfg64<W>::WARPS : Cfg64<W>::IWARPS);
    } else {
      fn = spread ? k_spread32<W> : k_interp32<W>;
      threads = 32 * kWarps32;
    }
    const size_t smem = tile_smem_bytes(g.T, W, sizeof(R) == 4);
    require(smem <= kMaxSmemPerBlock, "internal: spread tile exceeds shared memory");
    smem_attr(fn, smem);
    fn<<<nsm * resident_ctas(reinterpret_cast<const void *>(fn), threads, smem), threads, smem, st>>>(
        a, g, kc);
    cuda_check(cudaGetLastError(), spread ? "spread launch" : "interpolation launch");
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  }
  static void dispatch(int W, bool spread, int nsm, cudaStream_t st, const GridArgs &a,
                       const DevGeom &g, const DevKernel<R> &kc) {
    auto go = [&](auto wc) {
      constexpr int WW = decltype(wc)::value;
      if constexpr (sizeof(R) == 4 && WW > 8)
        throw std::runtime_error("support too large for mixed precision");
      else
        run<WW>(spread, nsm, st, a, g, kc);
    };
    switch (W) {
      case 4: go(std::integral_constant<int, 4>{}); break;
      case 5: go(std::integral_constant<int, 5>{}); break;
      case 6: go(std::integral_constant<int, 6>{}); break;
      case 7: go(std::integral_constant<int, 7>{}); break;
      case 8: go(std::integral_constant<int, 8>{}); break;
      case 9: go(std::integral_constant<int, 9>{}); break;
      case 10: go(std::integral_constant<int, 10>{}); break;
      case 11: go(std::integral_constant<int, 11>{}); break;
      case 12: go(std::integral_constant<int, 12>{}); break;
      case 13: go(std::integral_constant<int, 13>{}); break;
      case 14: go(std::integral_constant<int, 14>{}); break;
      case 15: go(std::integral_constant<int, 15>{}); break;
      case 16: go(std::integral_constant<int, 16>{}); break;
      default: throw std::runtime_error("unsupported kernel support");
    }
  }
};

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library has no link-time driver dependency); nullptr if unavailable.
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
    cudaGetLastError();
  });
  return fn;
}

// Whether `extra` bytes of shared memory fit beside a CTA's `base` bytes
// without lowering the CTAs an SM holds (228 KB a SM, 227 KB a CTA, 1 KB
// reserved a CTA).
bool twist_tables_fit(size_t base, size_t extra) {
  constexpr size_t kSM = 228 * 1024, kCTA = 227 * 1024, kRes = 1024;
  if (base + extra > kCTA) return false;
  return kSM / (base + extra + kRes) == kSM / (base + kRes);
}

// Pruned u-transform kernels, dispatched over log2(M).
template <typename R>
struct ColKernels {
  // The band-to-image transform with the band columns staged by the tensor
  // memory accelerator (k_ucol_bwd_tma), when its boxes can be used: a box
  // row of NB columns is a multiple of 16 bytes, column groups start on a
  // 16-byte boundary and do not straddle the wrap of the v axis.  Returns
  // false when not used.
  static bool column_map(const ColArgs &a, int npl, int NB, int rows, CUtensorMap &map) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc || env_int("WSG_UCOL_TMA", 1) == 0) return false;
    if (NB * 2 * int(sizeof(R)) % 16 != 0) return false;
    // (columns that start inside the row wrap after nv - joff of them)
    if (a.joff != 0 && (a.nv - a.joff) % NB != 0) return false;
    if (sizeof(R) == 4 && (a.joff % 2 != 0 || a.nv % 2 != 0)) return false;
    const cuuint64_t dims[2] = {cuuint64_t(2) * cuuint64_t(npl) * cuuint64_t(a.nv),
                                cuuint64_t(a.band_rows)};
    const cuuint64_t strides[1] = {cuuint64_t(a.P) * cuuint64_t(a.nv) * 2 * sizeof(R)};
    const cuuint32_t box[2] = {cuuint32_t(2 * NB), cuuint32_t(rows)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(&map,
               sizeof(R) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
               2, const_cast<void *>(a.band), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  template <int LOGM>
  static bool run_tma(const ColArgs &a, int npl, cudaStream_t st, int *err) {
    constexpr int M = 1 << LOGM;
    using Cfg = TmaCfg<R, M>;
    constexpr int NB = Cfg::NB;
    CUtensorMap map;
    if (!err || !column_map(a, npl, NB, Cfg::BR, map)) return false;
    const size_t base = Cfg::stage_bytes(a.L, a.band_full) +
                        (size_t(NB) * FftBuf<M>::value + M) * 2 * sizeof(R) + 128;
    // the twist factors go to shared memory too when that costs no resident CTA
    const size_t extra = size_t(a.K - 1) * M * 2 * sizeof(R);
    const bool tws = twist_tables_fit(base, extra);
    const size_t smem = tws ? base + extra : base;
    auto *kern = tws ? k_ucol_bwd_tma<R, LOGM, true> : k_ucol_bwd_tma<R, LOGM, false>;
    smem_attr(kern, smem);
    // (the shared memory depends on the band's height and on K)
    const int per_sm =
        resident_ctas(reinterpret_cast<const void *>(kern), ColCfg<R, M>::THREADS, smem);
    int dev = 0, nsm = 148;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    cuda_check(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "attribute");
    const long long nitems = (long long)((a.ny + NB - 1) / NB) * npl;
    const int grid = int(std::min<long long>(nitems, (long long)nsm * per_sm));
    kern<<<grid, ColCfg<R, M>::THREADS, smem, st>>>(a, map, npl, err);
    cuda_check(cudaGetLastError(), "k_ucol_bwd_tma launch");
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return true;
  }
  // The mixed 8192-point transforms as four of 2048 points (k_ucol_bwd_quad,
  // k_ucol_fwd_quad), under the conditions of the staged forms and where the
  // shared memory suffices: bands up to some 8000 rows, image rows up to some
  // 3500 K.  Returns false when not used.
  static bool run_quad(bool bwd, const ColArgs &a, int npl, cudaStream_t st, int *err) {
    if constexpr (sizeof(R) != 4) {
      return false;
    } else {
      if (!err || env_int("WSG_UCOL_TMA", 1) == 0) return false;
      int dev = 0, nsm = 148;
      cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
      cuda_check(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "attribute");
      const int grid = int(std::min<long long>((long long)((a.ny + 1) / 2) * npl, nsm));
      const size_t smem = bwd ? QuadCol::bwd_bytes(a.L, a.band_full, a.K)
                              : QuadCol::fwd_bytes(a.hseg, a.K);
      // (16 bytes go to the barrier)
      if (smem + 16 > kMaxSmemPerBlock) return false;
      if (bwd) {
        CUtensorMap map;
        if (!column_map(a, npl, 2, QuadCol::T::BR, map)) return false;
        smem_attr(k_ucol_bwd_quad, smem);
        k_ucol_bwd_quad<<<grid, Quad::THREADS, smem, st>>>(a, map, npl, err);
      } else {
        // bulk copies and the 16-byte stores of a pair
        if (a.hseg % 2 != 0 || a.nv % 2 != 0 || a.joff % 2 != 0 ||
            ((reinterpret_cast<uintptr_t>(a.H) | reinterpret_cast<uintptr_t>(a.band)) & 15) != 0)
          return false;
        smem_attr(k_ucol_fwd_quad, smem);
        k_ucol_fwd_quad<<<grid, Quad::THREADS, smem, st>>>(a, npl, err);
      }
      cuda_check(cudaGetLastError(), bwd ? "k_ucol_bwd_quad launch" : "k_ucol_fwd_quad launch");
      g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
      return true;
    }
  }
  // The image-to-band transform with each pass's H-row segments staged by
  // bulk copies (k_ucol_fwd_bulk), when its shared memory fits a CTA.
  // Returns false when not used.
  template <int LOGM>
  static bool run_bulk(const ColArgs &a, int npl, cudaStream_t st, int *err) {
    constexpr int M = 1 << LOGM;
    using Cfg = ColCfg<R, M>;
    constexpr int NB = Cfg::NB;
    if (!err || env_int("WSG_UCOL_TMA", 1) == 0) return false;
    // a CTA of one column (M = 8192 in FP32, 4096 in FP64) waits on each of
    // its copies with nothing else to do: the plain kernel is faster there
    // (config 5's forward transform: 30 ms plain, 65 ms staged)
    if (NB < 2) return false;
    const size_t cs = 2 * sizeof(R);
    if ((size_t(a.hseg) * cs) % 16 != 0 || (reinterpret_cast<uintptr_t>(a.H) & 15) != 0)
      return false;
    const size_t base = 128 + (size_t(NB) * a.hseg + size_t(NB) * FftBuf<M>::value + M) * cs;
    if (base > 227 * 1024) return false;
    // the twist factors go to shared memory too when that costs no resident
    // CTA (registers or shared memory, whichever binds)
    const size_t extra = size_t(a.K - 1) * M * cs;  // (the twist factors multiplied out)
    auto *k0 = k_ucol_fwd_bulk<R, LOGM, false>;
    auto *k1 = k_ucol_fwd_bulk<R, LOGM, true>;
    // resident CTAs of each instantiation at these sizes, memoised (the
    // query is a driver call, and plans enqueue while a stream is captured)
    static std::mutex mu;
    static std::map<std::tuple<size_t, size_t, int>, std::pair<int, int>> memo;
    int dev0 = 0;
    cuda_check(cudaGetDevice(&dev0), "cudaGetDevice");
    const auto key = std::make_tuple(base, extra, dev0);
    int n0 = 0, n1 = 0;
    smem_attr(k0, base);
    if (base + extra <= 227 * 1024) smem_attr(k1, base + extra);
    {
      std::lock_guard<std::mutex> lk(mu);
      auto it = memo.find(key);
      if (it != memo.end()) {
        n0 = it->second.first;
        n1 = it->second.second;
      } else {
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n0, k0, Cfg::THREADS, base),
                   "occupancy");
        if (base + extra <= 227 * 1024)
          cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n1, k1, Cfg::THREADS,
                                                                   base + extra),
                     "occupancy");
        memo[key] = std::make_pair(n0, n1);
      }
    }
    if (n0 < 1) return false;
    const bool tws = n1 >= n0;
    const size_t smem = tws ? base + extra : base;
    auto *kern = tws ? k1 : k0;
    const int per_sm = tws ? n1 : n0;
    int dev = 0, nsm = 148;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    cuda_check(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "attribute");
    const long long nitems = (long long)((a.ny + NB - 1) / NB) * npl;
    const int grid = int(std::min<long long>(nitems, (long long)nsm * per_sm));
    kern<<<grid, Cfg::THREADS, smem, st>>>(a, npl, err);
    cuda_check(cudaGetLastError(), "k_ucol_fwd_bulk launch");
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return true;
  }
  template <int LOGM>
  static void run1(bool bwd, const ColArgs &a, int npl, cudaStream_t st, int *err) {
    constexpr int M = 1 << LOGM;
    using Cfg = ColCfg<R, M>;
    if constexpr (sizeof(R) == 8 && LOGM == 13) {
      // FP64 8192-point transforms: one column a CTA, the last stage's
      // twiddles from global memory
      const size_t smem = ColBig<M>::bytes();
      auto *kern = bwd ? k_ucol_bwd_big<LOGM> : k_ucol_fwd_big<LOGM>;
      smem_attr(kern, smem);
      dim3 grid(a.ny, npl);
      kern<<<grid, ColBig<M>::TPF, smem, st>>>(a);
      cuda_check(cudaGetLastError(), bwd ? "k_ucol_bwd_big launch" : "k_ucol_fwd_big launch");
      g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    } else {
      run1s<LOGM>(bwd, a, npl, st, err);
    }
  }
  template <int LOGM>
  static void run1s(bool bwd, const ColArgs &a, int npl, cudaStream_t st, int *err) {
    constexpr int M = 1 << LOGM;
    using Cfg = ColCfg<R, M>;
    if (LOGM == 13 && run_quad(bwd, a, npl, st, err)) return;
    if (bwd && run_tma<LOGM>(a, npl, st, err)) return;
    if (!bwd && run_bulk<LOGM>(a, npl, st, err)) return;
    if constexpr (sizeof(R) == 4 && Cfg::NB == 1) {
      // one-column CTAs: two columns a CTA, loaded or stored together
      const size_t smem = (2 * size_t(FftBuf<M>::value) + M) * 2 * sizeof(R);
      auto *kern = bwd ? k_ucol_bwd_pair<R, LOGM> : k_ucol_fwd_pair<R, LOGM>;
      smem_attr(kern, smem);
      dim3 grid((a.ny + 1) / 2, npl);
      kern<<<grid, Cfg::THREADS, smem, st>>>(a);
      cuda_check(cudaGetLastError(), bwd ? "k_ucol_bwd_pair launch" : "k_ucol_fwd_pair launch");
      g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
      return;
    }
    const size_t smem = ColSmem2<R, M>::bytes();
    dim3 grid((a.ny + Cfg::NB - 1) / Cfg::NB, npl);
    if (bwd) {
      smem_attr(k_ucol_bwd<R, LOGM>, smem);
      k_ucol_bwd<R, LOGM><<<grid, Cfg::THREADS, smem, st>>>(a);
    } else {
      // the forward kernel keeps its twist tables in shared memory when they
      // fit without costing a resident CTA
      const size_t extra = size_t(a.K) * (M / 16 + 32) * 2 * sizeof(R);
      if (twist_tables_fit(smem, extra)) {
        smem_attr(k_ucol_fwd<R, LOGM, true>, smem + extra);
        k_ucol_fwd<R, LOGM, true><<<grid, Cfg::THREADS, smem + extra, st>>>(a);
      } else {
        smem_attr(k_ucol_fwd<R, LOGM, false>, smem);
        k_ucol_fwd<R, LOGM, false><<<grid, Cfg::THREADS, smem, st>>>(a);
      }
    }
    cuda_check(cudaGetLastError(), bwd ? "k_ucol_bwd launch" : "k_ucol_fwd launch");
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  }
  // err: the device error word (bit 2: a staged copy did not complete), or
  // nullptr to stay with the plain loads (either direction)
  static void run(int logM, bool bwd, const ColArgs &a, int npl, cudaStream_t st,
                  int *err = nullptr) {
    switch (logM) {
      case 8: run1<8>(bwd, a, npl, st, err); break;
      case 9: run1<9>(bwd, a, npl, st, err); break;
      case 10: run1<10>(bwd, a, npl, st, err); break;
      case 11: run1<11>(bwd, a, npl, st, err); break;
      case 12: run1<12>(bwd, a, npl, st, err); break;
      case 13: run1<13>(bwd, a, npl, st, err); break;
      default: throw std::runtime_error("unsupported pruned FFT length");
    }
  }
};

}  // namespace

template <typename R>
void grid_dispatch(int W, bool spread, int nsm, cudaStream_t st, const GridArgs &a,
                   const DevGeom &g, const DevKernel<R> &kc) {
  GridKernels<R>::dispatch(W, spread, nsm, st, a, g, kc);
}
template <typename R>
void col_run(int logM, bool bwd, const ColArgs &a, int npl, cudaStream_t st, int *err) {
  ColKernels<R>::run(logM, bwd, a, npl, st, err);
}
template <int LOGM>
void row_run1(bool bwd, const RowArgs &a, int nsm, cudaStream_t st) {
  using Cfg = RowCfg<(1 << LOGM)>;
  // the twist factors multiplied out when that costs no resident CTA
  auto pick = [&](bool full, int &occ, size_t &smem) {
    auto *fn = bwd ? (full ? k_vrow_bwd<LOGM, true> : k_vrow_bwd<LOGM, false>)
                   : (full ? k_vrow_fwd<LOGM, true> : k_vrow_fwd<LOGM, false>);
    smem = Cfg::smem(a.K, full);
    occ = 0;
    if (smem > kMaxSmemPerBlock) return fn;
    smem_attr(fn, smem);
    occ = resident_ctas(reinterpret_cast<const void *>(fn), Cfg::THREADS, smem);
    return fn;
  };
  int occ = 0, occ_full = 0;
  size_t smem = 0, smem_full = 0;
  auto *fn = pick(false, occ, smem);
  auto *fn_full = pick(true, occ_full, smem_full);
  if (occ_full >= occ) {
    fn = fn_full;
    occ = occ_full;
    smem = smem_full;
  }
  require(occ > 0, "internal: row transform exceeds shared memory");
  const long long items = (a.nrow + Cfg::NB - 1) / Cfg::NB;
  fn<<<unsigned(std::min<long long>(items, (long long)nsm * occ)), Cfg::THREADS, smem, st>>>(a);
  cuda_check(cudaGetLastError(), "row transform launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
// 8192 points: four of 2048 (k_vrow_fwd_quad stages a whole transformed row,
// and rows of more than some 16000 entries stay with k_vrow_fwd).
void row_run_quad(bool bwd, const RowArgs &a, int nsm, cudaStream_t st) {
  const size_t smem = bwd ? QuadRow::bwd_bytes(a.K) : QuadRow::fwd_bytes(a.ncol, a.K);
  if (smem > kMaxSmemPerBlock) return row_run1<13>(bwd, a, nsm, st);
  auto *fn = bwd ? k_vrow_bwd_quad : k_vrow_fwd_quad;
  smem_attr(fn, smem);
  fn<<<unsigned(std::min<long long>(a.nrow, nsm)), Quad::THREADS, smem, st>>>(a);
  cuda_check(cudaGetLastError(), "row transform launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void row_run(int logM, bool bwd, const RowArgs &a, int nsm, cudaStream_t st) {
  switch (logM) {
    case 8: row_run1<8>(bwd, a, nsm, st); break;
    case 9: row_run1<9>(bwd, a, nsm, st); break;
    case 10: row_run1<10>(bwd, a, nsm, st); break;
    case 11: row_run1<11>(bwd, a, nsm, st); break;
    case 12: row_run1<12>(bwd, a, nsm, st); break;
    case 13: row_run_quad(bwd, a, nsm, st); break;
    default: throw std::runtime_error("unsupported pruned FFT length");
  }
}
template <typename R>
void launch_screen_add(dim3 grid, cudaStream_t st, const ScreenArgs &s, const void *H,
                       double *img, void *out, int out_mode) {
  k_screen_add<R><<<grid, 256, 0, st>>>(s, H, img, out, out_mode);
  cuda_check(cudaGetLastError(), "k_screen_add launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
template <typename R>
void launch_screen_put(dim3 grid, cudaStream_t st, const ScreenArgs &s, const void *img,
                       int in_f32, void *H) {
  k_screen_put<R><<<grid, 256, 0, st>>>(s, img, in_f32, H);
  cuda_check(cudaGetLastError(), "k_screen_put launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

template <typename R>
void launch_screen_add_grid(dim3 grid, cudaStream_t st, const ScreenArgs &s, const void *G,
                            double *img, void *out, int out_mode) {
  k_screen_add_grid<R><<<grid, 256, 0, st>>>(s, G, img, out, out_mode);
  cuda_check(cudaGetLastError(), "k_screen_add_grid launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
template <typename R>
void launch_screen_put_grid(dim3 grid, cudaStream_t st, const ScreenArgs &s, const void *img,
                            int in_f32, void *G) {
  k_screen_put_grid<R><<<grid, 256, 0, st>>>(s, img, in_f32, G);
  cuda_check(cudaGetLastError(), "k_screen_put_grid launch");
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

#define WSG_LAUNCHERS(R)                                                                     \
  template void grid_dispatch<R>(int, bool, int, cudaStream_t, const GridArgs &,             \
                                 const DevGeom &, const DevKernel<R> &);                     \
  template void col_run<R>(int, bool, const ColArgs &, int, cudaStream_t, int *);            \
  template void launch_screen_add<R>(dim3, cudaStream_t, const ScreenArgs &, const void *,  \
                                     double *, void *, int);                                 \
  template void launch_screen_put<R>(dim3, cudaStream_t, const ScreenArgs &, const void *,  \
                                     int, void *);                                           \
  template void launch_screen_add_grid<R>(dim3, cudaStream_t, const ScreenArgs &,            \
                                          const void *, double *, void *, int);             \
  template void launch_screen_put_grid<R>(dim3, cudaStream_t, const ScreenArgs &,            \
                                          const void *, int, void *);
WSG_LAUNCHERS(float)
WSG_LAUNCHERS(double)
#undef WSG_LAUNCHERS

}  // namespace wsg
