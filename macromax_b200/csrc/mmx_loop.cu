// Configuration and launchers of the chunks in one launch (mmx_loop.cuh); one translation unit per precision.
#include <algorithm>
#include <atomic>

#include "mmx_loop.cuh"
#include "mmx_loop.h"

namespace {

constexpr size_t kSmemMax = 220 * 1024;

template <class R, int C, int CHI> cudaError_t prepare_kernels() {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(k_loop<R, C, CHI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_line<R, C, CHI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

template <class F> auto by_chi(int C, int chi_kind, F&& f) {
  if (C == 1) return f(std::integral_constant<int, 1>{}, std::integral_constant<int, MMX_CHI_SCALAR>{});
  if (chi_kind == MMX_CHI_SCALAR) return f(std::integral_constant<int, 3>{}, std::integral_constant<int, MMX_CHI_SCALAR>{});
  if (chi_kind == MMX_CHI_SYM6) return f(std::integral_constant<int, 3>{}, std::integral_constant<int, MMX_CHI_SYM6>{});
  return f(std::integral_constant<int, 3>{}, std::integral_constant<int, MMX_CHI_MAT3>{});
}

// The tile width (pencils or rows) that ends a pass over `pencils` per copy soonest on `ctas` CTAs: rounds of tiles, each
// with a constant part (first loads, barriers) and, per stage, the butterflies of its busiest thread.
int best_width(const GenAxis& g, int64_t pencils, int copies, int C, int ctas, int lo, int hi, bool pow2, size_t word_bytes,
               size_t cap) {
  int best = 0;
  double best_cost = 0;
  for (int P = lo; P <= hi; P = pow2 ? 2 * P : P + 1) {
    if (2 * (size_t)C * P * (g.n + (g.n >> 3)) * word_bytes > cap && best) break;
    const int64_t tiles = (pencils + P - 1) / P;
    const int64_t rounds = (tiles * copies + ctas - 1) / ctas;
    double cost = 40;
    for (int s = 0; s < g.nst; ++s) {
      const int64_t per = pow2 ? (C * g.T[s] + kLoopWorkers / P - 1) / (kLoopWorkers / P)
                               : ((int64_t)C * P * g.T[s] + kLoopWorkers - 1) / kLoopWorkers;
      cost += per * (g.r[s] + 8);
    }
    cost *= rounds;
    if (!best || cost < best_cost) {
      best = P;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace

template <class R> LoopCfg loop_config(int ndim, const int64_t* shape, int C, int chi_kind, int B, int sms) {
  LoopCfg c;
  const bool dbl = sizeof(R) == 8;
  int64_t N = 1;
  for (int i = 0; i < ndim; ++i) N *= shape[i];
  if (N > (int64_t)1 << 28 || B > 65535) return c;
  for (int k = 0; k < 3; ++k) {
    if (k == 1 && ndim != 3) continue;
    if (!gen_small_plan((int)shape[k == 2 ? ndim - 1 : k], &c.g[k])) return c;
  }
  const cudaError_t e = by_chi(C, chi_kind, [](auto cc, auto chi) {
    return prepare_kernels<R, decltype(cc)::value, decltype(chi)::value>();
  });
  if (e != cudaSuccess) {
    cudaGetLastError();
    return c;
  }
  if (ndim == 1) {
    const int M = chi_kind == MMX_CHI_SCALAR ? 1 : chi_kind == MMX_CHI_SYM6 ? 6 : 9;
    c.line = true;
    c.staged = line_bytes<R>((int)N, C, M, true) <= kSmemMax;
    c.smem = line_bytes<R>((int)N, C, M, c.staged);
    c.grid = B;
    c.ok = c.smem <= kSmemMax;
    return c;
  }
  if (B > kLoopMaxRhs) return c;
  const size_t word = 2 * sizeof(R);
  const int kept_words = by_chi(C, chi_kind, [](auto cc, auto chi) { return kLoopKept<decltype(cc)::value, decltype(chi)::value>; });
  auto tiles = [](int64_t pencils, int P) { return (int)((pencils + P - 1) / P); };
  for (int per_sm = 2; per_sm >= 1; --per_sm) {
    const int ctas = sms * per_sm;
    const size_t cap = 100 * 1024 / per_sm;
    const int floor = dbl ? 2 : 4;  // one 32-byte sector of a row
    const int64_t last = shape[ndim - 1];
    const int P0 = best_width(c.g[0], N / shape[0], B, C, ctas, floor, 16, true, word, cap);
    const int P1 = ndim == 3 ? best_width(c.g[1], N / shape[1], B * C, 1, ctas, floor, 16, true, word, cap) : 1;
    c.PR = best_width(c.g[2], N / last, B, C, ctas, 1, 32, false, word, cap);
    for (c.lP0 = 0; (1 << c.lP0) < P0;) ++c.lP0;
    for (c.lP1 = 0; (1 << c.lP1) < P1;) ++c.lP1;
    c.tiles[0] = tiles(N / shape[0], P0);
    c.tiles[1] = ndim == 3 ? tiles(N / shape[1], P1) : 0;
    c.tiles[2] = tiles(N / last, c.PR);
    const int64_t most = std::max<int64_t>((int64_t)B * c.tiles[2], std::max<int64_t>((int64_t)B * c.tiles[0],
                                                                                    (int64_t)B * C * c.tiles[1]));
    if (most > 1 << 30) return c;
    c.grid = (int)std::min<int64_t>(std::min(ctas, (int)kLeaveGaveUp - 1), most);
    c.kept = (int)(((int64_t)B * c.tiles[2] + c.grid - 1) / c.grid);
    size_t work = 2 * (size_t)C * shape[0] * P0 * word;
    work = std::max(work, 2 * (size_t)C * c.PR * last * word);
    if (ndim == 3) work = std::max(work, 2 * (size_t)shape[1] * P1 * word);
    c.smem = LoopShared<R>(c.g, ndim, B, (size_t)c.kept * kept_words * c.PR * last * word, work).bytes;
    if (c.smem > kSmemMax / per_sm) continue;
    int fit = 0;
    const cudaError_t q = by_chi(C, chi_kind, [&](auto cc, auto chi) {
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_loop<R, decltype(cc)::value, decltype(chi)::value>,
                                                           kLoopThreads, c.smem);
    });
    if (q != cudaSuccess) {
      cudaGetLastError();
      return c;
    }
    if (fit < per_sm) continue;
    c.ok = true;
    return c;
  }
  return c;
}

template <class R>
cudaError_t loop_launch(const LoopCfg& cfg, const IterArgs<R>& base, const FFTAxis* tab, int C, int chi_kind, int B,
                        int niter, unsigned polls, unsigned* counter, cudaStream_t s) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)cfg.grid);
  lc.dynamicSmemBytes = cfg.smem;
  lc.stream = s;
  if (cfg.line) {
    LineArgs<R> a;
    static_cast<IterArgs<R>&>(a) = base;
    a.ax = tab[0];
    a.g = cfg.g[2];
    a.niter = niter;
    a.staged = cfg.staged;
    lc.blockDim = dim3(kLineThreads);
    return by_chi(C, chi_kind, [&](auto cc, auto chi) {
      return cudaLaunchKernelEx(&lc, k_line<R, decltype(cc)::value, decltype(chi)::value>, a);
    });
  }
  LoopArgs<R> a;
  static_cast<IterArgs<R>&>(a) = base;
  a.nrhs = B;
  for (int k = 0; k < 3; ++k) {
    a.g[k] = cfg.g[k];
    a.tiles[k] = cfg.tiles[k];
  }
  a.tab[0] = tab[0];
  a.tab[1] = tab[1];
  a.tab[2] = tab[base.ndim - 1];
  a.lP0 = cfg.lP0;
  a.lP1 = cfg.lP1;
  a.PR = cfg.PR;
  a.kept = cfg.kept;
  a.niter = niter;
  a.polls = polls;
  a.counter = counter;
  lc.blockDim = dim3(kLoopThreads);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // all CTAs are resident: they wait for one another
  attr[0].val.cooperative = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  return by_chi(C, chi_kind, [&](auto cc, auto chi) {
    return cudaLaunchKernelEx(&lc, k_loop<R, decltype(cc)::value, decltype(chi)::value>, a);
  });
}

#ifdef MMX_GEN_DOUBLE
template LoopCfg loop_config<double>(int, const int64_t*, int, int, int, int);
template cudaError_t loop_launch<double>(const LoopCfg&, const IterArgs<double>&, const FFTAxis*, int, int, int, int,
                                         unsigned, unsigned*, cudaStream_t);
#else
template LoopCfg loop_config<float>(int, const int64_t*, int, int, int, int);
template cudaError_t loop_launch<float>(const LoopCfg&, const IterArgs<float>&, const FFTAxis*, int, int, int, int, unsigned,
                                        unsigned*, cudaStream_t);
#endif
