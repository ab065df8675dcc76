// Radix plans, tiles and launchers of the passes for axes of any length (mmx_gen.cuh).
#include <algorithm>
#include <atomic>

#include "mmx_gen.cuh"

namespace {

constexpr size_t kSmemCap = 220 * 1024;

}  // namespace

#ifndef MMX_GEN_DOUBLE  // plans and tiles, for both precisions
namespace {

// The radices of n, 2 .. 16 each: the fewest stages (at least two), then the smallest sum.  False if there are none in
// MMX_GEN_STAGES stages.
bool best_radices(int n, int stages, int top, int* r, int* sum) {
  if (stages == 1) {
    if (n < 2 || n > top) return false;
    r[0] = n;
    *sum = n;
    return true;
  }
  bool found = false;
  for (int f = std::min(top, n); f >= 2; --f) {
    if (n % f) continue;
    int rest[MMX_GEN_STAGES], s = 0;
    if (best_radices(n / f, stages - 1, f, rest, &s) && (!found || s + f < *sum)) {
      found = true;
      *sum = s + f;
      r[0] = f;
      for (int i = 1; i < stages; ++i) r[i] = rest[i - 1];
    }
  }
  return found;
}

void fill_axis(int n, int nst, const int* r, GenAxis* ax) {
  auto reciprocal = [](int d) { return d > 1 ? (unsigned)((1ull << 32) / d + 1) : 0u; };
  *ax = GenAxis();
  ax->n = n;
  ax->nst = nst;
  int L = 1;
  for (int s = 0; s < nst; ++s) {
    ax->r[s] = r[s];
    ax->T[s] = n / r[s];
    ax->L[s] = L;
    ax->ts[s] = n / r[s] / L;
    ax->mT[s] = reciprocal(ax->T[s]);
    ax->mL[s] = reciprocal(L);
    L *= r[s];
  }
  ax->mn = reciprocal(n);
}

// largest_first: the radices in descending order, else ascending
bool plan_axis(int n, bool largest_first, GenAxis* ax) {
  int r[MMX_GEN_STAGES], sum = 0, nst = 0;
  for (int stages = 2; stages <= 4 && !nst; ++stages)
    if (best_radices(n, stages, 16, r, &sum)) nst = stages;
  if (!nst) return false;
  if (!largest_first) std::reverse(r, r + nst);
  fill_axis(n, nst, r, ax);
  return true;
}

bool is_rows(GenKind k) { return k != GEN_STRIDED && k != GEN_GREEN; }

size_t tile_bytes(GenKind kind, const GenAxis& ax, int C, int P, bool dbl) {
  const size_t wb = dbl ? 16 : 8;
  const size_t n = ax.n;
  const size_t tables = n * 16;  // the twiddles: two floats or a double per part
  if (kind == GEN_STRIDED) return n * P * (ax.nst > 2 ? 2 : 1) * wb + tables;
  if (kind == GEN_GREEN) return 2 * C * n * P * wb + tables + n * sizeof(double);
  const size_t pitch = n + (n >> (dbl ? 3 : 4));
  const bool two = ax.nst > 2 || kind == GEN_PRO3 || kind == GEN_EPI3;
  return C * P * pitch * (two ? 2 : 1) * wb + tables;
}

}  // namespace

bool gen_small_plan(int n, GenAxis* ax) {
  int r[MMX_GEN_STAGES], primes = 0, m = n;
  for (int f : {13, 11})
    while (m % f == 0) {
      if (primes == MMX_GEN_STAGES) return false;
      r[primes++] = f;
      m /= f;
    }
  int nst = primes;
  if (m > 1) {
    int sum = 0;
    bool found = false;
    for (int stages = primes ? 1 : 2; !found && primes + stages <= MMX_GEN_STAGES; ++stages)
      if (best_radices(m, stages, 10, r + primes, &sum)) {
        found = true;
        nst = primes + stages;
      }
    if (!found) return false;
  }
  if (nst < 2) return false;
  fill_axis(n, nst, r, ax);
  return true;
}

GenTile gen_tile(GenKind kind, int n, int C, bool dbl, int64_t outer, int64_t inner, int64_t copies, int sms) {
  GenTile t;
  // the epilogue loads E and chi beside its last butterflies, the prologue beside its first: the smallest radix there
  if (!plan_axis(n, kind == GEN_EPI || kind == GEN_GREEN || kind == GEN_STRIDED, &t.ax)) return t;
  const int64_t pencils = outer * inner;
  if (pencils * n > (int64_t)1 << 31) return t;  // 32-bit offsets within a component
  const bool rows = is_rows(kind);
  int maxT = 0;
  for (int s = 0; s < t.ax.nst; ++s) maxT = std::max(maxT, t.ax.T[s]);
  // narrower tiles while the launch has fewer than two per SM, down to one 32-byte sector of a row
  int P = gen_width(kind, C, dbl, maxT);
  const int full = P, floor = rows ? 1 : dbl ? 2 : 4;
  while (P > floor && ((pencils + P - 1) / P) * copies < 2 * (int64_t)sms) P /= 2;
  while (P > floor && tile_bytes(kind, t.ax, C, P, dbl) > 72 * 1024) P /= 2;
  if (tile_bytes(kind, t.ax, C, P, dbl) > kSmemCap) return t;
  t.lP = 0;
  while ((1 << t.lP) < P) ++t.lP;
  t.fixed = P == full && len_has(n) && pencils < (int64_t)1 << 31;
  const int* r = t.ax.r;
  t.threads = gen_threads(t.ax.nst, r[0], r[1], t.ax.nst > 2 ? r[2] : 1, t.ax.nst > 3 ? r[3] : 1, n, C, P, rows,
                          (long)tile_bytes(kind, t.ax, C, P, dbl));
  t.smem = tile_bytes(kind, t.ax, C, P, dbl);
  t.tiles = (pencils + P - 1) / P;
  if (t.tiles > 0x7fffffff) t.threads = 0;
  return t;
}
#endif  // MMX_GEN_DOUBLE

namespace {

// Raise the kernel's dynamic shared-memory limit once per device; one static word per kernel instantiation.
cudaError_t allow_smem(std::atomic<uint64_t>& done, const void* kern) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

template <class R, auto Kern>
cudaError_t launch(const GenTile& t, const GenArgs<R>& a, int copies, bool pdl, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  const cudaError_t e = allow_smem(done, (const void*)Kern);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)t.tiles, (unsigned)copies);
  cfg.blockDim = dim3((unsigned)t.threads);
  cfg.dynamicSmemBytes = t.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, Kern, a);
}

}  // namespace

template <class R>
cudaError_t gen_launch(GenKind kind, const GenTile& t, const IterArgs<R>& base, int C, int chi_kind, int dir, int batch,
                       const void* in, void* out, R scale, bool pdl, cudaStream_t s) {
  if (t.fixed && chi_kind != MMX_CHI_MAT3) {
    static_assert(kLenParts == 4, "one case per part");
    switch (t.ax.n % kLenParts) {
      case 0: return len_launch<R, 0>(kind, t, base, C, dir, batch, in, out, scale, pdl, s);
      case 1: return len_launch<R, 1>(kind, t, base, C, dir, batch, in, out, scale, pdl, s);
      case 2: return len_launch<R, 2>(kind, t, base, C, dir, batch, in, out, scale, pdl, s);
      default: return len_launch<R, 3>(kind, t, base, C, dir, batch, in, out, scale, pdl, s);
    }
  }
  GenArgs<R> a;
  static_cast<IterArgs<R>&>(a) = base;
  a.g = t.ax;
  a.lP = t.lP;
  a.C = C;
  a.in = (const cpx<R>*)in;
  a.out = (cpx<R>*)out;
  a.scale = scale;
  switch (kind) {
    case GEN_STRIDED:
      return dir < 0 ? launch<R, k_gen_strided<R, -1>>(t, a, batch, pdl, s)
                     : launch<R, k_gen_strided<R, +1>>(t, a, batch, pdl, s);
    case GEN_GREEN:
      return C == 3 ? launch<R, k_gen_green<R, 3>>(t, a, batch, pdl, s) : launch<R, k_gen_green<R, 1>>(t, a, batch, pdl, s);
    case GEN_ROWS:
      return dir < 0 ? launch<R, k_gen_rows<R, GEN_ROWS, MMX_CHI_SCALAR, -1>>(t, a, batch, pdl, s)
                     : launch<R, k_gen_rows<R, GEN_ROWS, MMX_CHI_SCALAR, +1>>(t, a, batch, pdl, s);
    case GEN_PRO: return launch<R, k_gen_rows<R, GEN_PRO, MMX_CHI_SCALAR, -1>>(t, a, batch, pdl, s);
    case GEN_EPI: return launch<R, k_gen_rows<R, GEN_EPI, MMX_CHI_SCALAR, +1>>(t, a, batch, pdl, s);
    case GEN_PRO3:
      return chi_kind == MMX_CHI_SYM6 ? launch<R, k_gen_rows<R, GEN_PRO3, MMX_CHI_SYM6, -1>>(t, a, batch, pdl, s)
                                      : launch<R, k_gen_rows<R, GEN_PRO3, MMX_CHI_MAT3, -1>>(t, a, batch, pdl, s);
    case GEN_EPI3:
      return chi_kind == MMX_CHI_SYM6 ? launch<R, k_gen_rows<R, GEN_EPI3, MMX_CHI_SYM6, +1>>(t, a, batch, pdl, s)
                                      : launch<R, k_gen_rows<R, GEN_EPI3, MMX_CHI_MAT3, +1>>(t, a, batch, pdl, s);
  }
  return cudaErrorInvalidValue;
}

// one translation unit per precision (MMX_GEN_DOUBLE), so that they compile side by side
#ifdef MMX_GEN_DOUBLE
template cudaError_t gen_launch<double>(GenKind, const GenTile&, const IterArgs<double>&, int, int, int, int, const void*,
                                        void*, double, bool, cudaStream_t);
#else
template cudaError_t gen_launch<float>(GenKind, const GenTile&, const IterArgs<float>&, int, int, int, int, const void*,
                                       void*, float, bool, cudaStream_t);
#endif
