// Launchers of the passes compiled for one length (mmx_len.cuh).  One translation unit per precision (MMX_LEN_DOUBLE) and
// part (MMX_LEN_PART: the lengths n with n % kLenParts == MMX_LEN_PART), given on the command line.
#include <atomic>

#include "mmx_len.cuh"

namespace {

#if MMX_LEN_DOUBLE
using Real = double;
#else
using Real = float;
#endif

template <auto Kern>
cudaError_t launch(int threads, size_t smem, const GenTile& t, const LenArgs<Real>& a, int copies, bool pdl, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};  // devices on which the kernel's shared-memory limit is raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (!bit || !(done.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    done.fetch_or(bit, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)t.tiles, (unsigned)copies);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, Kern, a);
}

template <int N, class F> cudaError_t for_length(GenKind kind, int C, int dir, F&& f) {
  if constexpr (!len_has(N)) {
    return cudaErrorInvalidValue;
  } else {
    auto rows = [&](auto k, auto c, auto d) {
      constexpr int K = decltype(k)::value, CC = decltype(c)::value;
      using G = LenRows<Real, K, CC, N>;
      return f(std::integral_constant<void (*)(LenArgs<Real>), k_len_rows<Real, K, CC, decltype(d)::value, N>>{}, G::THREADS,
               G::SMEM, G::P);
    };
    using I1 = std::integral_constant<int, 1>;
    using I3 = std::integral_constant<int, 3>;
    using Fwd = std::integral_constant<int, -1>;
    using Inv = std::integral_constant<int, +1>;
    using S = LenStrided<Real, N>;
    using G1 = LenGreen<Real, 1, N>;
    using G3 = LenGreen<Real, 3, N>;
    switch (kind) {
      case GEN_STRIDED:
        return dir < 0 ? f(std::integral_constant<void (*)(LenArgs<Real>), k_len_strided<Real, -1, N>>{}, S::THREADS, S::SMEM, S::P)
                       : f(std::integral_constant<void (*)(LenArgs<Real>), k_len_strided<Real, +1, N>>{}, S::THREADS, S::SMEM, S::P);
      case GEN_GREEN:
        return C == 3 ? f(std::integral_constant<void (*)(LenArgs<Real>), k_len_green<Real, 3, N>>{}, G3::THREADS, G3::SMEM, G3::P)
                      : f(std::integral_constant<void (*)(LenArgs<Real>), k_len_green<Real, 1, N>>{}, G1::THREADS, G1::SMEM, G1::P);
      case GEN_ROWS:
        return dir < 0 ? rows(std::integral_constant<int, GEN_ROWS>{}, I1{}, Fwd{})
                       : rows(std::integral_constant<int, GEN_ROWS>{}, I1{}, Inv{});
      case GEN_PRO:
        return C == 3 ? rows(std::integral_constant<int, GEN_PRO>{}, I3{}, Fwd{})
                      : rows(std::integral_constant<int, GEN_PRO>{}, I1{}, Fwd{});
      case GEN_EPI:
        return C == 3 ? rows(std::integral_constant<int, GEN_EPI>{}, I3{}, Inv{})
                      : rows(std::integral_constant<int, GEN_EPI>{}, I1{}, Inv{});
      case GEN_PRO3: return rows(std::integral_constant<int, GEN_PRO3>{}, I3{}, Fwd{});
      case GEN_EPI3: return rows(std::integral_constant<int, GEN_EPI3>{}, I3{}, Inv{});
    }
    return cudaErrorInvalidValue;
  }
}

template <int N, class F> cudaError_t find_length(int n, GenKind kind, int C, int dir, F&& f) {
  if constexpr (N > kLenLast) {
    return cudaErrorInvalidValue;
  } else {
    if (n == N) return for_length<N>(kind, C, dir, f);
    return find_length<N + kLenParts>(n, kind, C, dir, f);
  }
}

}  // namespace

template <>
cudaError_t len_launch<Real, MMX_LEN_PART>(GenKind kind, const GenTile& t, const IterArgs<Real>& base, int C, int dir,
                                           int batch, const void* in, void* out, Real scale, bool pdl, cudaStream_t s) {
  LenArgs<Real> a;
  static_cast<IterArgs<Real>&>(a) = base;
  a.C = C;
  a.in = (const cpx<Real>*)in;
  a.out = (cpx<Real>*)out;
  a.scale = scale;
  constexpr int first = kLenFirst + (MMX_LEN_PART + kLenParts - kLenFirst % kLenParts) % kLenParts;
  return find_length<first>(t.ax.n, kind, C, dir, [&](auto kern, int threads, size_t smem, int P) {
    if (P != 1 << t.lP) return cudaErrorInvalidValue;
    return launch<decltype(kern)::value>(threads, smem, t, a, batch, pdl, s);
  });
}
