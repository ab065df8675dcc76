// FFT passes of the iteration (and of mmx_fftn) for axes of any length with prime factors up to 13, complex64 and
// complex128.
//
// Self-sorting stages as in mmx_fft.cuh, but with radices up to 16 (two stages up to 256 samples, three up to 4096), so
// that a pass exchanges its samples through shared memory once or twice, and as in mmx_reg.cuh the first stage reads
// global memory into registers and the last one writes it (or the epilogue's results) from registers.  The length is a
// run-time value: a stage is a switch over the radix around a fully unrolled butterfly, and the only divisions left,
// of a butterfly's index by the stage's span and of a flat index by the butterflies per pencil, are multiplications by
// a reciprocal that the host computes.  Stages between two shared-memory buffers need one barrier each.  What bounds
// the passes is the issue of instructions (44-66% of the slots at 100 x 126 x 90, a third of them for addresses and indices;
// mmx_len.cuh is these passes with the length known to the compiler); the runtime-radix passes of mmx_kernels.cuh
// (staged through shared memory at both ends, out-of-line stages at a 64-register budget, integer divisions per element,
// twiddles from global memory and O(r^2) butterflies for 7, 11 and 13) take three to four times as long (520 us per
// iteration of that grid against 145).
//
// Strided tiles: P = 2^lP consecutive pencils, shared memory [component][sample][pencil]; a warp's accesses are whole
// rows.  Contiguous tiles: P rows of every component, shared memory [row][sample] with a skew of one word per 128 bytes.
#pragma once
#include <cfloat>
#include <math_constants.h>
#include <type_traits>

#include "mmx_dft.cuh"
#include "mmx_gen.h"

template <class R> struct GenArgs : IterArgs<R> {
  GenAxis g;
  int lP;
  int C;
  const cpx<R>* in;
  cpx<R>* out;
  R scale;
};

// A twiddle factor in shared memory: in complex64 as the sum of two floats, for the same reason as the coefficients of
// mmx_dft.cuh (a length without tw_lo takes it as 0).
template <class R> struct GenTw;
template <> struct GenTw<float> {
  using type = float4;
  static __device__ __forceinline__ float4 load(const FFTAxis& ax, int t) {
    const float2 h = ((const float2*)ax.tw)[t];
    const float2 l = ax.tw_lo ? ((const float2*)ax.tw_lo)[t] : make_float2(0.f, 0.f);
    return make_float4(h.x, h.y, l.x, l.y);
  }
  // u w (DIR < 0) or u conj(w)
  template <int DIR> static __device__ __forceinline__ float2 mul(float2 u, float4 w) {
    if (DIR > 0) {
      w.y = -w.y;
      w.w = -w.w;
    }
    return make_float2(fmaf(u.x, w.x, fmaf(-u.y, w.y, fmaf(u.x, w.z, -u.y * w.w))),
                       fmaf(u.x, w.y, fmaf(u.y, w.x, fmaf(u.x, w.w, u.y * w.z))));
  }
};
template <> struct GenTw<double> {
  using type = double2;
  static __device__ __forceinline__ double2 load(const FFTAxis& ax, int t) { return ((const double2*)ax.tw)[t]; }
  template <int DIR> static __device__ __forceinline__ double2 mul(double2 u, double2 w) {
    return DIR > 0 ? u * conjc(w) : u * w;
  }
};
template <class R> using gtw = typename GenTw<R>::type;

__device__ __forceinline__ unsigned gen_div(unsigned x, unsigned m) { return __umulhi(x, m); }

// Radix policies: f(integral_constant<radix>) for the stage's radix.
struct WideRadices {  // 2 .. 16: few stages, so few exchanges and addresses, for passes of many tiles
  template <class F> static __device__ __forceinline__ void run(int r, F&& f) {
    switch (r) {
      case 2: f(std::integral_constant<int, 2>{}); break;
      case 3: f(std::integral_constant<int, 3>{}); break;
      case 4: f(std::integral_constant<int, 4>{}); break;
      case 5: f(std::integral_constant<int, 5>{}); break;
      case 6: f(std::integral_constant<int, 6>{}); break;
      case 7: f(std::integral_constant<int, 7>{}); break;
      case 8: f(std::integral_constant<int, 8>{}); break;
      case 9: f(std::integral_constant<int, 9>{}); break;
      case 10: f(std::integral_constant<int, 10>{}); break;
      case 11: f(std::integral_constant<int, 11>{}); break;
      case 12: f(std::integral_constant<int, 12>{}); break;
      case 13: f(std::integral_constant<int, 13>{}); break;
      case 14: f(std::integral_constant<int, 14>{}); break;
      case 15: f(std::integral_constant<int, 15>{}); break;
      default: f(std::integral_constant<int, 16>{}); break;
    }
  }
};
struct SmallRadices {  // up to 10 and the primes: shorter butterflies on more threads, for launches bound by latency
  template <class F> static __device__ __forceinline__ void run(int r, F&& f) {
    switch (r) {
      case 2: f(std::integral_constant<int, 2>{}); break;
      case 3: f(std::integral_constant<int, 3>{}); break;
      case 4: f(std::integral_constant<int, 4>{}); break;
      case 5: f(std::integral_constant<int, 5>{}); break;
      case 6: f(std::integral_constant<int, 6>{}); break;
      case 7: f(std::integral_constant<int, 7>{}); break;
      case 8: f(std::integral_constant<int, 8>{}); break;
      case 9: f(std::integral_constant<int, 9>{}); break;
      case 10: f(std::integral_constant<int, 10>{}); break;
      case 11: f(std::integral_constant<int, 11>{}); break;
      default: f(std::integral_constant<int, 13>{}); break;
    }
  }
};

// Butterfly i of a stage: its inputs ld(q), the samples i + q T, twiddled, and their DFT in u.  Returns the first of its
// outputs d0 = (i - k) RAD + k, k = i mod L; the others follow at the span L.  FIRST: span 1, no twiddles; ts = T / L.
template <class R, int RAD, int DIR, bool FIRST, class Ld>
__device__ __forceinline__ int gen_dft(int i, int L, unsigned mL, int ts, const gtw<R>* tw, cpx<R>* u, Ld&& ld) {
#pragma unroll
  for (int q = 0; q < RAD; ++q) u[q] = ld(q);
  int k = 0;
  if constexpr (!FIRST) {
    if (L > 1) {
      k = i - (int)gen_div((unsigned)i, mL) * L;
      const gtw<R>* w = tw;
      const int step = k * ts;  // k n / (L RAD)
#pragma unroll
      for (int q = 1; q < RAD; ++q) {
        w += step;
        u[q] = GenTw<R>::template mul<DIR>(u[q], *w);
      }
    }
  }
  gdft<R, RAD, DIR>(u);
  return (i - k) * RAD + k;
}
// ... and st(d0, q, value) for the outputs d0 + q L
template <class R, int RAD, int DIR, bool FIRST, class Ld, class St>
__device__ __forceinline__ void gen_butterfly(int i, const GenAxis& g, int s, const gtw<R>* tw, Ld&& ld, St&& st) {
  cpx<R> u[RAD];
  const int d0 = gen_dft<R, RAD, DIR, FIRST>(i, g.L[s], g.mL[s], g.ts[s], tw, u, ld);
#pragma unroll
  for (int q = 0; q < RAD; ++q) st(d0, q, u[q]);
}

// -i alpha_i / (|k|^2 - alpha) / N (solver.py:566-568, with the 1/N of the inverse transform), in FP64 and rounded once
// (the field converges to the fixed point of the rounded g): complex64 starts the reciprocal in float and takes one
// Newton step, about ten FP64 operations per sample.  An alpha whose alpha_i^2 is beyond the range of R (an alpha that the
// divergence guard has raised a hundred times) gives NaN, as the quotient in R does: every update is then rejected and the
// residue stays infinite.  (A g of 0 would give an update of 0, which counts as converged.)
template <class R> struct GenGreen {
  double ar, ai, ai2, s;
  __device__ __forceinline__ GenGreen(double re, double im, double inv_total) : ar(re), ai(im), ai2(im * im), s(inv_total) {
    // 1 / inf = 0 makes the Newton step 0 inf
    if (sizeof(R) == 4 && ai2 > (double)FLT_MAX) ai2 = CUDART_INF;
  }
  __device__ __forceinline__ cpx<R> operator()(double k2) const {
    const double dr = k2 - ar;
    const double den = fma(dr, dr, ai2);
    double r;
    if constexpr (sizeof(R) == 4) {
      r = (double)(1.0f / (float)den);
      r = fma(r, fma(-den, r, 1.0), r);
    } else {
      r = 1.0 / den;
    }
    r *= s;
    return mkc<R>((R)(ai2 * r), (R)(-ai * dr * r));
  }
};

// k along the other axes of pencil p of axis 0 (0 beyond the field)
template <class R>
__device__ __forceinline__ void gen_pencil_k(const IterArgs<R>& a, unsigned p, double* k1, double* k2) {
  *k1 = *k2 = 0.0;
  if (p >= (unsigned)(a.N / a.dims[0])) return;
  if (a.ndim == 3) {
    const unsigned i1 = p / (unsigned)a.dims[2];
    *k1 = a.kvd[1][i1];
    *k2 = a.kvd[2][p - i1 * (unsigned)a.dims[2]];
  } else if (a.ndim == 2) {
    *k1 = a.kvd[1][p];
  }
}

// registers: 85 (complex64) and 128 (complex128) per thread at 256 threads
template <class R> struct GenBounds { static constexpr int min_blocks = sizeof(R) == 4 ? 3 : 2; };

// i alpha_i / (alpha N) (solver.py:575)
template <class R> __device__ __forceinline__ cpx<R> gen_longitudinal(double ar, double ai, double inv_total) {
  const double s = ai * inv_total / (ar * ar + ai * ai);
  return mkc<R>((R)(ai * s), (R)(ar * s));
}

// The barrier between the stages of a tile: of the whole block, or of the first `threads` threads of it.
struct BlockSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
struct PartSync {
  int threads;
  __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }
};

// ---------------------------------------------------------------------------------------------------------------
// Strided axis, FFT only: tile `tile` of the component plane `in`, to `out` (may be `in`).  sm: one buffer of P n words,
// two with more than two stages.  The first barrier publishes tables that the caller has just written.
// ---------------------------------------------------------------------------------------------------------------
template <class R, int DIR, class Rad, class Sync>
__device__ __forceinline__ void strided_tile(const GenAxis& g, int lP, unsigned inner, int64_t pencils, int64_t tile,
                                             const cpx<R>* in, cpx<R>* out, const gtw<R>* tw, cpx<R>* sm, int threads,
                                             Sync sync) {
  const int n = g.n, P = 1 << lP, nst = g.nst;
  const int pl = threadIdx.x & (P - 1), slot = threadIdx.x >> lP, nslots = threads >> lP;
  const int64_t p = (tile << lP) + pl;
  const bool valid = p < pencils;
  const int64_t o = p / inner;
  const int64_t off = o * n * inner + (p - o * inner);
  const cpx<R>* gi = in + off;
  cpx<R>* go = out + off;
  Rad::run(g.r[0], [&](auto rad) {
    constexpr int RAD = decltype(rad)::value;
    const int T = g.T[0];
    for (int i = slot; i < T; i += nslots) {
      const cpx<R>* q0 = gi + (size_t)i * inner;
      gen_butterfly<R, RAD, DIR, true>(
          i, g, 0, tw, [&](int q) { return valid ? q0[(unsigned)(q * T) * inner] : mkc<R>((R)0, (R)0); },
          [&](int d, int q, cpx<R> v) { sm[((d + q) << lP) + pl] = v; });
    }
  });
  sync();
  cpx<R>* cur = sm;
  for (int s = 1; s + 1 < nst; ++s) {
    cpx<R>* dst = cur == sm ? sm + ((size_t)n << lP) : sm;
    Rad::run(g.r[s], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = g.T[s];
      const int L = g.L[s];
      for (int i = slot; i < T; i += nslots) {
        const cpx<R>* q0 = cur + (i << lP) + pl;
        gen_butterfly<R, RAD, DIR, false>(
            i, g, s, tw, [&](int q) { return q0[(q * T) << lP]; },
            [&](int d, int q, cpx<R> v) { dst[((d + q * L) << lP) + pl] = v; });
      }
    });
    sync();
    cur = dst;
  }
  if (!valid) return;
  Rad::run(g.r[nst - 1], [&](auto rad) {
    constexpr int RAD = decltype(rad)::value;
    const int T = g.T[nst - 1];
    for (int i = slot; i < T; i += nslots) {
      const cpx<R>* q0 = cur + (i << lP) + pl;
      cpx<R>* d0 = go + (size_t)i * inner;  // the last stage's outputs are i + q T
      gen_butterfly<R, RAD, DIR, false>(
          i, g, nst - 1, tw, [&](int q) { return q0[(q * T) << lP]; },
          [&](int, int q, cpx<R> v) { d0[(unsigned)(q * T) * inner] = v; });
    }
  });
}

// blockIdx.y: component plane (right-hand side * C + component), or transform.
template <class R, int DIR>
__global__ void __launch_bounds__(256, GenBounds<R>::min_blocks) k_gen_strided(const __grid_constant__ GenArgs<R> a) {
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + a.g.n);
  for (int t = threadIdx.x; t < a.g.n; t += blockDim.x) tw[t] = GenTw<R>::load(a.ax, t);
  pdl_wait();
  pdl_trigger();
  if (a.st && !a.st[blockIdx.y / a.C].active) return;
  const int64_t plane = (int64_t)blockIdx.y * a.N;
  strided_tile<R, DIR, WideRadices>(a.g, a.lP, (unsigned)a.inner, a.outer * a.inner, blockIdx.x, a.in + plane, a.out + plane, tw, sm,
                       blockDim.x, BlockSync());
}

// ---------------------------------------------------------------------------------------------------------------
// Axis 0: forward FFT, Green multiply, inverse FFT, in place, of the tile of pencils from tile << lP of one right-hand
// side (T0: its first component).  h: i alpha_i / (alpha N), the longitudinal factor; sm: two buffers of C P n words; sk0: k
// of axis 0; k1, k2: of this thread's pencil.
// ---------------------------------------------------------------------------------------------------------------
template <class R, int C, class Rad, class Sync>
__device__ __forceinline__ void green_tile(const GenAxis& g, int lP, int ndim, unsigned inner, int64_t N, unsigned p,
                                           cpx<R>* T0, double k1, double k2, GenGreen<R> green, cpx<R> h,
                                           const gtw<R>* tw, const double* sk0, cpx<R>* sm, int threads, Sync sync) {
  const int n = g.n, P = 1 << lP, nst = g.nst;
  const size_t words = ((size_t)C * n) << lP;
  const int pl = threadIdx.x & (P - 1), slot = threadIdx.x >> lP, nslots = threads >> lP;
  const bool valid = p < inner;  // axis 0 has outer == 1: a pencil is its inner index
  cpx<R>* gp = T0 + p;
  const double kt2 = k1 * k1 + k2 * k2;
  auto component = [&](int& i, int T) {  // i in [0, C T) -> component, i mod T
    int c = 0;
    if constexpr (C == 3) {
      c = (i >= T) + (i >= 2 * T);
      i -= c * T;
    }
    return c;
  };
  Rad::run(g.r[0], [&](auto rad) {
    constexpr int RAD = decltype(rad)::value;
    const int T = g.T[0];
    for (int e = slot; e < C * T; e += nslots) {
      int i = e;
      const int c = component(i, T);
      const cpx<R>* q0 = gp + (int64_t)c * N + (size_t)i * inner;
      cpx<R>* o = sm + ((c * n) << lP) + pl;
      gen_butterfly<R, RAD, -1, true>(
          i, g, 0, tw, [&](int q) { return valid ? q0[(unsigned)(q * T) * inner] : mkc<R>((R)0, (R)0); },
          [&](int d, int q, cpx<R> v) { o[(d + q) << lP] = v; });
    }
  });
  sync();
  cpx<R>*cur = sm, *oth = sm + words;
  for (int s = 1; s < nst; ++s) {
    const bool with_green = C == 1 && s + 1 == nst;
    Rad::run(g.r[s], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = g.T[s];
      for (int e = slot; e < C * T; e += nslots) {
        int i = e;
        const int c = component(i, T);
        const int base = ((c * n) << lP) + pl, L = g.L[s];
        const cpx<R>* q0 = cur + base + (i << lP);
        gen_butterfly<R, RAD, -1, false>(
            i, g, s, tw, [&](int q) { return q0[(q * T) << lP]; },
            [&](int d, int q, cpx<R> v) {
              const int j = d + q * L;
              if (with_green) v = v * green(sk0[j] * sk0[j] + kt2);
              oth[base + (j << lP)] = v;
            });
      }
    });
    sync();
    cpx<R>* t = cur;
    cur = oth;
    oth = t;
  }
  if constexpr (C == 3) {
    // the dyadic split g (F - P_L F) + (i alpha_i / alpha) P_L F (solver.py:571-577, backend/__init__.py:606-649), with
    // the reference's DC rule and no longitudinal part along absent axes
    for (int j = slot; j < n; j += nslots) {
      const double k0 = sk0[j];
      const double kk2 = k0 * k0 + kt2;
      const cpx<R> gf = green(kk2);
      const R kv[3] = {(R)k0, (R)k1, (R)k2};
      cpx<R> F[3], PL[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) F[c] = cur[((size_t)(c * n + j) << lP) + pl];
      if (j == 0 && p == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) PL[c] = c < ndim ? F[c] : mkc<R>((R)0, (R)0);
      } else {
        cpx<R> proj = mkc<R>((R)0, (R)0);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (c < ndim) proj += kv[c] * F[c];
        proj = proj * ((R)1 / (R)kk2);
#pragma unroll
        for (int c = 0; c < 3; ++c) PL[c] = c < ndim ? kv[c] * proj : mkc<R>((R)0, (R)0);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) cur[((size_t)(c * n + j) << lP) + pl] = gf * (F[c] - PL[c]) + h * PL[c];
    }
    sync();
  }
  for (int s = 0; s + 1 < nst; ++s) {
    Rad::run(g.r[s], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = g.T[s];
      for (int e = slot; e < C * T; e += nslots) {
        int i = e;
        const int c = component(i, T);
        const int base = ((c * n) << lP) + pl, L = g.L[s];
        const cpx<R>* q0 = cur + base + (i << lP);
        gen_butterfly<R, RAD, +1, false>(
            i, g, s, tw, [&](int q) { return q0[(q * T) << lP]; },
            [&](int d, int q, cpx<R> v) { oth[base + ((d + q * L) << lP)] = v; });
      }
    });
    sync();
    cpx<R>* t = cur;
    cur = oth;
    oth = t;
  }
  if (!valid) return;
  Rad::run(g.r[nst - 1], [&](auto rad) {
    constexpr int RAD = decltype(rad)::value;
    const int T = g.T[nst - 1];
    for (int e = slot; e < C * T; e += nslots) {
      int i = e;
      const int c = component(i, T);
      const cpx<R>* q0 = cur + ((c * n + i) << lP) + pl;
      cpx<R>* d0 = gp + (int64_t)c * N + (size_t)i * inner;
      gen_butterfly<R, RAD, +1, false>(
          i, g, nst - 1, tw, [&](int q) { return q0[(q * T) << lP]; },
          [&](int, int q, cpx<R> v) { d0[(unsigned)(q * T) * inner] = v; });
    }
  });
}

// blockIdx.y: right-hand side
template <class R, int C>
__global__ void __launch_bounds__(256, GenBounds<R>::min_blocks) k_gen_green(const __grid_constant__ GenArgs<R> a) {
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  const int n = a.g.n, P = 1 << a.lP;
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + n);
  double* sk0 = reinterpret_cast<double*>(sm + 2 * (((size_t)C * n) << a.lP));
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    tw[t] = GenTw<R>::load(a.ax, t);
    sk0[t] = a.kvd[0][t];
  }
  const unsigned p = (blockIdx.x << a.lP) + (threadIdx.x & (P - 1));
  double k1, k2;
  gen_pencil_k(a, p, &k1, &k2);
  pdl_wait();
  pdl_trigger();
  const mmx_rhs_state* st = a.st + blockIdx.y;
  if (!st->active) return;
  green_tile<R, C, WideRadices>(a.g, a.lP, a.ndim, (unsigned)a.inner, a.N, p, a.T + (int64_t)blockIdx.y * C * a.N, k1, k2,
                   GenGreen<R>(st->alpha_re, st->alpha_im, a.inv_total_d),
                   gen_longitudinal<R>(st->alpha_re, st->alpha_im, a.inv_total_d), tw, sk0, sm, blockDim.x, BlockSync());
}

// ---------------------------------------------------------------------------------------------------------------
// Contiguous axis.  A tile holds P rows of each of the C components: row r of the tile is component r >> lP, row
// r & (P - 1) of the P rows.  KIND: GEN_ROWS (in -> out, C = 1), GEN_PRO, GEN_EPI, GEN_PRO3, GEN_EPI3.
// ---------------------------------------------------------------------------------------------------------------
template <class R> struct GenSkew { static constexpr int shift = sizeof(R) == 4 ? 4 : 3; };
template <class R> __host__ __device__ __forceinline__ int gen_pitch(int n) { return n + (n >> GenSkew<R>::shift); }
template <class R> __device__ __forceinline__ int gen_at(int j) { return j + (j >> GenSkew<R>::shift); }

template <class R, int KIND, int CHI, int DIR>
__global__ void __launch_bounds__(256, GenBounds<R>::min_blocks) k_gen_rows(const __grid_constant__ GenArgs<R> a) {
  constexpr bool kPro = KIND == GEN_PRO, kEpi = KIND == GEN_EPI, kPro3 = KIND == GEN_PRO3, kEpi3 = KIND == GEN_EPI3;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  const int n = a.g.n, lP = a.lP, P = 1 << lP, nst = a.g.nst;
  const int C = KIND == GEN_ROWS ? 1 : (kPro3 || kEpi3) ? 3 : a.C;
  const int rows = C << lP, pitch = gen_pitch<R>(n);
  const int words = rows * pitch;
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + n);
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = GenTw<R>::load(a.ax, t);
  const int b = blockIdx.y;
  const int64_t row0 = (int64_t)blockIdx.x << lP;
  const int left = a.outer - row0 < P ? (int)(a.outer - row0) : P;  // rows of this tile within the field
  const int64_t N = a.N;
  pdl_wait();
  pdl_trigger();
  ChiCoef<R> cc;
  const cpx<R>* Ecur = nullptr;
  cpx<R>* Eoth = nullptr;
  const mmx_rhs_state* st = a.st + b;
  if constexpr (KIND != GEN_ROWS) {
    if (!st->active) return;
    cc = chi_coef<R>(st);
    const int cur = st->cur;
    const int64_t fbase = (int64_t)b * C * N + row0 * n;
    Ecur = (cur ? a.E1 : a.E0) + fbase;
    Eoth = (cur ? a.E0 : a.E1) + fbase;
  }
  // first word of tile row r relative to the tile's first word of component 0
  auto row_off = [&](int r) { return (int64_t)(r >> lP) * N + (int64_t)(r & (P - 1)) * n; };
  const cpx<R>* gi = KIND == GEN_ROWS ? a.in + row0 * n : a.T + (int64_t)b * C * N + row0 * n;
  cpx<R>* go = KIND == GEN_ROWS ? a.out + row0 * n : a.T + (int64_t)b * C * N + row0 * n;
  const cpx<R>* __restrict__ X = a.chi + row0 * n;
  const cpx<R>* __restrict__ S = a.src + (int64_t)b * C * N + row0 * n;

  cpx<R>* cur = sm;
  int s0 = 0;  // the next stage
  if constexpr (kPro3) {
    // all components of a voxel in one thread, chi E + s' to shared memory
#pragma unroll 2
    for (int e = threadIdx.x; e < left * n; e += blockDim.x) {
      const int row = (int)gen_div((unsigned)e, a.g.mn), j = e - row * n;
      cpx<R> v[3], t[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = Ecur[c * N + e];
      apply_chi<R, 3, CHI>(X, N, e, cc, v, t);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (!source_is_zero(st, c)) t[c] += cc.s * S[c * N + e];
        sm[((c << lP) + row) * pitch + gen_at<R>(j)] = t[c];
      }
    }
    __syncthreads();
  } else {
    WideRadices::run(a.g.r[0], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = a.g.T[0];
      for (int e = threadIdx.x; e < rows * T; e += blockDim.x) {
        const int r = (int)gen_div((unsigned)e, a.g.mT[0]), i = e - r * T;
        if ((r & (P - 1)) >= left) continue;
        const int64_t off = row_off(r);
        cpx<R>* d = sm + r * pitch;
        if constexpr (kPro) {
          const cpx<R>*eS = Ecur + off, *sS = S + off, *xS = X + (int64_t)(r & (P - 1)) * n;
          const bool with_src = !source_is_zero(st, r >> lP);
          gen_butterfly<R, RAD, DIR, true>(
              i, a.g, 0, tw,
              [&](int q) {
                const int j = i + q * T;
                cpx<R> v = (cc.a * xS[j] + cc.b) * eS[j];
                if (with_src) v += cc.s * sS[j];
                return v;
              },
              [&](int o, int q, cpx<R> v) { d[gen_at<R>(o + q)] = v; });
        } else {
          const cpx<R>* tS = gi + off + i;
          gen_butterfly<R, RAD, DIR, true>(
              i, a.g, 0, tw, [&](int q) { return KIND == GEN_ROWS ? tS[q * T] * a.scale : tS[q * T]; },
              [&](int o, int q, cpx<R> v) { d[gen_at<R>(o + q)] = v; });
        }
      }
    });
    __syncthreads();
    s0 = 1;
  }
  const int s1 = kEpi3 ? nst : nst - 1;  // the stages between shared-memory buffers
  for (int s = s0; s < s1; ++s) {
    cpx<R>* dst = cur == sm ? sm + words : sm;
    WideRadices::run(a.g.r[s], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = a.g.T[s];
      for (int e = threadIdx.x; e < rows * T; e += blockDim.x) {
        const int r = (int)gen_div((unsigned)e, a.g.mT[s]), i = e - r * T;
        const cpx<R>* src = cur + r * pitch;
        cpx<R>* d = dst + r * pitch;
        const int L = a.g.L[s];
        gen_butterfly<R, RAD, DIR, false>(
            i, a.g, s, tw, [&](int q) { return src[gen_at<R>(i + q * T)]; },
            [&](int o, int q, cpx<R> v) { d[gen_at<R>(o + q * L)] = v; });
      }
    });
    __syncthreads();
    cur = dst;
  }
  double dd2 = 0.0, en2 = 0.0;
  if constexpr (kEpi3) {
    // V voxels per thread and round, all their loads ahead of their stores
    constexpr int V = sizeof(R) == 4 ? 2 : 1;
    const int count = left * n;
    for (int e0 = threadIdx.x; e0 < count; e0 += V * blockDim.x) {
      cpx<R> ev[V][3], d[V][3];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int e = e0 + v * blockDim.x;
        if (e < count) {
          const int row = (int)gen_div((unsigned)e, a.g.mn), j = e - row * n;
          cpx<R> t[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            ev[v][c] = Ecur[c * N + e];
            t[c] = cur[((c << lP) + row) * pitch + gen_at<R>(j)] - ev[v][c];
          }
          apply_chi<R, 3, CHI>(X, N, e, cc, t, d[v]);
        }
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int e = e0 + v * blockDim.x;
        if (e < count) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const cpx<R> en = ev[v][c] + d[v][c];
            Eoth[c * N + e] = en;
            dd2 += norm2d(d[v][c]);
            en2 += norm2d(en);
          }
        }
      }
    }
  } else {
    WideRadices::run(a.g.r[nst - 1], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int T = a.g.T[nst - 1];
      for (int e = threadIdx.x; e < rows * T; e += blockDim.x) {
        const int r = (int)gen_div((unsigned)e, a.g.mT[nst - 1]), i = e - r * T;
        if ((r & (P - 1)) >= left) continue;
        const int64_t off = row_off(r);
        const cpx<R>* src = cur + r * pitch;
        if constexpr (kEpi) {
          const cpx<R>*eS = Ecur + off, *xS = X + (int64_t)(r & (P - 1)) * n;
          cpx<R>* eO = Eoth + off;
          cpx<R> u[RAD];
          gen_dft<R, RAD, DIR, false>(i, T, a.g.mL[nst - 1], 1, tw, u, [&](int q) { return src[gen_at<R>(i + q * T)]; });
          // the outputs at i + q T: E and chi of CH of them are in flight at a time
          constexpr int CH = RAD <= 8 ? RAD : (RAD + 1) / 2;
#pragma unroll
          for (int q0 = 0; q0 < RAD; q0 += CH) {
            cpx<R> ev[CH], xv[CH];
#pragma unroll
            for (int q = 0; q < CH; ++q)
              if (q0 + q < RAD) {
                ev[q] = eS[i + (q0 + q) * T];
                xv[q] = xS[i + (q0 + q) * T];
              }
#pragma unroll
            for (int q = 0; q < CH; ++q)
              if (q0 + q < RAD) {
                const cpx<R> d = (cc.a * xv[q] + cc.b) * (u[q0 + q] - ev[q]);
                const cpx<R> en = ev[q] + d;
                eO[i + (q0 + q) * T] = en;
                dd2 += norm2d(d);
                en2 += norm2d(en);
              }
          }
        } else {
          cpx<R>* tO = go + off + i;
          gen_butterfly<R, RAD, DIR, false>(
              i, a.g, nst - 1, tw, [&](int q) { return src[gen_at<R>(i + q * T)]; },
              [&](int, int q, cpx<R> v) { tO[q * T] = v; });
        }
      }
    });
  }
  if constexpr (kEpi || kEpi3) finish_pass_norms(a, b, dd2, en2);
}
