// The passes of mmx_gen.cuh compiled for one length: two stages of radix R0 and R1, N = R0 R1.
//
// The any-length passes are bound by the instructions they issue (44-66 % of the issue slots, a third of the instructions
// for addresses and indices).  With the length, the tile and the block size known to the compiler the addresses become
// immediate offsets, the loops unroll and the rows need no skew against bank conflicts: after the first stage a row is
// kept in groups of R0 words at an odd pitch, which the second stage reads at that pitch.  The arithmetic is that of the
// any-length passes.  Each of the kernels is compiled for every 13-smooth length from 32 to 192 that has two stages; a
// grid that wants narrower tiles (few of them), another length or a general 3x3 chi takes the any-length pass.
#pragma once
#include "mmx_gen.cuh"

// R0 >= R1 (or <= when !DESC), the pair with the smallest sum
template <int N, bool DESC> struct LenPlan {
  static constexpr int small() {
    int best = 0;
    for (int a = 2; a * a <= N; ++a)
      if (N % a == 0 && a <= 16 && N / a <= 16) best = a;
    return best;
  }
  static constexpr int A = small(), B = A ? N / A : 0;
  static constexpr bool ok = A >= 2;
  static constexpr int R0 = DESC ? B : A, R1 = DESC ? A : B;
  static constexpr int T0 = R1, T1 = R0;  // butterflies per pencil of the stages
  static constexpr int G = R0 | 1;        // odd pitch of a group of R0 words
};
// registers per thread that a kernel is compiled for, by precision and largest radix
template <class R, int RAD> constexpr int kLenRegs = sizeof(R) == 4 ? (RAD <= 10 ? 64 : 80) : (RAD <= 8 ? 96 : RAD <= 10 ? 112 : 128);
constexpr int len_blocks(int threads, int regs) {
  const int b = 65536 / (threads * regs);
  return b > 32 ? 32 : b > 0 ? b : 1;
}

template <class R> struct LenArgs : IterArgs<R> {
  int C;
  const cpx<R>* in;
  cpx<R>* out;
  R scale;
};

// ---------------------------------------------------------------------------------------------------------------
template <class R, int N> struct LenStrided {
  using L = LenPlan<N, true>;
  static constexpr int P = gen_width(GEN_STRIDED, 1, sizeof(R) == 8, 0);
  static constexpr size_t SMEM = N * sizeof(gtw<R>) + (size_t)N * P * sizeof(cpx<R>);
  static constexpr int THREADS = gen_threads(2, L::R0, L::R1, 0, 0, N, 1, P, false, SMEM);
  static constexpr int BLOCKS = len_blocks(THREADS, kLenRegs<R, L::R0>);
};
template <class R, int DIR, int N>
__global__ void __launch_bounds__(LenStrided<R, N>::THREADS, (LenStrided<R, N>::BLOCKS))
    k_len_strided(const __grid_constant__ LenArgs<R> a) {
  using K = LenStrided<R, N>;
  using L = typename K::L;
  constexpr int P = K::P, SLOTS = K::THREADS / P;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + N);
  for (int t = threadIdx.x; t < N; t += K::THREADS) tw[t] = GenTw<R>::load(a.ax, t);
  const int pl = threadIdx.x % P, slot = threadIdx.x / P;
  const unsigned inner = (unsigned)a.inner;
  const unsigned p = blockIdx.x * P + pl;
  const bool valid = p < (unsigned)(a.outer * a.inner);
  const unsigned o = p / inner;
  const int64_t off = (int64_t)blockIdx.y * a.N + (int64_t)o * N * inner + (p - o * inner);
  pdl_wait();
  pdl_trigger();
  if (a.st && !a.st[blockIdx.y / a.C].active) return;
  const cpx<R>* gi = a.in + off;
  cpx<R>* go = a.out + off;
#pragma unroll 1
  for (int i = slot; i < L::T0; i += SLOTS) {
    cpx<R> u[L::R0];
    const cpx<R>* q0 = gi + (size_t)((unsigned)i * inner);
#pragma unroll
    for (int q = 0; q < L::R0; ++q) u[q] = valid ? q0[(unsigned)(q * L::T0) * inner] : mkc<R>((R)0, (R)0);
    gdft<R, L::R0, DIR>(u);
    cpx<R>* d = sm + i * (L::R0 * P) + pl;
#pragma unroll
    for (int q = 0; q < L::R0; ++q) d[q * P] = u[q];
  }
  __syncthreads();
  if (!valid) return;
#pragma unroll 1
  for (int i = slot; i < L::T1; i += SLOTS) {
    cpx<R> u[L::R1];
    const cpx<R>* s = sm + i * P + pl;
#pragma unroll
    for (int q = 0; q < L::R1; ++q) u[q] = s[q * (L::T1 * P)];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) u[q] = GenTw<R>::template mul<DIR>(u[q], tw[q * i]);
    gdft<R, L::R1, DIR>(u);
    cpx<R>* d = go + (size_t)((unsigned)i * inner);
#pragma unroll
    for (int q = 0; q < L::R1; ++q) d[(unsigned)(q * L::T1) * inner] = u[q];
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Axis 0.  The inverse transform runs the radices in reverse, so its first butterfly reads what the last forward one of
// the same thread wrote: for scalar fields the two and the Green factor between them stay in registers; for vector fields
// a pass over the tile applies the dyadic Green function to all three components of a sample.
// ---------------------------------------------------------------------------------------------------------------
template <class R, int C, int N> struct LenGreen {
  using L = LenPlan<N, true>;
  static constexpr int P = gen_width(GEN_GREEN, C, sizeof(R) == 8, 0);
  static constexpr size_t SMEM =
      N * sizeof(gtw<R>) + (C == 3 ? 2 : 1) * (size_t)C * N * P * sizeof(cpx<R>) + N * sizeof(double);
  static constexpr int THREADS = gen_threads(2, L::R0, L::R1, 0, 0, N, C, P, false, SMEM);
  static constexpr int BLOCKS = len_blocks(THREADS, kLenRegs<R, L::R0>);
};
template <class R, int C, int N>
__global__ void __launch_bounds__(LenGreen<R, C, N>::THREADS, (LenGreen<R, C, N>::BLOCKS))
    k_len_green(const __grid_constant__ LenArgs<R> a) {
  using K = LenGreen<R, C, N>;
  using L = typename K::L;
  constexpr int P = K::P, SLOTS = K::THREADS / P;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + N);
  cpx<R>* sf = sm + (C == 3 ? C * N * P : 0);  // the spectrum of a vector tile
  double* sk0 = reinterpret_cast<double*>(sf + C * N * P);
  for (int t = threadIdx.x; t < N; t += K::THREADS) {
    tw[t] = GenTw<R>::load(a.ax, t);
    sk0[t] = a.kvd[0][t];
  }
  const int pl = threadIdx.x % P, slot = threadIdx.x / P;
  const unsigned inner = (unsigned)a.inner;
  const unsigned p = blockIdx.x * P + pl;
  const bool valid = p < inner;
  double k1, k2;
  gen_pencil_k(a, p, &k1, &k2);
  pdl_wait();
  pdl_trigger();
  const mmx_rhs_state* st = a.st + blockIdx.y;
  if (!st->active) return;
  cpx<R>* gp = a.T + (int64_t)blockIdx.y * C * a.N + p;
  const double kt2 = k1 * k1 + k2 * k2, ar = st->alpha_re, ai = st->alpha_im;
  const GenGreen<R> green(ar, ai, a.inv_total_d);
#pragma unroll 1
  for (int e = slot; e < C * L::T0; e += SLOTS) {
    const int c = e / L::T0, i = e - c * L::T0;
    cpx<R> u[L::R0];
    const cpx<R>* q0 = gp + c * a.N + (size_t)((unsigned)i * inner);
#pragma unroll
    for (int q = 0; q < L::R0; ++q) u[q] = valid ? q0[(unsigned)(q * L::T0) * inner] : mkc<R>((R)0, (R)0);
    gdft<R, L::R0, -1>(u);
    cpx<R>* d = sm + (c * N + i * L::R0) * P + pl;
#pragma unroll
    for (int q = 0; q < L::R0; ++q) d[q * P] = u[q];
  }
  __syncthreads();
  if constexpr (C == 1) {
    // in place: butterfly i reads and writes the samples i + q T1 of its pencil, in groups of T1 = R0 words
#pragma unroll 1
    for (int i = slot; i < L::T1; i += SLOTS) {
      cpx<R> u[L::R1];
      cpx<R>* s = sm + i * P + pl;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) u[q] = s[q * (L::T1 * P)];
#pragma unroll
      for (int q = 1; q < L::R1; ++q) u[q] = GenTw<R>::template mul<-1>(u[q], tw[q * i]);
      gdft<R, L::R1, -1>(u);
#pragma unroll
      for (int q = 0; q < L::R1; ++q) {
        const double k0 = sk0[i + q * L::T1];
        u[q] = u[q] * green(k0 * k0 + kt2);
      }
      gdft<R, L::R1, +1>(u);
      // output q of the first inverse stage (span 1) belongs at i R1 + q; kept where its inputs were
#pragma unroll
      for (int q = 0; q < L::R1; ++q) s[q * (L::T1 * P)] = u[q];
    }
    __syncthreads();
    if (!valid) return;
    // last inverse stage, radix R0, span R1: butterfly k reads the samples k + q R1, i.e. output k of butterfly q above
#pragma unroll 1
    for (int k = slot; k < L::R1; k += SLOTS) {
      cpx<R> u[L::R0];
      const cpx<R>* s = sm + k * (L::T1 * P) + pl;
#pragma unroll
      for (int q = 0; q < L::R0; ++q) u[q] = s[q * P];
#pragma unroll
      for (int q = 1; q < L::R0; ++q) u[q] = GenTw<R>::template mul<+1>(u[q], tw[q * k]);
      gdft<R, L::R0, +1>(u);
      cpx<R>* d = gp + (size_t)((unsigned)k * inner);
#pragma unroll
      for (int q = 0; q < L::R0; ++q) d[(unsigned)(q * L::R1) * inner] = u[q];
    }
  } else {
#pragma unroll 1
    for (int e = slot; e < C * L::T1; e += SLOTS) {
      const int c = e / L::T1, i = e - c * L::T1;
      cpx<R> u[L::R1];
      const cpx<R>* s = sm + (c * N + i) * P + pl;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) u[q] = s[q * (L::T1 * P)];
#pragma unroll
      for (int q = 1; q < L::R1; ++q) u[q] = GenTw<R>::template mul<-1>(u[q], tw[q * i]);
      gdft<R, L::R1, -1>(u);
      cpx<R>* d = sf + (c * N + i) * P + pl;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) d[q * (L::T1 * P)] = u[q];
    }
    __syncthreads();
    const cpx<R> h = gen_longitudinal<R>(ar, ai, a.inv_total_d);
#pragma unroll 1
    for (int j = slot; j < N; j += SLOTS) {
      const double k0 = sk0[j];
      const double kk2 = k0 * k0 + kt2;
      const cpx<R> gf = green(kk2);
      const R kv[3] = {(R)k0, (R)k1, (R)k2};
      cpx<R> F[3], PL[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) F[c] = sf[(c * N + j) * P + pl];
      if (j == 0 && p == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) PL[c] = c < a.ndim ? F[c] : mkc<R>((R)0, (R)0);
      } else {
        cpx<R> proj = kv[0] * F[0] + kv[1] * F[1] + kv[2] * F[2];  // k is 0 along absent axes
        proj = proj * ((R)1 / (R)kk2);
#pragma unroll
        for (int c = 0; c < 3; ++c) PL[c] = kv[c] * proj;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) sf[(c * N + j) * P + pl] = gf * (F[c] - PL[c]) + h * PL[c];
    }
    __syncthreads();
    // inverse, radix R1 (span 1), then R0 (span R1)
#pragma unroll 1
    for (int e = slot; e < C * L::T1; e += SLOTS) {
      const int c = e / L::T1, i = e - c * L::T1;
      cpx<R> u[L::R1];
      const cpx<R>* s = sf + (c * N + i) * P + pl;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) u[q] = s[q * (L::T1 * P)];
      gdft<R, L::R1, +1>(u);
      cpx<R>* d = sm + (c * N + i * L::R1) * P + pl;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) d[q * P] = u[q];
    }
    __syncthreads();
    if (!valid) return;
#pragma unroll 1
    for (int e = slot; e < C * L::R1; e += SLOTS) {
      const int c = e / L::R1, k = e - c * L::R1;
      cpx<R> u[L::R0];
      const cpx<R>* s = sm + (c * N + k) * P + pl;
#pragma unroll
      for (int q = 0; q < L::R0; ++q) u[q] = s[q * (L::R1 * P)];
#pragma unroll
      for (int q = 1; q < L::R0; ++q) u[q] = GenTw<R>::template mul<+1>(u[q], tw[q * k]);
      gdft<R, L::R0, +1>(u);
      cpx<R>* d = gp + c * a.N + (size_t)((unsigned)k * inner);
#pragma unroll
      for (int q = 0; q < L::R0; ++q) d[(unsigned)(q * L::R1) * inner] = u[q];
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Contiguous axis (KIND as in k_gen_rows; 3x3: MMX_CHI_SYM6).
// ---------------------------------------------------------------------------------------------------------------
template <class R, int KIND, int C, int N> struct LenRows {
  static constexpr bool k3 = KIND == GEN_PRO3 || KIND == GEN_EPI3;
  using L = LenPlan<N, KIND == GEN_EPI>;
  static constexpr int P = gen_width((GenKind)KIND, C, sizeof(R) == 8, L::T0 > L::T1 ? L::T0 : L::T1);
  static constexpr int ROWS = C * P;
  static constexpr int W0 = L::T0 * L::G;  // words of a row after the first stage
  static constexpr size_t SMEM = N * sizeof(gtw<R>) + (size_t)ROWS * (W0 + (k3 ? N : 0)) * sizeof(cpx<R>);
  static constexpr int THREADS = gen_threads(2, L::R0, L::R1, 0, 0, N, C, P, true, SMEM);
  // the epilogue holds E and chi of half a butterfly beside it
  static constexpr int REGS = kLenRegs<R, (L::R0 > L::R1 ? L::R0 : L::R1)>;
  static constexpr int BLOCKS = len_blocks(THREADS, KIND == GEN_EPI && REGS < 80 ? 80 : REGS);
};
template <class R, int KIND, int C, int DIR, int N>
__global__ void __launch_bounds__(LenRows<R, KIND, C, N>::THREADS, (LenRows<R, KIND, C, N>::BLOCKS))
    k_len_rows(const __grid_constant__ LenArgs<R> a) {
  using K = LenRows<R, KIND, C, N>;
  using L = typename K::L;
  constexpr bool kPro = KIND == GEN_PRO, kEpi = KIND == GEN_EPI, kPro3 = KIND == GEN_PRO3, kEpi3 = KIND == GEN_EPI3;
  constexpr int CHI = K::k3 ? MMX_CHI_SYM6 : MMX_CHI_SCALAR;
  constexpr int P = K::P, THREADS = K::THREADS, ROWS = K::ROWS;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(tw + N);  // [row][T0 groups of R0 words at pitch G]
  cpx<R>* sn = sm + ROWS * K::W0;                  // 3x3: [row][N]
  const int tid = threadIdx.x;
  // the factors of butterfly i at [q - 1][i]: neighbouring threads read neighbouring words
  for (int t = tid; t < (L::R1 - 1) * L::T1; t += THREADS) {
    const int q = t / L::T1;
    tw[t] = GenTw<R>::load(a.ax, (q + 1) * (t - q * L::T1));
  }
  const int b = blockIdx.y;
  const int64_t row0 = (int64_t)blockIdx.x * P;
  const int left = a.outer - row0 < P ? (int)(a.outer - row0) : P;
  const int64_t NV = a.N;
  pdl_wait();
  pdl_trigger();
  const mmx_rhs_state* st = a.st + b;
  ChiCoef<R> cc;
  const cpx<R>* E = nullptr;
  cpx<R>* En = nullptr;
  const int64_t base = row0 * N, field = KIND == GEN_ROWS ? base : (int64_t)b * C * NV + base;
  if constexpr (KIND != GEN_ROWS) {
    if (!st->active) return;
    cc = chi_coef<R>(st);
    const int cur = st->cur;
    E = (cur ? a.E1 : a.E0) + field;
    En = (cur ? a.E0 : a.E1) + field;
  }
  const cpx<R>* gi = (KIND == GEN_ROWS ? a.in : a.T) + field;
  cpx<R>* go = (KIND == GEN_ROWS ? a.out : a.T) + field;
  const cpx<R>* X = a.chi + base;
  const cpx<R>* S = a.src + field;

  if constexpr (kPro3) {
#pragma unroll 2
    for (int e = tid; e < left * N; e += THREADS) {
      cpx<R> v[3], t[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = E[c * NV + e];
      apply_chi<R, 3, CHI>(X, NV, e, cc, v, t);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (!source_is_zero(st, c)) t[c] += cc.s * S[c * NV + e];
        sn[c * (P * N) + e] = t[c];
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int e = tid; e < ROWS * L::T0; e += THREADS) {
    const int r = e / L::T0, i = e - r * L::T0, row = r % P, c = r / P;
    if (row >= left) continue;
    const int64_t off = c * NV + row * N + i;
    cpx<R> u[L::R0];
    if constexpr (kPro3) {
      const cpx<R>* s = sn + r * N + i;
#pragma unroll
      for (int q = 0; q < L::R0; ++q) u[q] = s[q * L::T0];
    } else if constexpr (kPro) {
      const cpx<R>*eS = E + off, *xS = X + row * N + i, *sS = S + off;
      const bool with_src = !source_is_zero(st, c);
#pragma unroll
      for (int q = 0; q < L::R0; ++q) {
        u[q] = (cc.a * xS[q * L::T0] + cc.b) * eS[q * L::T0];
        if (with_src) u[q] += cc.s * sS[q * L::T0];
      }
    } else {
      const cpx<R>* s = gi + off;
#pragma unroll
      for (int q = 0; q < L::R0; ++q) u[q] = KIND == GEN_ROWS ? s[q * L::T0] * a.scale : s[q * L::T0];
    }
    gdft<R, L::R0, DIR>(u);
    cpx<R>* d = sm + r * K::W0 + i * L::G;
#pragma unroll
    for (int q = 0; q < L::R0; ++q) d[q] = u[q];
  }
  __syncthreads();
  double dd2 = 0.0, en2 = 0.0;
#pragma unroll 1
  for (int e = tid; e < ROWS * L::T1; e += THREADS) {
    const int r = e / L::T1, i = e - r * L::T1, row = r % P, c = r / P;
    if (row >= left) continue;
    const int64_t off = c * NV + row * N + i;
    cpx<R> u[L::R1];
    const cpx<R>* s = sm + r * K::W0 + i;
    // E and chi of CH samples are in flight at a time, the first ones while the butterfly is computed
    constexpr int CH = !kEpi ? 1 : L::R1 <= 6 ? L::R1 : (L::R1 + 1) / 2;
    cpx<R> ev[CH], xv[CH];
    const cpx<R>*eS = E + off, *xS = X + row * N + i;
    auto fetch = [&](int q0) {
#pragma unroll
      for (int q = 0; q < CH; ++q)
        if (q0 + q < L::R1) {
          ev[q] = eS[(q0 + q) * L::T1];
          xv[q] = xS[(q0 + q) * L::T1];
        }
    };
    if constexpr (kEpi) fetch(0);
#pragma unroll
    for (int q = 0; q < L::R1; ++q) u[q] = s[q * L::G];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) u[q] = GenTw<R>::template mul<DIR>(u[q], tw[(q - 1) * L::T1 + i]);
    gdft<R, L::R1, DIR>(u);
    if constexpr (kEpi) {
      cpx<R>* eO = En + off;
#pragma unroll
      for (int q0 = 0; q0 < L::R1; q0 += CH) {
        if (q0 > 0) fetch(q0);
#pragma unroll
        for (int q = 0; q < CH; ++q)
          if (q0 + q < L::R1) {
            const cpx<R> d = (cc.a * xv[q] + cc.b) * (u[q0 + q] - ev[q]);
            const cpx<R> en = ev[q] + d;
            eO[(q0 + q) * L::T1] = en;
            dd2 += norm2d(d);
            en2 += norm2d(en);
          }
      }
    } else if constexpr (kEpi3) {
      cpx<R>* d = sn + r * N + i;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) d[q * L::T1] = u[q];
    } else {
      cpx<R>* d = go + off;
#pragma unroll
      for (int q = 0; q < L::R1; ++q) d[q * L::T1] = u[q];
    }
  }
  if constexpr (kEpi3) {
    __syncthreads();
    constexpr int V = sizeof(R) == 4 ? 2 : 1;  // voxels per thread and round, all their loads ahead of their stores
    const int count = left * N;
#pragma unroll 1
    for (int e0 = tid; e0 < count; e0 += V * THREADS) {
      cpx<R> ev[V][3], d[V][3];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int e = e0 + v * THREADS;
        if (e < count) {
          cpx<R> t[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            ev[v][c] = E[c * NV + e];
            t[c] = sn[c * (P * N) + e] - ev[v][c];
          }
          apply_chi<R, 3, CHI>(X, NV, e, cc, t, d[v]);
        }
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int e = e0 + v * THREADS;
        if (e < count) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const cpx<R> en = ev[v][c] + d[v][c];
            En[c * NV + e] = en;
            dd2 += norm2d(d[v][c]);
            en2 += norm2d(en);
          }
        }
      }
    }
  }
  if constexpr (kEpi || kEpi3) finish_pass_norms(a, b, dd2, en2);
}
