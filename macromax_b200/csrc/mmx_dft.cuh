// Small DFTs in registers for the passes of any length (mmx_gen.cuh): gdft<R, RAD, DIR>(u) replaces u[0..RAD-1] by its
// DFT of length RAD (DIR = -1 forward, +1 inverse, unscaled), RAD = 2 .. 16.
//
//   2, 3, 4, 5, 8, 16  the butterflies of mmx_complex.cuh
//   7, 11, 13          odd primes: with t_q = x_q + x_{r-q} and d_q = x_q - x_{r-q}, outputs k and r - k are a_k +- i b_k
//                      with a_k = x_0 + sum_q cos(2 pi q k / r) t_q, b_k = sum_q sin(2 pi q k / r) d_q: two real products
//                      per complex term of half the sum instead of a complex product per term of the whole sum
//   6, 10, 12, 14, 15  coprime factors A B: Good's prime-factor mapping, input (B n1 + A n2) mod A B, output the k with
//                      k = k1 mod A, k = k2 mod B: no twiddle factors
//   9                  3 x 3 Cooley-Tukey with the ninth roots of unity
// All coefficients are compile-time constants, so no stage before the first barrier needs the twiddle table.
#pragma once
#include "mmx_complex.cuh"

// cos and sin of 2 pi m / RAD, 0 <= m < RAD, RAD in {7, 9, 11, 13}
template <int RAD> __host__ __device__ __forceinline__ constexpr double root_cos(int m) {
  if (2 * m > RAD) m = RAD - m;
  if (RAD == 7)
    return m == 0 ? 1.0 : m == 1 ? 0.62348980185873353053 : m == 2 ? -0.22252093395631440429 : -0.90096886790241912624;
  if (RAD == 9)
    return m == 0 ? 1.0 : m == 1 ? 0.76604444311897803520 : m == 2 ? 0.17364817766693034885 : m == 3 ? -0.5
                                                                                      : -0.93969262078590838405;
  if (RAD == 11)
    return m == 0   ? 1.0
           : m == 1 ? 0.84125353283118116886
           : m == 2 ? 0.41541501300188642553
           : m == 3 ? -0.14231483827328514044
           : m == 4 ? -0.65486073394528506406
                    : -0.95949297361449738989;
  return m == 0   ? 1.0
         : m == 1 ? 0.88545602565320989590
         : m == 2 ? 0.56806474673115580251
         : m == 3 ? 0.12053668025532305335
         : m == 4 ? -0.35460488704253562597
         : m == 5 ? -0.74851074817110109863
                  : -0.97094181742605202716;
}
template <int RAD> __host__ __device__ __forceinline__ constexpr double root_sin(int m) {
  const double s = 2 * m > RAD ? -1.0 : 1.0;
  if (2 * m > RAD) m = RAD - m;
  double v = 0.0;
  if (RAD == 7)
    v = m == 0 ? 0.0 : m == 1 ? 0.78183148246802980871 : m == 2 ? 0.97492791218182360702 : 0.43388373911755812048;
  else if (RAD == 9)
    v = m == 0 ? 0.0 : m == 1 ? 0.64278760968653932632 : m == 2 ? 0.98480775301220805937 : m == 3 ? MMX_SQRT3_2
                                                                                     : 0.34202014332566873304;
  else if (RAD == 11)
    v = m == 0   ? 0.0
        : m == 1 ? 0.54064081745559758211
        : m == 2 ? 0.90963199535451837141
        : m == 3 ? 0.98982144188093273238
        : m == 4 ? 0.75574957435425828377
                 : 0.28173255684142969771;
  else
    v = m == 0   ? 0.0
        : m == 1 ? 0.46472317204376854566
        : m == 2 ? 0.82298386589365639458
        : m == 3 ? 0.99270887409805399280
        : m == 4 ? 0.93501624268541482344
        : m == 5 ? 0.66312265824079520238
                 : 0.23931566428755776715;
  return s * v;
}

template <class R, int RAD, int DIR> __host__ __device__ __forceinline__ void gdft_prime(cpx<R>* u) {
  constexpr int H = (RAD - 1) / 2;
  cpx<R> t[H], d[H];
  const cpx<R> x0 = u[0];
  cpx<R> sum = x0;
#pragma unroll
  for (int q = 1; q <= H; ++q) {
    t[q - 1] = u[q] + u[RAD - q];
    d[q - 1] = u[q] - u[RAD - q];
    sum += t[q - 1];
  }
  u[0] = sum;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    cpx<R> a = x0, b = mkc<R>((R)0, (R)0);
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      const R c = (R)root_cos<RAD>((q * k) % RAD), s = (R)root_sin<RAD>((q * k) % RAD);
      a.x += c * t[q - 1].x;
      a.y += c * t[q - 1].y;
      b.x += s * d[q - 1].x;
      b.y += s * d[q - 1].y;
    }
    const cpx<R> ib = mul_i(b, DIR);
    u[k] = a + ib;
    u[RAD - k] = a - ib;
  }
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft9(cpx<R>* u) {
  // x[n1 + 3 n2]: DFT3 over n2 for each n1, w9^(n1 k2), DFT3 over n1; X[k2 + 3 k1]
  auto tw = [](cpx<R> a, int m) {
    const R c = (R)root_cos<9>(m), s = (R)(DIR * root_sin<9>(m));
    return mkc<R>(a.x * c - a.y * s, a.y * c + a.x * s);
  };
  cpx<R> y[9];
#pragma unroll
  for (int n1 = 0; n1 < 3; ++n1) {
    cpx<R> v[3] = {u[n1], u[n1 + 3], u[n1 + 6]};
    bfly3<R, DIR>(v);
    y[n1 * 3] = v[0];
    y[n1 * 3 + 1] = n1 ? tw(v[1], n1) : v[1];
    y[n1 * 3 + 2] = n1 ? tw(v[2], 2 * n1) : v[2];
  }
#pragma unroll
  for (int k2 = 0; k2 < 3; ++k2) {
    cpx<R> v[3] = {y[k2], y[3 + k2], y[6 + k2]};
    bfly3<R, DIR>(v);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) u[k2 + 3 * k1] = v[k1];
  }
}

template <class R, int RAD, int DIR> __host__ __device__ __forceinline__ void gdft(cpx<R>* u);

// coprime A and B
template <class R, int A, int B, int DIR> __host__ __device__ __forceinline__ void gdft_coprime(cpx<R>* u) {
  constexpr int N = A * B;
  cpx<R> y[N];  // y[k1 + A n2]
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    cpx<R> v[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) v[n1] = u[(B * n1 + A * n2) % N];
    gdft<R, A, DIR>(v);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) y[k1 + A * n2] = v[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    cpx<R> v[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) v[n2] = y[k1 + A * n2];
    gdft<R, B, DIR>(v);
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (k % A == k1) u[k] = v[k % B];
  }
}

template <class R, int RAD, int DIR> __host__ __device__ __forceinline__ void gdft(cpx<R>* u) {
  static_assert(RAD >= 2 && RAD <= 16, "radices of 2 to 16");
  if constexpr (RAD == 2) bfly2<R, DIR>(u);
  else if constexpr (RAD == 3) bfly3<R, DIR>(u);
  else if constexpr (RAD == 4) bfly4<R, DIR>(u);
  else if constexpr (RAD == 5) bfly5<R, DIR>(u);
  else if constexpr (RAD == 6) gdft_coprime<R, 2, 3, DIR>(u);
  else if constexpr (RAD == 8) bfly8<R, DIR>(u);
  else if constexpr (RAD == 9) gdft9<R, DIR>(u);
  else if constexpr (RAD == 10) gdft_coprime<R, 2, 5, DIR>(u);
  else if constexpr (RAD == 12) gdft_coprime<R, 4, 3, DIR>(u);
  else if constexpr (RAD == 14) gdft_coprime<R, 2, 7, DIR>(u);
  else if constexpr (RAD == 15) gdft_coprime<R, 3, 5, DIR>(u);
  else if constexpr (RAD == 16) bfly16<R, DIR>(u);
  else gdft_prime<R, RAD, DIR>(u);
}
