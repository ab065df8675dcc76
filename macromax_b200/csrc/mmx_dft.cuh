// Small DFTs in registers for the passes of any length (mmx_gen.cuh): gdft<R, RAD, DIR>(u) replaces u[0..RAD-1] by its
// DFT of length RAD (DIR = -1 forward, +1 inverse, unscaled), RAD = 2 .. 16.
//
//   2, 4               the butterflies of mmx_complex.cuh; 8 and 16 from them and the eighth and sixteenth roots of unity
//   3, 5               as in mmx_complex.cuh
//   7, 11, 13          odd primes: with t_q = x_q + x_{r-q} and d_q = x_q - x_{r-q}, outputs k and r - k are a_k +- i b_k
//                      with a_k = x_0 + sum_q cos(2 pi q k / r) t_q, b_k = sum_q sin(2 pi q k / r) d_q: two real products
//                      per complex term of half the sum instead of a complex product per term of the whole sum
//   6, 10, 12, 14, 15  coprime factors A B: Good's prime-factor mapping, input (B n1 + A n2) mod A B, output the k with
//                      k = k1 mod A, k = k2 mod B: no twiddle factors
//   9                  3 x 3 Cooley-Tukey with the ninth roots of unity
// All coefficients are compile-time constants, so no stage before the first barrier needs the twiddle table.  In complex64
// a product with a coefficient uses it as the sum of two floats (one more fused multiply-add): a coefficient rounded to
// float scales the same spectral lines by the same wrong factor in every iteration, and the converged field shows that
// error many times over.
#pragma once
#include "mmx_complex.cuh"

// x c with c in FP64 (float: as hi + lo), and acc + x c
__host__ __device__ __forceinline__ double mul_const(double x, double c) { return x * c; }
__host__ __device__ __forceinline__ float mul_const(float x, double c) {
  const float hi = (float)c, lo = (float)(c - (double)hi);
  return fmaf(x, hi, x * lo);
}
__host__ __device__ __forceinline__ double add_const(double acc, double x, double c) { return fma(x, c, acc); }
__host__ __device__ __forceinline__ float add_const(float acc, float x, double c) {
  const float hi = (float)c, lo = (float)(c - (double)hi);
  return fmaf(x, hi, fmaf(x, lo, acc));
}

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
      const double c = root_cos<RAD>((q * k) % RAD), s = root_sin<RAD>((q * k) % RAD);
      a.x = add_const(a.x, t[q - 1].x, c);
      a.y = add_const(a.y, t[q - 1].y, c);
      b.x = add_const(b.x, d[q - 1].x, s);
      b.y = add_const(b.y, d[q - 1].y, s);
    }
    const cpx<R> ib = mul_i(b, DIR);
    u[k] = a + ib;
    u[RAD - k] = a - ib;
  }
}

// a (c + i s)
template <class R> __host__ __device__ __forceinline__ cpx<R> rotate(cpx<R> a, double c, double s) {
  return mkc<R>(add_const(mul_const(a.x, c), a.y, -s), add_const(mul_const(a.y, c), a.x, s));
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft3(cpx<R>* u) {
  const cpx<R> t = u[1] + u[2], d = mul_i(u[1] - u[2], DIR);
  const cpx<R> m = u[0] - (R)0.5 * t, s = mkc<R>(mul_const(d.x, MMX_SQRT3_2), mul_const(d.y, MMX_SQRT3_2));
  u[0] = u[0] + t;
  u[1] = m + s;
  u[2] = m - s;
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft5(cpx<R>* u) {
  const cpx<R> a = u[0], t1 = u[1] + u[4], t2 = u[2] + u[3], t3 = mul_i(u[1] - u[4], DIR), t4 = mul_i(u[2] - u[3], DIR);
  auto comb = [](R a0, R x, R y, double c, double d) { return add_const(add_const(a0, x, c), y, d); };
  const cpx<R> m1 = mkc<R>(comb(a.x, t1.x, t2.x, MMX_C5_1, MMX_C5_2), comb(a.y, t1.y, t2.y, MMX_C5_1, MMX_C5_2));
  const cpx<R> m2 = mkc<R>(comb(a.x, t1.x, t2.x, MMX_C5_2, MMX_C5_1), comb(a.y, t1.y, t2.y, MMX_C5_2, MMX_C5_1));
  const cpx<R> s1 = mkc<R>(comb((R)0, t3.x, t4.x, MMX_S5_1, MMX_S5_2), comb((R)0, t3.y, t4.y, MMX_S5_1, MMX_S5_2));
  const cpx<R> s2 = mkc<R>(comb((R)0, t3.x, t4.x, MMX_S5_2, -MMX_S5_1), comb((R)0, t3.y, t4.y, MMX_S5_2, -MMX_S5_1));
  u[0] = a + t1 + t2;
  u[1] = m1 + s1;
  u[4] = m1 - s1;
  u[2] = m2 + s2;
  u[3] = m2 - s2;
}

// a exp(DIR 2 pi i m / 8), m = 1 or 3
template <class R, int DIR> __host__ __device__ __forceinline__ cpx<R> eighth(cpx<R> a, int m) {
  const cpx<R> v = m == 1 ? mkc<R>(a.x - DIR * a.y, a.y + DIR * a.x) : mkc<R>(-a.x - DIR * a.y, DIR * a.x - a.y);
  return mkc<R>(mul_const(v.x, MMX_SQRT1_2), mul_const(v.y, MMX_SQRT1_2));
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft8(cpx<R>* u) {
  cpx<R> e[4] = {u[0], u[2], u[4], u[6]}, o[4] = {u[1], u[3], u[5], u[7]};
  bfly4<R, DIR>(e);
  bfly4<R, DIR>(o);
  o[1] = eighth<R, DIR>(o[1], 1);
  o[2] = mul_i(o[2], DIR);
  o[3] = eighth<R, DIR>(o[3], 3);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u[k] = e[k] + o[k];
    u[k + 4] = e[k] - o[k];
  }
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft16(cpx<R>* u) {
  // x[n1 + 4 n2]: DFT4 over n2 for each n1, w16^(n1 k2), DFT4 over n1; X[k2 + 4 k1]
  auto tw = [](cpx<R> a, int m) {
    switch (m) {
      case 0: return a;
      case 1: return rotate<R>(a, MMX_C16_1, DIR * MMX_S16_1);
      case 2: return eighth<R, DIR>(a, 1);
      case 3: return rotate<R>(a, MMX_S16_1, DIR * MMX_C16_1);
      case 4: return mul_i(a, DIR);
      case 6: return eighth<R, DIR>(a, 3);
      default: return rotate<R>(a, -MMX_C16_1, -DIR * MMX_S16_1);  // 9
    }
  };
  cpx<R> y[4][4];
#pragma unroll
  for (int n1 = 0; n1 < 4; ++n1) {
    cpx<R> v[4] = {u[n1], u[n1 + 4], u[n1 + 8], u[n1 + 12]};
    bfly4<R, DIR>(v);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) y[n1][k2] = tw(v[k2], n1 * k2);
  }
#pragma unroll
  for (int k2 = 0; k2 < 4; ++k2) {
    cpx<R> v[4] = {y[0][k2], y[1][k2], y[2][k2], y[3][k2]};
    bfly4<R, DIR>(v);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) u[k2 + 4 * k1] = v[k1];
  }
}

template <class R, int DIR> __host__ __device__ __forceinline__ void gdft9(cpx<R>* u) {
  // x[n1 + 3 n2]: DFT3 over n2 for each n1, w9^(n1 k2), DFT3 over n1; X[k2 + 3 k1]
  auto tw = [](cpx<R> a, int m) { return rotate<R>(a, root_cos<9>(m), DIR * root_sin<9>(m)); };
  cpx<R> y[9];
#pragma unroll
  for (int n1 = 0; n1 < 3; ++n1) {
    cpx<R> v[3] = {u[n1], u[n1 + 3], u[n1 + 6]};
    gdft3<R, DIR>(v);
    y[n1 * 3] = v[0];
    y[n1 * 3 + 1] = n1 ? tw(v[1], n1) : v[1];
    y[n1 * 3 + 2] = n1 ? tw(v[2], 2 * n1) : v[2];
  }
#pragma unroll
  for (int k2 = 0; k2 < 3; ++k2) {
    cpx<R> v[3] = {y[k2], y[3 + k2], y[6 + k2]};
    gdft3<R, DIR>(v);
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
  else if constexpr (RAD == 3) gdft3<R, DIR>(u);
  else if constexpr (RAD == 4) bfly4<R, DIR>(u);
  else if constexpr (RAD == 5) gdft5<R, DIR>(u);
  else if constexpr (RAD == 6) gdft_coprime<R, 2, 3, DIR>(u);
  else if constexpr (RAD == 8) gdft8<R, DIR>(u);
  else if constexpr (RAD == 9) gdft9<R, DIR>(u);
  else if constexpr (RAD == 10) gdft_coprime<R, 2, 5, DIR>(u);
  else if constexpr (RAD == 12) gdft_coprime<R, 4, 3, DIR>(u);
  else if constexpr (RAD == 14) gdft_coprime<R, 2, 7, DIR>(u);
  else if constexpr (RAD == 15) gdft_coprime<R, 3, 5, DIR>(u);
  else if constexpr (RAD == 16) gdft16<R, DIR>(u);
  else gdft_prime<R, RAD, DIR>(u);
}
