// Device code shared by every pass of the split-Richardson iteration: pass arguments, programmatic dependent launch,
// the per-RHS coefficients, chi products, block reductions and the accept / reject decision.
#pragma once
#include "../../include/macromax_b200.h"
#include "mmx_fft.cuh"

enum : int {
  OP_PRO = 1,      // prologue: T = chi(alpha) E + s'(alpha)
  OP_FWD = 2,      // forward FFT along the pass axis
  OP_G = 4,        // Green multiply (axis-0 pass only)
  OP_INV = 8,      // inverse FFT along the pass axis
  OP_EPI = 16,     // iteration epilogue: d = chi (T - E); E' = E + d; partial norms
  OP_GINV = 32,    // with OP_G: apply G^{-1} instead of G
  OP_XLOAD = 64,   // first pass of the defect: load x instead of T
  OP_DEFECT = 128  // defect epilogue: s_out = s' + chi x - T, stored as complex64
};

template <class R> struct IterArgs {
  FFTAxis ax;
  int64_t outer, inner;  // pencil geometry of the pass axis (per component, per RHS)
  int P, sP;             // pencils per tile, shared-memory row pitch
  int64_t N;             // voxels per component
  int ndim;
  int dims[3];
  const R* kv[3];        // k-vector tables per axis
  const double* kvd[3];  // the same in FP64
  cpx<R>* T;             // work [B][C][N]
  cpx<R>* E0;            // field buffers [B][C][N] (E0 is x for the defect)
  cpx<R>* E1;
  const cpx<R>* chi;     // [m][N]
  const cpx<R>* src;     // [B][C][N]
  const mmx_rhs_state* st;
  double* partials;      // [B][gridDim.x][2]
  unsigned int* done;    // [B] tiles of the epilogue pass finished (reset by the last one)
  R inv_total;           // 1 / N
  double inv_total_d;    // the same in FP64
  float2* aux;           // defect output [B][C][N] complex64
  size_t l2_window;      // bytes of T kept L2-resident (0: off); host-side launch attribute only
  int nrhs;              // number of right-hand sides (persistent passes)
  int poll_limit;        // polls of a staged-input wait before the pass falls back to global loads (k_pipe_pass)
  int csplit;            // > 1: a one-component strided pass over the csplit components of each RHS, which
                         //      blockIdx.y enumerates (RHS-major); 0 or 1: blockIdx.y is the RHS
};

// Programmatic dependent launch.  The pass kernels are launched so that the next pass's CTAs may become resident
// while this grid drains; each pass calls pdl_wait() before it reads anything an earlier kernel writes (the fields,
// the work buffer, the right-hand-side state), which returns once those grids have completed and their memory is
// visible.  pdl_trigger() lets the dependent grid be scheduled as soon as every CTA of this grid has started.
// Both are no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// |z|^2 accumulated in FP64 (the squares of complex64 words are exact in double)
__device__ __forceinline__ double norm2d(float2 z) { return (double)z.x * z.x + (double)z.y * z.y; }
__device__ __forceinline__ double norm2d(double2 z) { return z.x * z.x + z.y * z.y; }

template <class R> struct ChiCoef {
  cpx<R> a;   // chi(alpha) = a chi0 + b I
  cpx<R> b;
  R s;        // s'(alpha) = s s'0
  R alpha_re, alpha_im;
};

// Component c of this right-hand side's normalised source is identically zero (bit c of reserved[1], set by the
// caller that wrote the source; 0 claims nothing): the prologue may skip reading it.
__device__ __forceinline__ bool source_is_zero(const mmx_rhs_state* st, int c) { return (st->reserved[1] >> c) & 1; }

template <class R> __device__ __forceinline__ ChiCoef<R> chi_coef(const mmx_rhs_state* st) {
  // chi(alpha) = chi0 alpha0_i / alpha_i + i (alpha0 - alpha) / alpha_i ; s'(alpha) = s'0 alpha0_i / alpha_i
  const double ai = st->alpha_im, ar = st->alpha_re;
  const double ratio = st->alpha0_im / ai;
  ChiCoef<R> c;
  c.a = mkc<R>((R)ratio, (R)0);
  // i (d_re + i d_im) / ai = (-d_im + i d_re) / ai
  const double dre = st->alpha0_re - ar, dim = st->alpha0_im - ai;
  c.b = mkc<R>((R)(-dim / ai), (R)(dre / ai));
  c.s = (R)ratio;
  c.alpha_re = (R)ar;
  c.alpha_im = (R)ai;
  return c;
}

__device__ __forceinline__ int64_t pencil_base(int64_t p, int64_t inner, int n) {
  const int64_t o = p / inner;
  return o * (int64_t)n * inner + (p - o * inner);
}

// bulk prefetch of a contiguous global range into L2 (16-byte aligned address, size a multiple of 16)
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// chi(alpha) applied to the C-vector v at voxel vox: out_r = sum_s (a chi_rs + b delta_rs) v_s
template <class R, int C, int CHI>
__device__ __forceinline__ void apply_chi(const cpx<R>* __restrict__ chi, int64_t N, int64_t vox, const ChiCoef<R>& cc,
                                          const cpx<R>* v, cpx<R>* out) {
  if constexpr (CHI == MMX_CHI_SCALAR) {
    const cpx<R> x = cc.a * chi[vox] + cc.b;
#pragma unroll
    for (int c = 0; c < C; ++c) out[c] = x * v[c];
  } else if constexpr (CHI == MMX_CHI_SYM6) {
    // the six distinct entries are read once each (row-major position -> stored entry)
    constexpr int K[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    cpx<R> m[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) m[k] = cc.a * chi[k * N + vox];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      cpx<R> acc = cc.b * v[r];
#pragma unroll
      for (int s = 0; s < 3; ++s) acc += m[K[r * 3 + s]] * v[s];
      out[r] = acc;
    }
  } else {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      cpx<R> acc = cc.b * v[r];
#pragma unroll
      for (int s = 0; s < 3; ++s) acc += (cc.a * chi[(r * 3 + s) * N + vox]) * v[s];
      out[r] = acc;
    }
  }
}

template <class R>
__device__ __forceinline__ void block_reduce_2(double x, double y, double* out2) {
  __shared__ double red[2][32];
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_down_sync(full, x, o);
    y += __shfl_down_sync(full, y, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][warp] = x;
    red[1][warp] = y;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    x = lane < nw ? red[0][lane] : 0.0;
    y = lane < nw ? red[1][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_down_sync(full, x, o);
      y += __shfl_down_sync(full, y, o);
    }
    if (lane == 0) {
      out2[0] = x;
      out2[1] = y;
    }
  }
}

// apply_chi at the neighbouring voxels vox and vox + 1 (vox even, N even), complex64: each stored chi entry of the
// two voxels is one 16-byte load
template <int C, int CHI>
__device__ __forceinline__ void apply_chi2(const float2* __restrict__ chi, int64_t N, int64_t vox,
                                           const ChiCoef<float>& cc, const float2* v0, const float2* v1, float2* o0,
                                           float2* o1) {
  constexpr int M = CHI == MMX_CHI_SCALAR ? 1 : (CHI == MMX_CHI_SYM6 ? 6 : 9);
  float2 m0[M], m1[M];
#pragma unroll
  for (int k = 0; k < M; ++k) {
    const float4 w = *reinterpret_cast<const float4*>(chi + k * N + vox);
    m0[k] = cc.a * make_float2(w.x, w.y);
    m1[k] = cc.a * make_float2(w.z, w.w);
  }
  if constexpr (CHI == MMX_CHI_SCALAR) {
    const float2 x0 = m0[0] + cc.b, x1 = m1[0] + cc.b;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      o0[c] = x0 * v0[c];
      o1[c] = x1 * v1[c];
    }
  } else {
    constexpr int K6[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      float2 a0 = cc.b * v0[r], a1 = cc.b * v1[r];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int k = CHI == MMX_CHI_SYM6 ? K6[r * 3 + s] : r * 3 + s;
        a0 += m0[k] * v0[s];
        a1 += m1[k] * v1[s];
      }
      o0[r] = a0;
      o1[r] = a1;
    }
  }
}

// The decision itself, from |d|^2 and |E + d|^2, by one thread.
static __device__ __forceinline__ void apply_decision(mmx_rhs_state* S, double dd2, double en2) {
  const double nu = sqrt(dd2);
  S->iteration += 1;
  S->last_norm = nu;
  const double prev = S->prev_norm;
  if (prev == 0.0) {  // Python float division by zero in solver.py:1079
    S->status = MMX_STATUS_ZERODIV;
    S->active = 0;
    return;
  }
  const double rel = nu / prev;
  if (rel < 1.0) {
    S->cur ^= 1;
    S->prev_norm = nu;
    S->field_norm = sqrt(en2);
    S->accepted = 1;
  } else {
    S->alpha_im = 1.5 * S->alpha_im;  // solver.py:1092
    S->rejections += 1;
    S->accepted = 0;
  }
  S->residue = S->prev_norm > 0.0 ? S->prev_norm / S->field_norm : 0.0;
  S->active = ((double)S->iteration < S->maxiter) && (S->residue > S->rtol);
}

// Accept / reject of Solution.__iter__ (solver.py:1077-1096) and the stop rule of solve (solver.py:81-83,
// 1112-1121) for one right-hand side, from the epilogue pass partials (deterministic fixed-order reduction).
// Executed by one whole block.
static __device__ void decide_rhs(mmx_rhs_state* S, const double* __restrict__ pp, int ntiles) {
  // The block is the only one still running when it gets here, so the reduction is on the critical path: every
  // thread issues its loads U at a time into U independent accumulators (a fixed order for a given ntiles and
  // block size, hence deterministic) instead of one dependent load-add chain.
  constexpr int U = 8;
  const double2* __restrict__ p2 = reinterpret_cast<const double2*>(pp);
  const int nt = blockDim.x;
  double sd[U], se[U];
#pragma unroll
  for (int u = 0; u < U; ++u) sd[u] = se[u] = 0.0;
  int i = threadIdx.x;
  for (; i + (U - 1) * nt < ntiles; i += U * nt) {
    double2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = p2[i + u * nt];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      sd[u] += v[u].x;
      se[u] += v[u].y;
    }
  }
  for (int u = 0; i < ntiles; i += nt, ++u) {
    const double2 v = p2[i];
    sd[u & (U - 1)] += v.x;
    se[u & (U - 1)] += v.y;
  }
  double dd2 = 0.0, en2 = 0.0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    dd2 += sd[u];
    en2 += se[u];
  }
  double out2[2];
  block_reduce_2<double>(dd2, en2, out2);
  if (threadIdx.x == 0) apply_decision(S, out2[0], out2[1]);
}

// End of the epilogue pass for one tile: publish the tile's partial norms; the last tile of the RHS to finish
// (counted with an atomic after a fence, no waiting) reduces them in a fixed order and takes the decision.
template <class R>
__device__ __forceinline__ void finish_pass_norms(const IterArgs<R>& a, int b, double dd2, double en2) {
  __shared__ int s_last;
  double out2[2];
  block_reduce_2<R>(dd2, en2, out2);
  if (threadIdx.x == 0) {
    double* dst = a.partials + ((int64_t)b * gridDim.x + blockIdx.x) * 2;
    dst[0] = out2[0];
    dst[1] = out2[1];
    __threadfence();
    const unsigned int prev = atomicAdd(a.done + b, 1u);
    s_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    decide_rhs(const_cast<mmx_rhs_state*>(a.st) + b, a.partials + (int64_t)b * gridDim.x * 2, gridDim.x);
    if (threadIdx.x == 0) a.done[b] = 0u;
  }
}
