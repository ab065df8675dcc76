// A chunk of iterations of a small grid in one launch.
//
// On grids of up to a few hundred thousand samples the passes of an iteration take a few microseconds of work each, and
// the launch, the first loads and the drain of each take longer.  Here one cooperative launch keeps every CTA resident
// and runs all passes of all iterations of the chunk; a barrier over the grid takes the place of a kernel boundary.
// Per iteration a 2D grid needs two barriers and a 3D one four:
//
//   axis 0 (forward, Green, inverse) | contiguous axis (inverse, epilogue, and the next iteration's prologue, forward)
//   in 3D the middle axis forward before and inverse after axis 0
//
// What bounds it is latency: a thread's instructions from one barrier to the next, and the trips to L2.  So the stages
// have radices up to 10 (a radix-16 butterfly is one thread's work for a thousand cycles), and whatever a CTA meets again
// stays in shared memory: the fields, chi and sources of its rows (loaded once, the fields written back at the end), the
// twiddles, the k tables, the states of the right-hand sides and the coefficients that follow from them.  Only the work
// buffer crosses L2.
//
// The contiguous-axis tile goes on from E' to the next input chi E' + s'.  That is speculative, as in the fused epilogue
// of mmx_epro.cuh: the divergence guard needs the norms of all tiles.  An extra warp of every CTA reduces them (each CTA
// for itself, in the same order) while the others already run the next pass; if it rejects an update, the rejected
// right-hand sides' prologue and first pass are done again from the old field.  When no right-hand side is active any
// more the launch ends, so a chunk longer than the solve costs nothing.
//
// Waits: a CTA polls the grid barrier's counter at most `polls` times (kLoopPolls; several seconds), then gives up and
// leaves, and the others after it.  The last CTA to leave writes the states: those of the chunk's end, or, when any CTA gave
// up, the old ones as MMX_STATUS_STALLED and inactive (mmx_leave.h).
#pragma once
#include "mmx_gen.cuh"
#include "mmx_leave.h"

constexpr int kLoopWorkers = 256;                // threads of a CTA that run the tiles
constexpr int kLoopThreads = kLoopWorkers + 32;  // and the warp that takes the decisions
constexpr int kLoopMaxRhs = 64;

template <class R> struct LoopArgs : IterArgs<R> {
  GenAxis g[3];     // axis 0, the middle axis of a 3D grid, the contiguous axis
  FFTAxis tab[3];   // their twiddle tables
  int lP0, lP1, PR; // log2 of the pencils per tile (axis 0, middle axis), rows per tile
  int tiles[3];     // per right-hand side (middle axis: per component)
  int kept;         // row tiles per CTA, at most
  int niter;
  unsigned polls;     // of a wait
  unsigned* counter;  // LEAVE_WORDS words
};

enum : int { LOOP_EPI = 1, LOOP_PRO = 2 };

// What the passes need of a right-hand side's state
template <class R> struct LoopCoef {
  ChiCoef<R> cc;
  GenGreen<R> green;
  cpx<R> h;
};
template <class R> __device__ __forceinline__ LoopCoef<R> loop_coef(const mmx_rhs_state* st, double inv_total) {
  const double ar = st->alpha_re, ai = st->alpha_im;
  return LoopCoef<R>{chi_coef<R>(st), GenGreen<R>(ar, ai, inv_total), gen_longitudinal<R>(ar, ai, inv_total)};
}

// chi(alpha) v + (cc.s) s' of one sample from a kept tile (words of one component: `words`)
template <class R, int C, int CHI>
__device__ __forceinline__ void loop_input(const cpx<R>* chi, const cpx<R>* src, int words, int e, const ChiCoef<R>& cc,
                                           const cpx<R>* v, cpx<R>* t) {
  apply_chi<R, C, CHI>(chi, words, e, cc, v, t);
#pragma unroll
  for (int c = 0; c < C; ++c) t[c] += cc.s * src[c * words + e];
}

// One tile of PR rows of all components, whose fields (E, to En), chi and sources are in shared memory as [component]
// [row][sample].  LOOP_EPI: inverse transform of T, E' = E + chi (T - E) to En and the sums of |d|^2 and |E'|^2;
// LOOP_PRO: the transform of chi E + s' to T, with E' (after LOOP_EPI) or E (alone).  T0: the right-hand side's first
// component.  sm: two buffers of C PR n words.
template <class R, int C, int CHI, class Sync>
__device__ __forceinline__ void rows_tile(const GenAxis& g, int PR, int64_t rows, int64_t tile, int64_t N, int mode,
                                          cpx<R>* T0, const cpx<R>* E, cpx<R>* En, const cpx<R>* chi, const cpx<R>* src,
                                          const ChiCoef<R>& cc, const gtw<R>* tw, cpx<R>* sm, int threads, Sync sync,
                                          double& dd2, double& en2) {
  const int n = g.n, nst = g.nst;
  const int64_t row0 = tile * PR;
  cpx<R>* T = T0 + row0 * n;
  const int left = rows - row0 < PR ? (int)(rows - row0) : PR;
  const int all = C * PR, words = PR * n, tid = threadIdx.x;
  cpx<R>*cur = sm, *oth = sm + all * n;
  // tile row r -> its words of T, or null beyond the field
  auto row_of = [&](int r) -> cpx<R>* {
    int c = 0;
    if constexpr (C == 3) c = (r >= PR) + (r >= 2 * PR);
    const int row = r - c * PR;
    return row < left ? T + c * N + row * n : nullptr;
  };
  auto stage = [&](auto dir, int s) {  // between the buffers
    constexpr int DIR = decltype(dir)::value;
    SmallRadices::run(g.r[s], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int Ts = g.T[s];
      for (int e = tid; e < all * Ts; e += threads) {
        const int r = (int)gen_div((unsigned)e, g.mT[s]);
        const cpx<R>* q = cur + r * n;
        cpx<R>* d = oth + r * n;
        const int i = e - r * Ts, L = g.L[s];
        gen_butterfly<R, RAD, DIR, false>(
            i, g, s, tw, [&](int x) { return q[i + x * Ts]; },
            [&](int o, int x, cpx<R> v) { d[o + x * L] = v; });
      }
    });
    sync();
    cpx<R>* t = cur;
    cur = oth;
    oth = t;
  };
  if (mode & LOOP_EPI) {
    SmallRadices::run(g.r[0], [&](auto rad) {
      constexpr int RAD = decltype(rad)::value;
      const int Ts = g.T[0];
      for (int e = tid; e < all * Ts; e += threads) {
        const int r = (int)gen_div((unsigned)e, g.mT[0]);
        const cpx<R>* q = row_of(r);
        cpx<R>* d = cur + r * n;
        const int i = e - r * Ts;
        if (q)
          gen_butterfly<R, RAD, +1, true>(
              i, g, 0, tw, [&](int x) { return q[i + x * Ts]; }, [&](int o, int x, cpx<R> v) { d[o + x] = v; });
      }
    });
    sync();
    for (int s = 1; s < nst; ++s) stage(std::integral_constant<int, +1>{}, s);
    for (int e = tid; e < left * n; e += threads) {
      const int row = (int)gen_div((unsigned)e, g.mn), j = e - row * n;
      cpx<R> ev[C], v[C], d[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        ev[c] = E[c * words + e];
        v[c] = cur[(c * PR + row) * n + j] - ev[c];
      }
      apply_chi<R, C, CHI>(chi, words, e, cc, v, d);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        ev[c] = ev[c] + d[c];
        En[c * words + e] = ev[c];
        dd2 += norm2d(d[c]);
        en2 += norm2d(ev[c]);
      }
      loop_input<R, C, CHI>(chi, src, words, e, cc, ev, v);
#pragma unroll
      for (int c = 0; c < C; ++c) cur[(c * PR + row) * n + j] = v[c];
    }
  } else {
    for (int e = tid; e < left * n; e += threads) {
      const int row = (int)gen_div((unsigned)e, g.mn), j = e - row * n;
      cpx<R> v[C], t[C];
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = E[c * words + e];
      loop_input<R, C, CHI>(chi, src, words, e, cc, v, t);
#pragma unroll
      for (int c = 0; c < C; ++c) cur[(c * PR + row) * n + j] = t[c];
    }
  }
  if (!(mode & LOOP_PRO)) return;
  sync();
  for (int s = 0; s + 1 < nst; ++s) stage(std::integral_constant<int, -1>{}, s);
  SmallRadices::run(g.r[nst - 1], [&](auto rad) {
    constexpr int RAD = decltype(rad)::value;
    const int Ts = g.T[nst - 1];
    for (int e = tid; e < all * Ts; e += threads) {
      const int r = (int)gen_div((unsigned)e, g.mT[nst - 1]);
      cpx<R>* d = row_of(r);
      const cpx<R>* q = cur + r * n;
      const int i = e - r * Ts;
      if (d)
        gen_butterfly<R, RAD, -1, false>(
            i, g, nst - 1, tw, [&](int x) { return q[i + x * Ts]; }, [&](int, int x, cpx<R> v) { d[i + x * Ts] = v; });
    }
  });
}

// sum of x and y over the worker threads, to out by thread 0; red: 2 * kLoopWorkers / 32 doubles
template <class Sync>
__device__ __forceinline__ void worker_sums(double x, double y, double* red, double* out, Sync sync) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, o);
    y += __shfl_down_sync(0xffffffffu, y, o);
  }
  constexpr int W = kLoopWorkers / 32;
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[2 * warp] = x;
    red[2 * warp + 1] = y;
  }
  sync();
  if (threadIdx.x == 0) {
    double sx = 0.0, sy = 0.0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      sx += red[2 * w];
      sy += red[2 * w + 1];
    }
    out[0] = sx;
    out[1] = sy;
  }
}

// The layout of a CTA's shared memory, in bytes.
template <class R> struct LoopShared {
  size_t tw[3], k[3], states, coef, red, flags, kept, work, bytes;
  __host__ __device__ static size_t up(size_t x) { return (x + 15) & ~(size_t)15; }
  // kept_bytes: of the row tiles; work_bytes: the buffers of a tile in progress
  __host__ __device__ LoopShared(const GenAxis* g, int ndim, int nrhs, size_t kept_bytes, size_t work_bytes) {
    size_t o = 0;
    for (int a = 0; a < 3; ++a) {
      tw[a] = o;
      if (a != 1 || ndim == 3) o += (size_t)g[a].n * sizeof(gtw<R>);
    }
    for (int a = 0; a < 3; ++a) {
      k[a] = o;
      if (a != 1 || ndim == 3) o += (size_t)g[a].n * sizeof(double);
    }
    states = o = up(o);
    o = up(o + 2 * (size_t)nrhs * sizeof(mmx_rhs_state));
    coef = o;
    o = up(o + 2 * (size_t)nrhs * sizeof(LoopCoef<R>));
    red = o;
    o += 2 * (kLoopWorkers / 32) * sizeof(double);
    flags = o;
    o = up(o + 4 * sizeof(int));
    kept = o;
    o = up(o + kept_bytes);
    work = o;
    bytes = o + work_bytes;
  }
};
// words of a kept row tile: the field twice, chi and the source
template <int C, int CHI> constexpr int kLoopKept = 3 * C + (CHI == MMX_CHI_SCALAR ? 1 : CHI == MMX_CHI_SYM6 ? 6 : 9);

template <class R, int C, int CHI>
__global__ void __launch_bounds__(kLoopThreads, sizeof(R) == 4 ? 2 : 1) k_loop(const __grid_constant__ LoopArgs<R> a) {
  constexpr int M = kLoopKept<C, CHI> - 3 * C;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  const int tid = threadIdx.x, B = a.nrhs, ndim = a.ndim;
  const int words = a.PR * a.g[2].n;  // of one component of a row tile
  const LoopShared<R> lay(a.g, ndim, B, (size_t)a.kept * kLoopKept<C, CHI> * words * sizeof(cpx<R>), 0);
  auto tw = [&](int x) { return reinterpret_cast<gtw<R>*>(mmx_smem_raw + lay.tw[x]); };
  auto kt = [&](int x) { return reinterpret_cast<double*>(mmx_smem_raw + lay.k[x]); };
  for (int x = 0; x < 3; ++x)
    if (x != 1 || ndim == 3) {
      const double* from = a.kvd[x == 2 ? ndim - 1 : x];
      for (int i = tid; i < a.g[x].n; i += kLoopThreads) {
        tw(x)[i] = GenTw<R>::load(a.tab[x], i);
        kt(x)[i] = from[i];
      }
    }
  mmx_rhs_state* S = reinterpret_cast<mmx_rhs_state*>(mmx_smem_raw + lay.states);    // [2][B]
  LoopCoef<R>* coef = reinterpret_cast<LoopCoef<R>*>(mmx_smem_raw + lay.coef);       // [2][B]
  constexpr int kWords = sizeof(mmx_rhs_state) / sizeof(int);
  for (int w = tid; w < B * kWords; w += kLoopThreads)
    reinterpret_cast<int*>(S)[w] = reinterpret_cast<const int*>(a.st)[w];
  double* red = reinterpret_cast<double*>(mmx_smem_raw + lay.red);
  volatile int* flags = reinterpret_cast<int*>(mmx_smem_raw + lay.flags);  // any active, any rejected, stalled or last, -
  cpx<R>* kept = reinterpret_cast<cpx<R>*>(mmx_smem_raw + lay.kept);
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(mmx_smem_raw + lay.work);
  __syncthreads();
  bool any = false;
  for (int b = 0; b < B; ++b) any |= S[b].active != 0;
  auto leave = [&](bool gave_up) {  // by the whole CTA; the last one clears the counters
    __syncthreads();
    if (tid == 0) {
      const LeaveResult r = leave_launch(gridDim.x, gave_up, [&](int word, unsigned v) {
        __threadfence();
        return atomicAdd(a.counter + word, v);
      });
      if (r.last)
        for (int w = 0; w < LEAVE_WORDS; ++w) a.counter[w] = 0u;
      flags[2] = r.last;
      flags[3] = r.stalled;
    }
    __syncthreads();
    return LeaveResult{flags[2] != 0, flags[3] != 0};
  };
  if (!any) {  // the same in every CTA: nobody writes the states before all have left
    leave(false);
    return;
  }
  for (int b = tid; b < B; b += kLoopThreads) coef[b] = loop_coef<R>(S + b, a.inv_total_d);

  const bool worker = tid < kLoopWorkers;
  const PartSync sync{kLoopWorkers};
  const int64_t N = a.N;
  const unsigned inner0 = (unsigned)(N / a.dims[0]);
  const int64_t rows = N / a.g[2].n;
  const int row_tiles = B * a.tiles[2];
  // f(k, b, tile, rows of it): the row tiles of this CTA
  auto each_row_tile = [&](auto&& f) {
    for (int k = 0, t = blockIdx.x; t < row_tiles; ++k, t += gridDim.x) {
      const int b = t / a.tiles[2], tile = t - b * a.tiles[2];
      f(k, b, tile);
    }
  };
  auto tile_of = [&](int k) { return kept + (size_t)k * kLoopKept<C, CHI> * words; };  // [E0 | E1 | chi | source]
  each_row_tile([&](int k, int b, int tile) {
    const int64_t row0 = (int64_t)tile * a.PR, v0 = row0 * a.g[2].n;
    const int count = (int)(rows - row0 < a.PR ? rows - row0 : a.PR) * a.g[2].n;
    const int64_t f = (int64_t)b * C * N + v0;
    const cpx<R>* E = (S[b].cur ? a.E1 : a.E0) + f;
    cpx<R>* to = tile_of(k);
    for (int c = 0; c < C; ++c)
      for (int e = tid; e < count; e += kLoopThreads) {
        to[(S[b].cur ? C + c : c) * words + e] = E[c * N + e];
        to[(2 * C + M + c) * words + e] = a.src[f + c * N + e];
      }
    for (int m = 0; m < M; ++m)
      for (int e = tid; e < count; e += kLoopThreads) to[(2 * C + m) * words + e] = a.chi[m * N + v0 + e];
  });
  unsigned rounds = 0;
  int cur = 0;  // S + cur * B: the states

  // grid barrier; false when it gave up
  auto barrier = [&]() -> bool {
    __syncthreads();
    ++rounds;
    if (tid == 0) {
      // release: what the CTA's threads wrote before the block barrier; acquire: what the others' did
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counter) : "memory");
      const unsigned want = rounds * gridDim.x;
      int stalled = 0;
      for (unsigned polls = 0;; ++polls) {
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.counter) : "memory");
        if ((int)(seen - want) >= 0) break;
        if (polls >= a.polls) {
          stalled = 1;
          break;
        }
      }
      flags[2] = stalled;
    }
    __syncthreads();
    return !flags[2];
  };
  // the rows of every active right-hand side (redo: of the rejected ones)
  auto rows_pass = [&](int mode, bool redo) {
    each_row_tile([&](int k, int b, int tile) {
      const mmx_rhs_state* st = S + cur * B + b;
      if (!st->active || (redo && st->accepted)) return;
      cpx<R>* E = tile_of(k);
      const int now = st->cur ? C * words : 0;
      double dd2 = 0.0, en2 = 0.0;
      rows_tile<R, C, CHI>(a.g[2], a.PR, rows, tile, N, mode, a.T + (int64_t)b * C * N, E + now, E + (C * words - now),
                           E + 2 * C * words, E + (2 * C + M) * words, coef[cur * B + b].cc, tw(2), sm, kLoopWorkers, sync,
                           dd2, en2);
      if (mode & LOOP_EPI) worker_sums(dd2, en2, red, a.partials + 2 * ((int64_t)b * a.tiles[2] + tile), sync);
      sync();  // the tile's shared memory and the sums are free again
    });
  };
  auto middle_pass = [&](auto dir, bool redo) {
    constexpr int DIR = decltype(dir)::value;
    const mmx_rhs_state* st = S + cur * B;
    for (int t = blockIdx.x; t < B * C * a.tiles[1]; t += gridDim.x) {
      const int f = t / a.tiles[1], tile = t - f * a.tiles[1], b = f / C;
      if (!st[b].active || (redo && st[b].accepted)) continue;
      cpx<R>* plane = a.T + (int64_t)f * N;
      strided_tile<R, DIR, SmallRadices>(a.g[1], a.lP1, (unsigned)a.dims[2], N / a.dims[1], tile, plane, plane, tw(1), sm,
                                         kLoopWorkers, sync);
      sync();
    }
  };
  auto green_pass = [&](bool redo) {
    const mmx_rhs_state* st = S + cur * B;
    for (int t = blockIdx.x; t < B * a.tiles[0]; t += gridDim.x) {
      const int b = t / a.tiles[0], tile = t - b * a.tiles[0];
      if (!st[b].active || (redo && st[b].accepted)) continue;
      const unsigned p = ((unsigned)tile << a.lP0) + (tid & ((1 << a.lP0) - 1));
      double k1 = 0.0, k2 = 0.0;
      if (p < inner0) {
        if (ndim == 3) {
          const unsigned i1 = gen_div(p, a.g[2].mn);
          k1 = kt(1)[i1];
          k2 = kt(2)[p - i1 * a.g[2].n];
        } else {
          k1 = kt(2)[p];
        }
      }
      const LoopCoef<R>& q = coef[cur * B + b];
      green_tile<R, C, SmallRadices>(a.g[0], a.lP0, ndim, inner0, N, p, a.T + (int64_t)b * C * N, k1, k2, q.green, q.h,
                                     tw(0), kt(0), sm, kLoopWorkers, sync);
      sync();
    }
  };
  auto decide = [&] {  // the last warp
    const int lane = tid & 31;
    int any_active = 0, any_rejected = 0;
    for (int b = 0; b < B; ++b) {
      const mmx_rhs_state* from = S + cur * B + b;
      mmx_rhs_state* to = S + (cur ^ 1) * B + b;
      if (lane < kWords) reinterpret_cast<int*>(to)[lane] = reinterpret_cast<const int*>(from)[lane];
      __syncwarp();
      if (!from->active) {
        if (lane == 0) coef[(cur ^ 1) * B + b] = coef[cur * B + b];
        continue;
      }
      const double2* p = reinterpret_cast<const double2*>(a.partials) + (int64_t)b * a.tiles[2];
      constexpr int U = 4;
      double x[U], y[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = y[u] = 0.0;
      for (int i = lane; i < a.tiles[2]; i += 32 * U) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i + 32 * u < a.tiles[2]) {
            const double2 v = p[i + 32 * u];
            x[u] += v.x;
            y[u] += v.y;
          }
      }
      double dd2 = (x[0] + x[1]) + (x[2] + x[3]), en2 = (y[0] + y[1]) + (y[2] + y[3]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        dd2 += __shfl_down_sync(0xffffffffu, dd2, o);
        en2 += __shfl_down_sync(0xffffffffu, en2, o);
      }
      if (lane == 0) {
        apply_decision(to, dd2, en2);
        coef[(cur ^ 1) * B + b] =
            to->alpha_im == from->alpha_im ? coef[cur * B + b] : loop_coef<R>(to, a.inv_total_d);
      }
      __syncwarp();
      any_active |= to->active;
      any_rejected |= to->active && !to->accepted;
    }
    if (lane == 0) {
      flags[0] = any_active;
      flags[1] = any_rejected;
    }
  };

  __syncthreads();
  // One pass and one barrier per round.  `pending`: the norms of an update wait for their decision, which is taken beside
  // the pass that follows the contiguous axis (speculatively also on rejected or finished right-hand sides).
  enum { ROWS, FORWARD, GREEN, INVERSE };
  const int after_rows = ndim == 3 ? FORWARD : GREEN;
  int pass = ROWS, mode = LOOP_PRO, done = 0;
  bool ok = true, pending = false, redo = false;
  for (;;) {
    const bool finished = done == a.niter && pass == after_rows && !redo;
    if (worker) {
      if (finished) {
      } else if (pass == ROWS) {
        rows_pass(mode, redo);
      } else if (pass == FORWARD) {
        middle_pass(std::integral_constant<int, -1>{}, redo);
      } else if (pass == GREEN) {
        green_pass(redo);
      } else {
        middle_pass(std::integral_constant<int, +1>{}, false);
      }
    } else if (pending && pass == after_rows) {
      decide();
    }
    if (finished) {  // nothing follows the last decision, which every CTA has taken for itself
      __syncthreads();
      cur ^= 1;
      break;
    }
    if (!(ok = barrier())) break;
    if (pass == ROWS) {
      pending = (mode & LOOP_EPI) != 0;
      pass = after_rows;
      continue;
    }
    if (pass == after_rows) {
      if (pending) {
        pending = false;
        cur ^= 1;
        if (!flags[0]) break;
        if (flags[1]) {  // the rejected right-hand sides' input again, from the old field
          redo = true;
          mode = LOOP_PRO;
          pass = ROWS;
          continue;
        }
      }
      redo = false;
    }
    if (pass == INVERSE || (pass == GREEN && ndim == 2)) {
      pass = ROWS;
      ++done;
      mode = LOOP_EPI | (done < a.niter ? LOOP_PRO : 0);
    } else {
      ++pass;
    }
  }
  if (ok) {
    each_row_tile([&](int k, int b, int tile) {
      const int64_t row0 = (int64_t)tile * a.PR, v0 = row0 * a.g[2].n;
      const int count = (int)(rows - row0 < a.PR ? rows - row0 : a.PR) * a.g[2].n;
      const int now = S[cur * B + b].cur;
      cpx<R>* E = (now ? a.E1 : a.E0) + (int64_t)b * C * N + v0;
      const cpx<R>* from = tile_of(k) + (now ? C * words : 0);
      for (int c = 0; c < C; ++c)
        for (int e = tid; e < count; e += kLoopThreads) E[c * N + e] = from[c * words + e];
    });
  }
  const LeaveResult r = leave(!ok);
  if (!r.last) return;
  mmx_rhs_state* out = const_cast<mmx_rhs_state*>(a.st);
  if (r.stalled) {
    for (int b = tid; b < B; b += kLoopThreads) {
      out[b].status |= MMX_STATUS_STALLED;
      out[b].active = 0;
    }
  } else {
    for (int w = tid; w < B * kWords; w += kLoopThreads)
      reinterpret_cast<int*>(out)[w] = reinterpret_cast<const int*>(S + cur * B)[w];
  }
}

// ---------------------------------------------------------------------------------------------------------------
// A chunk of iterations of a 1D grid: one CTA per right-hand side, everything in shared memory (chi and the source if
// they fit), nothing to wait for.  The epilogue forms the next input at once, from the old field again after a rejection.
// ---------------------------------------------------------------------------------------------------------------
template <class R> struct LineArgs : IterArgs<R> {
  GenAxis g;
  int niter;
  int staged;  // chi and the source are kept in shared memory
};
constexpr int kLineThreads = kLoopWorkers;

template <class R> __host__ __device__ inline size_t line_bytes(int n, int C, int M, bool staged) {
  const size_t word = sizeof(cpx<R>);
  return n * sizeof(gtw<R>) + (2 * C * n + 2 * C * (size_t)n + (staged ? (M + C) * (size_t)n : 0)) * word +
         ((n * sizeof(double) + 15) & ~(size_t)15) + 2 * (kLineThreads / 32) * sizeof(double) + sizeof(mmx_rhs_state) + 16;
}

template <class R, int C, int CHI>
__global__ void __launch_bounds__(kLineThreads, 1) k_line(const __grid_constant__ LineArgs<R> a) {
  constexpr int M = CHI == MMX_CHI_SCALAR ? 1 : CHI == MMX_CHI_SYM6 ? 6 : 9;
  extern __shared__ __align__(16) unsigned char mmx_smem_raw[];
  const int tid = threadIdx.x, b = blockIdx.x, n = a.g.n, nst = a.g.nst;
  gtw<R>* tw = reinterpret_cast<gtw<R>*>(mmx_smem_raw);
  cpx<R>* cur = reinterpret_cast<cpx<R>*>(tw + n);
  cpx<R>* oth = cur + C * n;
  cpx<R>* E = oth + C * n;  // the field, and the next one
  cpx<R>* En = E + C * n;
  cpx<R>* staged = En + C * n;
  double* sk0 = reinterpret_cast<double*>(staged + (a.staged ? (M + C) * n : 0));
  double* red = sk0 + ((n + 1) & ~1);
  mmx_rhs_state* st = reinterpret_cast<mmx_rhs_state*>(red + 2 * (kLineThreads / 32));
  constexpr int kWords = sizeof(mmx_rhs_state) / sizeof(int);
  if (tid < kWords) reinterpret_cast<int*>(st)[tid] = reinterpret_cast<const int*>(a.st + b)[tid];
  for (int i = tid; i < n; i += kLineThreads) {
    tw[i] = GenTw<R>::load(a.ax, i);
    sk0[i] = a.kvd[0][i];
  }
  __syncthreads();
  if (!st->active) return;
  const int64_t f = (int64_t)b * C * n;
  const cpx<R>* from = (st->cur ? a.E1 : a.E0) + f;
  for (int i = tid; i < C * n; i += kLineThreads) E[i] = from[i];
  const cpx<R>*chi = a.chi, *src = a.src + f;
  if (a.staged) {
    for (int i = tid; i < M * n; i += kLineThreads) staged[i] = a.chi[i];
    for (int i = tid; i < C * n; i += kLineThreads) staged[M * n + i] = a.src[f + i];
    chi = staged;
    src = staged + M * n;
  }
  __syncthreads();

  auto stages = [&](auto dir) {
    constexpr int DIR = decltype(dir)::value;
    for (int s = 0; s < nst; ++s) {
      SmallRadices::run(a.g.r[s], [&](auto rad) {
        constexpr int RAD = decltype(rad)::value;
        const int T = a.g.T[s];
        for (int e = tid; e < C * T; e += kLineThreads) {
          const int c = C == 3 ? (e >= T) + (e >= 2 * T) : 0;
          const cpx<R>* q = cur + c * n;
          cpx<R>* d = oth + c * n;
          const int i = e - c * T, L = a.g.L[s];
          gen_butterfly<R, RAD, DIR, false>(
              i, a.g, s, tw, [&](int x) { return q[i + x * T]; }, [&](int o, int x, cpx<R> v) { d[o + x * L] = v; });
        }
      });
      __syncthreads();
      cpx<R>* t = cur;
      cur = oth;
      oth = t;
    }
  };
  auto input = [&] {  // chi E + s'
    const ChiCoef<R> cc = chi_coef<R>(st);
    for (int j = tid; j < n; j += kLineThreads) {
      cpx<R> v[C], t[C];
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = E[c * n + j];
      apply_chi<R, C, CHI>(chi, n, j, cc, v, t);
#pragma unroll
      for (int c = 0; c < C; ++c) cur[c * n + j] = t[c] + cc.s * src[c * n + j];
    }
    __syncthreads();
  };
  input();
  int side = st->cur;  // of E
  for (int it = 0; it < a.niter; ++it) {
    const ChiCoef<R> cc = chi_coef<R>(st);
    const double ar = st->alpha_re, ai = st->alpha_im, inv = a.inv_total_d;
    stages(std::integral_constant<int, -1>{});
    const GenGreen<R> green(ar, ai, inv);
    const cpx<R> h = C == 3 ? gen_longitudinal<R>(ar, ai, inv) : mkc<R>((R)0, (R)0);
    for (int j = tid; j < n; j += kLineThreads) {
      const double k0 = sk0[j];
      const cpx<R> g = green(k0 * k0);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        cpx<R>& F = cur[c * n + j];
        // along the axis P_L passes the field (at k = 0 too), across it nothing
        F = (C == 3 && c == 0) ? F * h : F * g;
      }
    }
    __syncthreads();
    stages(std::integral_constant<int, +1>{});
    double dd2 = 0.0, en2 = 0.0;
    for (int j = tid; j < n; j += kLineThreads) {
      cpx<R> ev[C], v[C], d[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        ev[c] = E[c * n + j];
        v[c] = cur[c * n + j] - ev[c];
      }
      apply_chi<R, C, CHI>(chi, n, j, cc, v, d);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        ev[c] = ev[c] + d[c];
        En[c * n + j] = ev[c];
        dd2 += norm2d(d[c]);
        en2 += norm2d(ev[c]);
      }
      apply_chi<R, C, CHI>(chi, n, j, cc, ev, v);
#pragma unroll
      for (int c = 0; c < C; ++c) cur[c * n + j] = v[c] + cc.s * src[c * n + j];
    }
    double sums[2];
    worker_sums(dd2, en2, red, sums, BlockSync());
    if (tid == 0) apply_decision(st, sums[0], sums[1]);
    __syncthreads();
    if (st->cur != side) {  // (a state that ends with a status keeps `accepted` and its field)
      side ^= 1;
      cpx<R>* t = E;
      E = En;
      En = t;
    }
    if (!st->active) break;
    if (!st->accepted) input();
  }
  cpx<R>* to = (st->cur ? a.E1 : a.E0) + f;
  for (int i = tid; i < C * n; i += kLineThreads) to[i] = E[i];
  if (tid < kWords) reinterpret_cast<int*>(const_cast<mmx_rhs_state*>(a.st + b))[tid] = reinterpret_cast<int*>(st)[tid];
}
