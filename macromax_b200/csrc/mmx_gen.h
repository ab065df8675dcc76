// Plans and launchers of the passes for axes of any length (kernels: mmx_gen.cuh, launchers: mmx_gen.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mmx_device.cuh"

#define MMX_GEN_STAGES 8

// Radix plan of one axis: stage s has radix r[s], T[s] = n / r[s] butterflies per pencil and span L[s] (the product of
// the radices before it); m* are the multipliers of the exact division x / d = (x m) >> 32, m = 2^32 / d + 1, valid for
// x d < 2^32.
struct GenAxis {
  int n, nst;
  int r[MMX_GEN_STAGES], T[MMX_GEN_STAGES], L[MMX_GEN_STAGES], ts[MMX_GEN_STAGES];  // ts = T / L
  unsigned mT[MMX_GEN_STAGES], mL[MMX_GEN_STAGES], mn;
};

enum GenKind : int {
  GEN_STRIDED,  // FFT along a strided axis, one component per CTA
  GEN_GREEN,    // axis 0: forward FFT, Green multiply, inverse FFT, all components of a tile in one CTA
  GEN_ROWS,     // FFT along the contiguous axis
  GEN_PRO,      // prologue and forward FFT along the contiguous axis, isotropic chi
  GEN_EPI,      // inverse FFT along the contiguous axis and epilogue, isotropic chi
  GEN_PRO3,     // the same with a 3x3 chi
  GEN_EPI3
};

// Pencils (rows) per tile, before a launch of few tiles narrows them.  Strided: rows of 128 bytes (64 for the Green pass of
// a vector field, whose tile holds three components twice).  Contiguous: rows for about 256 threads (maxT: the most
// butterflies per row of a stage).
constexpr int gen_width(GenKind kind, int C, bool dbl, int maxT) {
  if (kind == GEN_STRIDED || kind == GEN_GREEN) return (dbl ? 8 : 16) >> (kind == GEN_GREEN && C == 3 ? 1 : 0);
  int P = 1;
  while (2 * P * C * maxT <= 256 && P < 32) P *= 2;
  return P;
}
// Threads of a tile: the fewest thread-steps over its stages (a step costs its radix and a constant), where the tiles that
// fit an SM at once (smem bytes each, at most 1024 threads) bring it 1024 threads or nearly; more threads on a tie.
// C: components in the tile.  The 126-sample strided pass took 16.5 us with 64 threads, which is 24 warps on an SM.
constexpr int gen_threads(int nst, int r0, int r1, int r2, int r3, int n, int C, int P, bool rows, long smem) {
  const int r[4] = {r0, r1, r2, r3};
  int threads = 0;
  long best = 0;
  for (int thr = 64; thr <= 256; thr += 32) {
    if (!rows && thr % P) continue;
    const int cols = rows ? thr : thr / P, per = rows ? C * P : C;
    long cost = 0;
    for (int s = 0; s < nst; ++s) cost += (long)((per * (n / r[s]) + cols - 1) / cols) * (r[s] + 4);
    const long by_smem = 227 * 1024 / (smem + 1024), by_regs = 1024 / thr;
    const long resident = (by_smem < by_regs ? by_smem : by_regs) * thr;
    cost = cost * thr * 1024 / (resident < 1 ? 1 : resident);
    if (!threads || cost <= best) {
      best = cost;
      threads = thr;
    }
  }
  return threads;
}

struct GenTile {
  GenAxis ax;
  bool fixed = false;  // the length has a kernel of its own (mmx_len.cuh) and the tile is the one it is compiled for
  int lP = 0;       // log2 of the pencils (rows) per tile
  int threads = 0;  // 0: no such pass (the axis has no plan, or its tile does not fit)
  size_t smem = 0;
  int64_t tiles = 0;
};

// The plan of an axis for chunks in one launch: radices up to 10 and the primes 11 and 13, in the fewest stages.  Measured
// with radices up to 5 / 8 / 10, us per iteration: 1000 samples in 1D 7.9 / 6.5 / 6.2, 256^2 complex64 13.0 / 11.9 / 11.9,
// 300 x 420 15.9 / 15.9 / 14.3, 640 x 600 32.1 / 28.7 / 24.6, 48 x 42 x 44 19.3 / 18.5 / 18.5; up to 16 they need twice the
// registers and leave a quarter of the threads.
bool gen_small_plan(int n, GenAxis* ax);

// Tile of a pass over `outer * inner` pencils of n samples for C components (GEN_STRIDED, GEN_ROWS: C = 1); copies: the
// number of independent such passes in one launch (right-hand sides, or components of them).
GenTile gen_tile(GenKind kind, int n, int C, bool dbl, int64_t outer, int64_t inner, int64_t copies, int sms);

// Lengths with kernels of their own: 32 .. 192, the product of two radices up to 16.
constexpr int kLenFirst = 32, kLenLast = 192;
constexpr bool len_has(int n) {
  if (n < kLenFirst || n > kLenLast) return false;
  for (int a = 2; a <= 16; ++a)
    if (n % a == 0 && n / a <= 16) return true;
  return false;
}

// Launch one pass.  a: the iteration arguments (outer, inner, T, ... set by the caller; st may be null for the plain
// transforms).  in / out / scale: the plain transforms' buffers and factor; C: the field's components; fields: the
// launch's second dimension for the plain transforms; dir: -1 forward, +1 inverse.  pdl: programmatic dependent launch.
template <class R>
cudaError_t gen_launch(GenKind kind, const GenTile& t, const IterArgs<R>& a, int C, int chi_kind, int dir, int batch,
                       const void* in, void* out, R scale, bool pdl, cudaStream_t s);

// The same for a tile with `fixed` set, by length; part: lengths with n % kLenParts == part are compiled there.
constexpr int kLenParts = 4;
template <class R, int PART>
cudaError_t len_launch(GenKind kind, const GenTile& t, const IterArgs<R>& a, int C, int dir, int batch, const void* in,
                       void* out, R scale, bool pdl, cudaStream_t s);
