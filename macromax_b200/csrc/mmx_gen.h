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

struct GenTile {
  GenAxis ax;
  int lP = 0;       // log2 of the pencils (rows) per tile
  int threads = 0;  // 0: no such pass (the axis has no plan, or its tile does not fit)
  size_t smem = 0;
  int64_t tiles = 0;
};

// The plan of an axis for launches bound by latency: radices 4, 5, 3, 2, 7, 11, 13.
bool gen_small_plan(int n, GenAxis* ax);

// Tile of a pass over `outer * inner` pencils of n samples for C components (GEN_STRIDED, GEN_ROWS: C = 1); copies: the
// number of independent such passes in one launch (right-hand sides, or components of them).
GenTile gen_tile(GenKind kind, int n, int C, bool dbl, int64_t outer, int64_t inner, int64_t copies, int sms);

// Launch one pass.  a: the iteration arguments (outer, inner, T, ... set by the caller; st may be null for the plain
// transforms).  in / out / scale: the plain transforms' buffers and factor; C: the field's components; fields: the
// launch's second dimension for the plain transforms; dir: -1 forward, +1 inverse.  pdl: programmatic dependent launch.
template <class R>
cudaError_t gen_launch(GenKind kind, const GenTile& t, const IterArgs<R>& a, int C, int chi_kind, int dir, int batch,
                       const void* in, void* out, R scale, bool pdl, cudaStream_t s);
