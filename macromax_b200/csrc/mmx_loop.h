// Chunks of iterations in one launch (kernels: mmx_loop.cuh, launchers: mmx_loop.cu).
#pragma once
#include "mmx_gen.h"
#include "mmx_leave.h"

constexpr unsigned kLoopPolls = 1u << 24;  // of a wait between CTAs, unless the plan says otherwise

struct LoopCfg {
  bool ok = false;
  bool line = false;  // a 1D grid (k_line)
  GenAxis g[3] = {};
  int lP0 = 0, lP1 = 0, PR = 1, tiles[3] = {0, 0, 0}, kept = 0, grid = 0, staged = 0;
  size_t smem = 0;
};

// How a chunk of this plan's iterations runs in one launch; ok == false: it cannot.
template <class R> LoopCfg loop_config(int ndim, const int64_t* shape, int C, int chi_kind, int B, int sms);

// tab: the twiddle tables per grid axis; polls: of a wait between CTAs, at most; counter: LEAVE_WORDS words (mmx_leave.h).
template <class R>
cudaError_t loop_launch(const LoopCfg& cfg, const IterArgs<R>& a, const FFTAxis* tab, int C, int chi_kind, int B, int niter,
                        unsigned polls, unsigned* counter, cudaStream_t s);
