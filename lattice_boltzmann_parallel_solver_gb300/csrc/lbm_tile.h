// lbm_tile.h -- host interface of the several-steps-per-launch tile kernels
// (lbm_tile.cuh) for one lattice.
#pragma once
#include <cstddef>

#include "lbm_fused.cuh"

namespace lbm {

// How a lattice is cut: tiles_x x tiles_y tiles, each taken through ksteps
// steps per launch (odd, so that the buffer a run of n steps ends in does not
// depend on the cut) by a block of `threads`; ksteps == 1: no tiling.
struct TilePlan {
  int ksteps = 1, tiles_x = 1, tiles_y = 1, threads = 0;
  bool wide = false;  // regions of up to twice the columns
  size_t smem = 0;     // shared memory of a launch
  int smem_limit = 0;  // the most a block of this device may ask for
};

// the plan for runs of at least three steps of this lattice in this storage
TilePlan tile_plan(int storage, const KParams& P);
// one launch of plan.ksteps steps (or fewer, odd); `overlap`: the launch before
// it in the stream was one of the same run, so its start may overlap that
// one's end.  P.seed is the unhashed seed of the first step.
int tile_launch(int storage, const TilePlan& plan, int ksteps, const KParams& P, bool overlap, cudaStream_t s);
// once per run, before the first launch
int tile_prepare(int storage, const TilePlan& plan, const KParams& P);

}  // namespace lbm
