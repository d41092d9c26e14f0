// BatchArgs for host code (the batched kernel itself is in fc3dgpu_batch.cuh).
#pragma once
#include "fc3dgpu_layout.cuh"

// Most blocks of a batched launch
#define FC3D_BATCH_BLOCKS 1024
// Warps of a block of the FP32 batched kernel
#define FC3D_BATCH_WARPS32 10
// Contacts a colour and block up to which a problem's FP64 sweeps go as
// dataflow: of a team's blocks, of a block alone (measured in fc3dgpu_batch.cuh)
#define FC3D_BATCH_FLOW64_MAX 110
#define FC3D_BATCH_FLOW64_ALONE 40

namespace fc3dgpu {

template <typename Real>
struct BatchArgs {
  SweepArgs<Real> base;      // layout, state, controls (sptr/ncol unused)
  int nscenes;
  const int* order;          // problems by decreasing size
  const int* scene_ncol;
  const int* scene_sptr;     // nscenes x (FC3D_MAX_COLOURS + 1), absolute slab indices
  const double* scene_normq; // |q| of each problem
  const int* scene_budget;   // sweep budget of each problem (nullptr: base.max_sweeps)
  int* queue;                // next problem of the queue, zero at launch
  // teams: per block (first block, size, problem in `order`, unused) with
  // size 1 for none; the first team_scenes problems of `order` have teams, the
  // others are queued.  nullptr: no teams.
  const int4* teams;
  int team_scenes;
  double* team_part;         // 2 slots x FC3D_BATCH_BLOCKS x 4 block sums of the teams
  double* scene_out;         // nscenes x 8: sweeps, incr, full error, info, working tol, local tol
  // outputs of the previous (FP32) phase, or nullptr: a problem whose FP32
  // iterate met the tolerance gets its FP64 error checked before any sweep
  const double* scene_out_prev;
};

}  // namespace fc3dgpu
