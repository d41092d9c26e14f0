// Batched persistent NSGS: many independent FC3D problems in one launch.
//
// The problems are one block-diagonal union layout (rows permuted by
// problem, then colour, each (problem, colour) group padded to 32-row slabs).
// A problem is solved by one block, or by a team of blocks that splits every
// colour's slabs evenly and meets at a bounded barrier of its own between
// colours; blocks without a team, and teams that are done, pull problems one
// by one from a work queue ordered by decreasing size.  There is no grid-wide
// synchronisation.  Within a problem the arithmetic is that of the
// single-problem kernel (same row product, same local solver, same reference
// convergence logic with fc3d_compute_error and the tolerance manager), so
// each problem's iterates equal a solo solve's.
//
// What bounds a sweep of one problem is its rounds of slabs per block, each a
// latency chain, so a batch with few problems is as slow as its largest
// problem on one SM; the teams (batch_plan in fc3dgpu_ctx.cu) give the large
// problems the idle SMs.  48 lattices of 130 to 8,901 contacts, 100 FP32
// sweeps: 28.3 ms one block each, 7.6 ms in teams by colours, 3.6 as dataflow
// (fc3dgpu_batch_flow.cuh); 200 lattices, 30 sweeps: 11.1, 7.2 and 3.0 ms.
// In FP64, us a sweep in teams by colours and as dataflow: 2 lattices 279 and
// 214, 10: 294 and 240, 24: 385 and 326; with more than 110 contacts a colour
// and block the FP64 pipes are full either way (40 lattices 463 and 489), and
// so they are with one block a problem (100 small lattices 443 and 455 with
// the same line there): those of up to 40 contacts a colour are dataflow.
#pragma once
#include "fc3dgpu_batch_args.cuh"
#include "fc3dgpu_sweep.cuh"

namespace fc3dgpu {

// The blocks that share a problem: `size` of them from block `first` on.
struct BatchTeam {
  int first, size, rank;
  unsigned epoch;  // barriers passed (the blocks of a team pass the same ones)
};

// Orders every write of the team before it, reactions in global memory
// included, ahead of every read after it.  False when a block of the team did
// not arrive within the poll limit (recorded in the status).
__device__ __forceinline__ bool team_sync(BatchTeam& t, unsigned* flags, unsigned long long limit, int* status) {
  __shared__ int s_ok;
  __syncthreads();
  if (t.size == 1) return true;
  t.epoch++;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) st_release_u32(&flags[blockIdx.x * FC3D_FLAG_STRIDE], t.epoch);
    unsigned long long n = 0;
    int ok = 1;
    for (;;) {
      bool mine = true;
      for (int k = lane; k < t.size; k += 32)
        mine &= (ld_relaxed_u32(&flags[(t.first + k) * FC3D_FLAG_STRIDE]) >= t.epoch);
      if (__all_sync(0xffffffffu, mine)) break;
      if (++n > limit) {
        ok = 0;
        if (lane == 0) atomicOr(status, 1);
        break;
      }
      if (n > 256) __nanosleep(32);
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (lane == 0) s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Sums of three values per thread over the team in a fixed order (warps, then
// the block's warps, then the team's blocks, each a butterfly that carries the
// three values; all but the first by one warp), the same bits in every thread;
// LIGHT: out[0] alone, the light error of the sums 0 and 1.  The block sums of
// a team go through a ring of two slots in global memory: a block writes slot
// k & 1 only after the barrier of call k - 1, which every block passes after
// reading call k - 2's slot.
struct TeamSum {
  double warp[FC3D_BLOCK_MAX / 32][3];
  double out[3];
};
template <bool LIGHT, typename Real>
__device__ __forceinline__ bool team_reduce3(const BatchArgs<Real>& b, BatchTeam& t, TeamSum& S, double v[3],
                                             double out[3]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = lane >> 3, k = lane & 7;
  {
    // value 0 in lane 0, 1 in lane 8, 2 in lane 16
    const bool b16 = lane & 16, b8 = lane & 8;
    const double x = (b16 ? v[2] : v[0]) + __shfl_xor_sync(full, b16 ? v[0] : v[2], 16);
    const double y = v[1] + __shfl_xor_sync(full, v[1], 16);
    double z = (b8 ? y : x) + __shfl_xor_sync(full, b8 ? x : y, 8);
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) z += __shfl_xor_sync(full, z, o);
    if (k == 0 && i < 3) S.warp[w][i] = z;
  }
  __syncthreads();
  double* ring = b.team_part + (size_t)(t.epoch & 1) * FC3D_BATCH_BLOCKS * 4;
  double y = 0.0;
  if (w == 0) {
    if (i < 3)
      for (int q = k; q < (int)(blockDim.x >> 5); q += 8) y += S.warp[q][i];
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) y += __shfl_xor_sync(full, y, o);
    if (t.size > 1 && k == 0 && i < 3) __stcg(&ring[4 * blockIdx.x + i], y);
  }
  if (t.size > 1 && !team_sync(t, b.base.barrier, b.base.spin_limit, b.base.status)) return false;
  if (w == 0) {
    if (t.size > 1) {
      y = 0.0;
      if (i < 3)
        for (int q = k; q < t.size; q += 8) y += __ldcg(&ring[4 * (t.first + q) + i]);
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) y += __shfl_xor_sync(full, y, o);
    }
    if (LIGHT) {
      // the second sum to lane 16, where warp_light_error takes it
      const double second = __shfl_sync(full, y, 8);
      y = warp_light_error(lane == 16 ? second : y);
      if (lane == 0) S.out[0] = y;
    } else if (k == 0 && i < 3) {
      S.out[i] = y;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < (LIGHT ? 1 : 3); q++) out[q] = S.out[q];
  return true;
}

template <typename Real>
__device__ __forceinline__ bool scene_full_error(const BatchArgs<Real>& b, int p0, int p1, double norm_q,
                                                 BatchTeam& t, TeamSum& S, double& full) {
  double v[3], s[3];
  full_error_rows(b.base, v, p0, p1, t.rank * blockDim.x + threadIdx.x, t.size * blockDim.x);
  if (!team_reduce3<false>(b, t, S, v, s)) return false;
  double e = ie_sqrt(s[0]);
  const double scal = fmax(norm_q, fmax(ie_sqrt(s[2]), ie_sqrt(s[1])));
  if (fabs(scal) > DBL_EPSILON) e = ie_div(e, scal);
  full = e;
  return true;
}

// How a block sweeps a problem's colours.  ColourSweep: colour by colour, the
// team's barrier between them (the sums' barrier closes the last one); in FP64
// as dataflow (fc3dgpu_flow64.cuh) where stamped reactions are given and the
// team's blocks have few contacts of a colour.
template <typename Real>
struct ColourSweep {
  typename RangeList<Real>::type& wk;
  int rows;  // of a dataflow unit, 0: by colours
  __device__ __forceinline__ void open(const BatchArgs<Real>& b, const int* sptr, int ncol, const BatchTeam& t) {
    rows = 0;
#ifndef FC3D_FAST_F64
    if constexpr (sizeof(Real) == sizeof(double))
      if (b.base.rs && (sptr[ncol] - sptr[0]) * FC3D_SLAB <=
                           ncol * (t.size > 1 ? FC3D_BATCH_FLOW64_MAX * t.size : FC3D_BATCH_FLOW64_ALONE))
        rows = flow64_rows(sptr, ncol, t.size);
#endif
  }
  __device__ __forceinline__ bool sweep(const BatchArgs<Real>& b, const int* sptr, int ncol, int sweep, Real local_tol,
                                        double acc[3], BatchTeam& t) {
    const SweepArgs<Real>& a = b.base;
#ifndef FC3D_FAST_F64
    if constexpr (sizeof(Real) == sizeof(double))
      if (rows > 0) return flow64_sweep(a, sptr, ncol, rows, t.rank, t.size, sweep, local_tol, acc[0], acc[1]);
#endif
    for (int c = 0; c < ncol; c++) {
      const int s0 = sptr[c], n = sptr[c + 1] - s0;
      process_range<Real>(a, s0 + n * t.rank / t.size, s0 + n * (t.rank + 1) / t.size, local_tol, acc[0], acc[1], wk,
                          nullptr);
      if (c + 1 < ncol && !team_sync(t, a.barrier, a.spin_limit, a.status)) return false;
    }
    return true;
  }
  __device__ __forceinline__ void close(const BatchArgs<Real>&) {}
};

// All sweeps of one problem; false when a wait of the team gave up.
template <typename Real, typename Sweep>
__device__ __forceinline__ bool solve_scene(const BatchArgs<Real>& b, int scene, Sweep& sw, BatchTeam& t, TeamSum& S) {
  const SweepArgs<Real>& a = b.base;
  const int ncol = b.scene_ncol[scene];
  const int* sptr = b.scene_sptr + (size_t)scene * (FC3D_MAX_COLOURS + 1);
  const int p0 = sptr[0] * FC3D_SLAB, p1 = sptr[ncol] * FC3D_SLAB;
  const double norm_q = b.scene_normq[scene];
  const int max_sweeps = b.scene_budget ? b.scene_budget[scene] : a.max_sweeps;
  double working = a.mode == 1 ? a.user_tol : fmax(a.user_tol, a.switch_tol), local_tol = a.local_tol;
  double incr = INFINITY, full = INFINITY, best = INFINITY;
  int sweep = 0, best_sweep = 0;
  bool converged = false;
  if (a.mode == 1 && b.scene_out_prev && b.scene_out_prev[(size_t)scene * 8 + 3] == 0.0) {
    // the FP32 iterate met the tolerance in FP32 arithmetic: FP64 check first
    if (!scene_full_error(b, p0, p1, norm_q, t, S, full)) return false;
    if (full < a.user_tol) {
      if (t.rank == 0 && threadIdx.x == 0) {
        double* o = b.scene_out + (size_t)scene * 8;
        o[0] = 0;
        o[1] = b.scene_out_prev[(size_t)scene * 8 + 1];
        o[2] = full;
        o[3] = 0;
        o[4] = working;
        o[5] = local_tol;
      }
      return true;
    }
  }
  if (max_sweeps > 0) sw.open(b, sptr, ncol, t);
  while (sweep < max_sweeps) {
    sweep++;
    double acc[3] = {0.0, 0.0, 0.0};
    if (!sw.sweep(b, sptr, ncol, sweep, (Real)local_tol, acc, t)) return false;
    double s[3];
    if (!team_reduce3<true>(b, t, S, acc, s)) return false;
    incr = s[0];
    bool stop = false;
    if (a.mode == 1) {
      if (incr < working) {
        if (!scene_full_error(b, p0, p1, norm_q, t, S, full)) return false;
        if (full <= a.user_tol) {
          converged = true;
          stop = true;
        } else if (incr < 1e-15 || incr < DBL_EPSILON * 100.0) {
          local_tol = fmax(local_tol / 100.0, DBL_EPSILON * 1e-6);
        } else if (full > 0.0 && incr > 0.0) {
          double nt = (incr / full) * a.user_tol;
          const double user_min = a.user_tol * 1e-6, floor_tol = DBL_EPSILON * 1e-6;
          const double mint = user_min > floor_tol ? user_min : floor_tol;
          if (nt < mint) nt = mint;
          if (nt > 0.0 && nt < working) working = nt;
        }
        if (!(working > 0.0)) stop = true;
      }
    } else {
      if (!(incr == incr)) {
        if (threadIdx.x == 0) atomicOr(a.status, 2);
        stop = true;
      }
      if (incr < a.switch_tol) stop = true;
      if (incr < 0.99 * best) {
        best = incr;
        best_sweep = sweep;
      } else if (a.stall_window > 0 && sweep - best_sweep >= a.stall_window) {
        stop = true;
      }
      // the reference's adaptive test on this precision's iterate, against
      // max(tol, switch_tol), as in the single-problem kernel
      if (!stop && incr < working) {
        if (!scene_full_error(b, p0, p1, norm_q, t, S, full)) return false;
        const double target = fmax(a.user_tol, a.switch_tol);
        if (full <= target) {
          converged = true;
          stop = true;
        } else if (full > 0.0 && incr > 0.0) {
          double nt = (incr / full) * target;
          const double mint = fmax(target * 1e-6, DBL_EPSILON * 1e-6);
          if (nt < mint) nt = mint;
          if (nt < working) working = nt;
        }
      }
    }
    if (stop) break;
  }
  sw.close(b);
  int info = 1;
  if (a.mode == 1) {
    if (!scene_full_error(b, p0, p1, norm_q, t, S, full)) return false;
    info = full < a.user_tol ? 0 : 1;
    if (sweep == max_sweeps && info > 0) info = -20;
  } else {
    info = converged ? 0 : 1;
  }
  if (t.rank == 0 && threadIdx.x == 0) {
    double* o = b.scene_out + (size_t)scene * 8;
    o[0] = sweep;
    o[1] = incr;
    o[2] = full;
    o[3] = info;
    o[4] = working;
    o[5] = local_tol;
  }
  return true;
}

// The block's problems: its team's, then the queue's.
template <typename Real, typename Sweep>
__device__ __forceinline__ void batch_problems(const BatchArgs<Real>& b, Sweep& sw) {
  __shared__ TeamSum S;
  __shared__ int s_next;
  BatchTeam t = {(int)blockIdx.x, 1, 0, 0};
  if (b.teams) {
    const int4 m = b.teams[blockIdx.x];
    if (m.y > 1) {
      t.first = m.x;
      t.size = m.y;
      t.rank = (int)blockIdx.x - m.x;
      const bool ok = solve_scene<Real>(b, b.order[m.z], sw, t, S);
      if (!ok) {
        sw.close(b);
        return;
      }
      __syncthreads();
      t.size = 1;
      t.rank = 0;
    }
  }
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(b.queue, 1);
    __syncthreads();
    const int k = b.team_scenes + s_next;
    __syncthreads();
    if (k >= b.nscenes) break;
    if (!solve_scene<Real>(b, b.order[k], sw, t, S)) {
      sw.close(b);
      return;
    }
    __syncthreads();
  }
}

template <typename Real>
__global__ void __launch_bounds__(BlockDim<Real>::value, 1) nsgs_batch_kernel(const BatchArgs<Real> b) {
  __shared__ typename RangeList<Real>::type wk;
  ColourSweep<Real> sw = {wk, 0};
  batch_problems<Real>(b, sw);
}

// Launch of `grid` blocks, co-resident (a cooperative launch) when some of
// them form teams.
template <typename Real>
static cudaError_t launch_batch_t(const BatchArgs<Real>& b, int grid, cudaStream_t s) {
  if (grid < 1 || grid > FC3D_BATCH_BLOCKS) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(BlockDim<Real>::value);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = b.teams ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, nsgs_batch_kernel<Real>, b);
}

// Resident blocks of the batched kernel on the current device.
template <typename Real>
static cudaError_t batch_grid_t(int* grid) {
  auto kern = nsgs_batch_kernel<Real>;
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BlockDim<Real>::value, 0);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  *grid = nsm * per_sm < FC3D_BATCH_BLOCKS ? nsm * per_sm : FC3D_BATCH_BLOCKS;
  return cudaSuccess;
}

}  // namespace fc3dgpu
