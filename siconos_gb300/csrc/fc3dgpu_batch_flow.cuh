// The batched FP32 sweeps as dataflow: each problem's team sweeps its slabs as
// the single-problem dataflow kernel does (fc3dgpu_flow.cuh), with no barrier
// between colours.  What bounds a sweep of the colour-by-colour form is its
// six barriers with a load, product, list and solve phase each (76 us a sweep
// for the largest of 48 lattices in teams, 36 us as dataflow; 512 lattices, 30
// sweeps: 13.4 and 6.8 ms).  Needs a symmetric block
// pattern (stamped reactions) and slabs that fit the warps' buffers; the
// colour-by-colour form stays for the others.
#pragma once
#include "fc3dgpu_batch.cuh"
#include "fc3dgpu_flow.cuh"

namespace fc3dgpu {

// FlowSweep: the stamped dataflow sweep of fc3dgpu_flow.cuh over the
// problem's slabs and the team's warps, with no barrier inside a sweep (the
// one of the sums at its end keeps the colour sweep's stop rules).
struct FlowSweep {
  const FlowArgs& f;
  unsigned char* buf;       // the warp's staging buffer
  unsigned long long* bar;  // and its barrier
  unsigned parity;
  bool pending;
  int sh, units, gw, tw, slab0;
  FlowRow xs;

  __device__ __forceinline__ int row_of(int u, int lane) const {
    return lane < (FC3D_SLAB >> sh) ? (u & ((1 << sh) - 1)) * (FC3D_SLAB >> sh) + lane : FC3D_SLAB;
  }
  __device__ __forceinline__ void open(const BatchArgs<float>& b, const int* sptr, int ncol, const BatchTeam& t) {
    const int lane = threadIdx.x & 31;
    slab0 = sptr[0];
    const int n = sptr[ncol] - slab0;
    tw = t.size * FC3D_BATCH_WARPS32;
    // a colour's units over the team's blocks first (warps first: 2 lattices 1.48
    // ms for 30 sweeps, 1.38 so; 48 lattices, 100 sweeps 4.33 and 4.13)
    gw = (threadIdx.x >> 5) * t.size + t.rank;
    for (sh = 0; sh < 5 && (n << (sh + 1)) <= tw;) sh++;
    units = n << sh;
    if (gw < units) {
      const int s = slab0 + (gw >> sh);
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        flow_issue(f, flow_next(b.base, f, s), buf, bar);
      }
      pending = true;
      xs = flow_static<true>(b.base, f, s, row_of(gw, lane), lane);
    }
  }
  __device__ __forceinline__ bool sweep(const BatchArgs<float>& b, const int*, int, int sweep, float local_tol,
                                        double acc[3], BatchTeam&) {
    const SweepArgs<float>& a = b.base;
    const int lane = threadIdx.x & 31;
    bool failed = false;
    for (int u = gw; u < units && !failed; u += tw) {
      const int s = slab0 + (u >> sh), rl = row_of(u, lane);
      const int un = u + tw < units ? u + tw : gw;
      const FlowNext next = flow_next(a, f, slab0 + (un >> sh));
      FlowRow x = xs;
      xs = flow_static<true>(a, f, slab0 + (un >> sh), row_of(un, lane), lane);
      flow_own_r(a, s, rl, x);
      if (pending) {
        if (!mbar_wait_bounded(bar, parity, a.spin_limit, a.status)) {
          failed = true;
          break;
        }
        parity ^= 1u;
        pending = false;
      }
      const bool refill = un != u;
      float rn[3];
      if (!flow_slab<true>(a, f, s, next, buf, bar, rl, lane, local_tol, rn, nullptr, x, sweep, refill)) {
        failed = true;
        break;
      }
      pending = refill;
      if (x.row) {
        const double d0 = (double)x.ro[0] - (double)rn[0], d1 = (double)x.ro[1] - (double)rn[1],
                     d2 = (double)x.ro[2] - (double)rn[2];
        acc[0] += d0 * d0 + d1 * d1 + d2 * d2;
        acc[1] += (double)rn[0] * rn[0] + (double)rn[1] * rn[1] + (double)rn[2] * rn[2];
      }
    }
    return !__syncthreads_or(failed);
  }
  // the record still on its way lands before the buffer is used again
  __device__ __forceinline__ void close(const BatchArgs<float>& b) {
    if (pending) {
      mbar_wait_bounded(bar, parity, exit_wait_limit(b.base.spin_limit), b.base.status);
      parity ^= 1u;
      pending = false;
    }
  }
};

// The FP32 sweeps of a batch whose block pattern is symmetric, as dataflow.
__global__ void __launch_bounds__(FC3D_BATCH_WARPS32 * 32, 1) nsgs_batch_flow_kernel(const BatchArgs<float> b,
                                                                                     const FlowArgs f) {
  extern __shared__ __align__(128) unsigned char batch_smem[];
  __shared__ __align__(8) unsigned long long bars[FC3D_BATCH_WARPS32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    mbar_init(&bars[w], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  FlowSweep sw = {f, batch_smem + (size_t)w * f.buf_bytes, &bars[w], 0u, false, 0, 0, 0, 0, 0, {}};
  batch_problems<float>(b, sw);
}

}  // namespace fc3dgpu
