// Coloured NSGS for 2D friction contact on the GPU (include/fc2dgpu.h).
//
// Layout: contacts permuted by colour (stable in contact order); per permuted
// row its blocks in the caller's order (diagonal included, at dpos), each a
// 2x2 column-major block, with the permuted column index; q, mu, r, u in
// permuted order.  One thread-block cluster per problem, or, for larger
// colours, a cooperative grid over every SM, as dataflow where the block
// pattern is symmetric (k_fc2d_nsgs).
// FP64 without FMA contraction, in the reference's operation order.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <new>
#include <numeric>
#include <type_traits>
#include <vector>

#include "fc2dgpu.h"
#include "fc3dgpu_copy.h"
#include "fc3dgpu_grid_count.cuh"
#include "fc3dgpu_ieee64.cuh"
#include "fc3dgpu_word128.cuh"

extern "C" void fc3dgpu_set_error(const char* fmt, ...);

namespace fc2dgpu {

namespace cg = cooperative_groups;

constexpr int NT_MAX = 512;  // threads per block at most
constexpr int CS_MAX = 16;   // blocks per cluster at most (non-portable size)
constexpr int MAXC = 128;
constexpr int TRACE_CAP = 1 << 16;
constexpr size_t REP_MAX_BYTES = 208 * 1024;  // shared-memory copy of the reactions at most
constexpr int GRID_MAX = 1024;                 // blocks of a cooperative grid at most
constexpr unsigned long long SPIN = 1ull << 22;  // polls of a dataflow wait where no limit is set

template <typename T>
struct Vec2;
template <>
struct Vec2<double> {
  using type = double2;
};
template <>
struct Vec2<float> {
  using type = float2;
};

// Sweep modes: the reference's error evaluations (fc2d_nsgs.c:438-448,
// :496-500) in FP64, and the FP32 phase of the mixed-precision solve.
enum Mode { FULL_FINAL = 0, LIGHT = 1, NO_EVAL = 2, FP32_PHASE = 3 };

template <typename T>
struct Args {
  int nc, ncol;
  const int* cptr;  // ncol + 1 permuted-row bounds of the colours
  const int* rp;    // nc + 1 slot pointer per permuted row
  const int* col;   // permuted column of each slot
  const int* dpos;  // offset in the row of its first diagonal block
  const T* W;       // 4 per slot
  const T* det;     // determinant of each row's diagonal block
  const T* q;
  const T* mu;
  // the sweep's copy of the rows, coalesced: contact k of colour c is lane
  // k % 32 of slab sp[c] + k / 32; per slab its slots (off-diagonal blocks of
  // its longest row, in row order), per slot and lane the permuted column
  // (-1: none) and the block's entries (a00, a01, a10, a11)
  const int* sp;
  const int2* slab;  // (first slot, slots)
  const int* scol;
  const T* sW;
  const T* D;       // 4 per contact: its diagonal block, column-major
  double* r;        // the reactions (FP64, permuted order)
  T* rw;            // the sweep's copy in HBM when it is not replicated
  double* u;
  double norm_q, tol;
  int max_iter;
  int mode;
  double switch_tol;      // FP32 phase: stop below this light error
  int stall;              // FP32 phase: stop after this many sweeps without a new lowest error
  const double* before;   // out[] of the phase run before this one (or null)
  double* part;           // grid team: 2 x GRID_MAX x 4 block partial sums
  // dataflow: the reactions with the sweep that wrote them, contacts of a
  // unit, the grid barrier's count, where a wait that gave up is told
  T* rs;
  int rows;
  unsigned* arrived;
  double* fail;
  unsigned long long spin;  // polls of a wait
  double* trace;
  double* out;  // [0] sweeps, [1] final error, [2] info, [3] last light error
};

// The blocks that share a solve.  A thread-block cluster (up to 16 SMs):
// hardware cluster barrier, partial sums exchanged through distributed
// shared memory.  A cooperative grid (every SM, for colours too large for a
// cluster): grid barrier, partial sums through a ring in global memory.
struct ClusterTeam {
  static constexpr bool grid = false, flow = false, alone = false;
  cg::cluster_group cl;
  template <typename T>
  __device__ explicit ClusterTeam(const Args<T>&) : cl(cg::this_cluster()) {}
  __device__ __forceinline__ int rank() const { return (int)cl.block_rank(); }
  __device__ __forceinline__ int size() const { return (int)cl.num_blocks(); }
  // barrier between colours: the hardware cluster barrier (about 670 cycles
  // on this part), or the block barrier (about 290) for a one-block cluster
  __device__ __forceinline__ void sync() {
    if (size() == 1)
      __syncthreads();
    else
      cl.sync();
  }
  __device__ __forceinline__ void sync_all() { cl.sync(); }
  // the barrier in two halves: what stands between them overlaps its latency
  __device__ __forceinline__ void arrive() {
    if (size() > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  __device__ __forceinline__ void wait() {
    if (size() > 1)
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
      __syncthreads();
  }
};

struct GridTeam {
  static constexpr bool grid = true, flow = false, alone = false;
  unsigned* arrived;
  double* fail;
  unsigned long long spin;
  fc3dgpu::GridCount g;
  template <typename T>
  __device__ explicit GridTeam(const Args<T>& a) : arrived(a.arrived), fail(a.fail), spin(a.spin) {}
  __device__ __forceinline__ bool dead() const { return g.dead; }
  __device__ __forceinline__ void give_up() { g.give_up(*this); }
  __device__ __forceinline__ void sync() { g.sync(*this); }
  __device__ __forceinline__ int rank() const { return (int)blockIdx.x; }
  __device__ __forceinline__ int size() const { return (int)gridDim.x; }
  __device__ __forceinline__ void sync_all() { sync(); }
  __device__ __forceinline__ void arrive() {}
  __device__ __forceinline__ void wait() { sync(); }
};

// The same with FP64 contacts on one lane each (sweep_alone).
struct ClusterAlone : ClusterTeam {
  static constexpr bool alone = true;
  using ClusterTeam::ClusterTeam;
};
struct GridAlone : GridTeam {
  static constexpr bool alone = true;
  using GridTeam::GridTeam;
};

// A cooperative grid whose sweeps are dataflow: the sums of a sweep pass its one
// barrier; the waits for reactions give up as the barrier's do.
struct FlowTeam : GridTeam {
  static constexpr bool flow = true;
  using GridTeam::GridTeam;
};

// Where the sweep keeps the reactions.  HBM: read past L1 (ld.global.cg)
// so every block sees the cluster's latest values after a cluster barrier.
// Replicated: a full copy in the shared memory of every block of the
// cluster; the owner of a contact writes its new reaction into all copies
// (distributed shared memory stores), so every read in the sweep is a local
// shared-memory load.  W and the per-contact constants are read-only and
// stay in the L1 of the block that owns the contact.
template <typename T, bool REP>
struct Reactions {
  using V = typename Vec2<T>::type;
  V* rs;  // this block's copy (REP)
  T* rw;  // HBM copy
  __device__ __forceinline__ V get(int j) const {
    if (REP) return rs[j];
    return __ldcg(reinterpret_cast<const V*>(rw) + j);
  }
  // the reactions of a row's next slots (column -1: none)
  template <int N>
  __device__ __forceinline__ void gather(const int (&col)[N], int, V (&r)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++)
      if (col[i] >= 0) r[i] = get(col[i]);
  }
  __device__ __forceinline__ bool any(bool more) const { return more; }
  template <typename Team>
  __device__ __forceinline__ void put(int j, T x0, T x1, Team& t) const {
    V v;
    v.x = x0;
    v.y = x1;
    if constexpr (REP && !Team::grid) {
      const int cs = t.size();
      for (int k = 0; k < cs; k++) t.cl.map_shared_rank(rs, k)[j] = v;
    } else {
      __stcg(reinterpret_cast<V*>(rw) + j, v);
    }
  }
  // component `comp` alone
  template <typename Team>
  __device__ __forceinline__ void put_component(int j, int comp, T x, Team& t) const {
    if constexpr (REP && !Team::grid) {
      const int cs = t.size();
      for (int k = 0; k < cs; k++) reinterpret_cast<T*>(t.cl.map_shared_rank(rs, k))[2 * j + comp] = x;
    } else {
      __stcg(rw + 2 * (size_t)j + comp, x);
    }
  }
};

// Team-wide sum of N values per thread, in a fixed order (xor-shuffle tree
// in each warp, the warps in order, then the blocks in rank order), so every
// block gets the same bits.  The barrier inside also orders every reaction
// update made before the call.  The block partials go through a two-slot
// ring (shared memory of each cluster block, or global memory for a grid): a
// block writes slot k & 1 only after the barrier of call k - 1, which every
// block passes after reading call k - 2's slot.
template <typename T>
struct Reduce {
  T part[2][4];
  T warp[NT_MAX / 32][4];
  T bcast[4];
  int calls;
};

// The sum of two FP64 values: the same steps as trees of depth log2 (an FP64
// addition takes 64 cycles, so the sums over warps and blocks in order above
// cost more than a colour): the two values share each butterfly, 16 lanes
// each.
template <typename Team>
__device__ __forceinline__ void team_sum2(double v[2], Reduce<double>& R, Team& team, double* gpart) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, which = lane >> 4, k16 = lane & 15;
  auto tree = [&](double x) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  // lanes 0-15 take over value 0, lanes 16-31 value 1
  const double send = which ? v[0] : v[1], keep = which ? v[1] : v[0];
  const double x = tree(keep + __shfl_xor_sync(0xffffffffu, send, 16));
  if (k16 == 0) R.warp[w][which] = x;
  __syncthreads();
  const int slot = R.calls & 1, nw = blockDim.x >> 5;
  double* gslot = gpart + (size_t)slot * GRID_MAX * 4;
  if (w == 0) {
    const double y = tree(k16 < nw ? R.warp[k16][which] : 0.0);
    if (k16 == 0) {
      if constexpr (Team::grid)
        __stcg(&gslot[4 * blockIdx.x + which], y);
      else
        R.part[slot][which] = y;
    }
  }
  team.sync();
  if (w == 0) {
    double y = 0.0;
    if constexpr (Team::grid) {
      for (int b = k16; b < (int)gridDim.x; b += 16) y += __ldcg(&gslot[4 * b + which]);
    } else if (k16 < team.size()) {
      y = team.cl.map_shared_rank(&R.part[slot][0], k16)[which];
    }
    y = tree(y);
    if (k16 == 0) R.bcast[which] = y;
    if (lane == 0) R.calls++;
  }
  __syncthreads();
  v[0] = R.bcast[0];
  v[1] = R.bcast[1];
  __syncthreads();
}

// The sum of N values over the dataflow grid, each step a tree.
template <int N, typename T>
__device__ __forceinline__ void flow_sum(T v[N], Reduce<T>& R, FlowTeam& team, double* gpart) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto tree = [&](T x) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
#pragma unroll
  for (int i = 0; i < N; i++) {
    const T x = tree(v[i]);
    if (lane == 0) R.warp[w][i] = x;
  }
  __syncthreads();
  double* gslot = gpart + (size_t)(R.calls & 1) * GRID_MAX * 4;
  if (threadIdx.x < N) {
    T x = 0;
    for (int k = 0; k < nw; k++) x += R.warp[k][threadIdx.x];
    __stcg(&gslot[4 * blockIdx.x + threadIdx.x], (double)x);
  }
  team.sync();
  if (w == 0) {
    T x[N];
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = 0;
    for (int b = lane; b < (int)gridDim.x; b += 32)
#pragma unroll
      for (int i = 0; i < N; i++) x[i] += (T)__ldcg(&gslot[4 * b + i]);
#pragma unroll
    for (int i = 0; i < N; i++) {
      x[i] = tree(x[i]);
      if (lane == 0) R.bcast[i] = x[i];
    }
    if (lane == 0) R.calls++;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = R.bcast[i];
  __syncthreads();
}

template <int N, typename T, typename Team>
__device__ __forceinline__ void team_sum(T v[N], Reduce<T>& R, Team& team, double* gpart) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; i++) {
    T x = v[i];
    for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) R.warp[w][i] = x;
  }
  __syncthreads();
  const int slot = R.calls & 1;
  double* gslot = gpart + (size_t)slot * GRID_MAX * 4;
  if (threadIdx.x == 0) {
    for (int i = 0; i < N; i++) {
      T s = 0;
      for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += R.warp[k][i];
      if constexpr (Team::grid)
        __stcg(&gslot[4 * blockIdx.x + i], (double)s);
      else
        R.part[slot][i] = s;
    }
  }
  team.sync();
  if constexpr (Team::grid) {
    // the blocks' partials added in order; a warp fetches 32 of them at once
    if (w == 0) {
      T s[N];
#pragma unroll
      for (int i = 0; i < N; i++) s[i] = 0;
      for (int b = 0; b < (int)gridDim.x; b += 32) {
        const int n = min(32, (int)gridDim.x - b);
#pragma unroll
        for (int i = 0; i < N; i++) {
          const T mine = lane < n ? (T)__ldcg(&gslot[4 * (b + lane) + i]) : T(0);
          for (int k = 0; k < n; k++) s[i] += __shfl_sync(0xffffffffu, mine, k);
        }
      }
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < N; i++) R.bcast[i] = s[i];
        R.calls++;
      }
    }
  } else if (w == 0) {
    // lane k fetches block k's partials (the remote loads overlap), lane 0
    // adds them in rank order
    const int cs = team.size();
    T mine[N];
#pragma unroll
    for (int i = 0; i < N; i++) mine[i] = lane < cs ? team.cl.map_shared_rank(&R.part[slot][0], lane)[i] : T(0);
#pragma unroll
    for (int i = 0; i < N; i++) {
      T s = 0;
      for (int k = 0; k < cs; k++) s += __shfl_sync(0xffffffffu, mine[i], k);
      if (lane == 0) R.bcast[i] = s;
    }
    if (lane == 0) R.calls++;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = R.bcast[i];
  __syncthreads();
}

// fc2d_compute_error (fc2d_compute_error.c:40-140): u = q + W r block by
// block (per block w_i = 1.0 w_i + 1.0 (a_i0 r0 + a_i1 r1), the reference's
// 2x2 gemv), natural-map error, relative to max(|r|, |u|, |q|).  FP64 only.
template <bool REP, typename Team>
__device__ double full_error(const Args<double>& a, const Reactions<double, REP>& rx, Reduce<double>& R,
                             Team& team) {
  double v[3] = {0.0, 0.0, 0.0};
  const int g0 = team.rank() * blockDim.x + threadIdx.x, G = team.size() * blockDim.x;
  for (int p = g0; p < a.nc; p += G) {
    double w[2] = {a.q[2 * p], a.q[2 * p + 1]};
    for (int s = a.rp[p]; s < a.rp[p + 1]; s++) {
      const double* blk = a.W + 4 * (size_t)s;
      const double2 x = rx.get(a.col[s]);
      for (int i = 0; i < 2; i++) {
        double t = 0.0;
        t += blk[i] * x.x;
        t += blk[2 + i] * x.y;
        w[i] = 1.0 * w[i] + 1.0 * t;
      }
    }
    __stcg(reinterpret_cast<double2*>(a.u) + p, make_double2(w[0], w[1]));
    const double2 rr = rx.get(p);
    const double r0 = rr.x, r1 = rr.y, mu = a.mu[p];
    double t0 = r0 - w[0] - mu * fabs(w[1]);
    double t1 = r1 - w[1];
    const double normT = fabs(t1);
    if (mu * normT <= -t0) {
      t0 = 0.;
      t1 = 0.;
    } else if (normT > mu * t0) {
      t0 = (mu * normT + t0) / (mu * mu + 1.0);
      t1 = mu * t0 * (double)((t1 > 0) - (t1 < 0));
    }
    t0 = r0 - t0;
    t1 = r1 - t1;
    v[0] += t0 * t0 + t1 * t1;
    v[1] += r0 * r0 + r1 * r1;
    v[2] += w[0] * w[0] + w[1] * w[1];
  }
  team_sum<3>(v, R, team, a.part);
  double e = sqrt(v[0]);
  const double scal = fmax(sqrt(v[1]), fmax(sqrt(v[2]), a.norm_q));
  if (fabs(scal) > DBL_EPSILON) e /= scal;
  return e;
}

// fc2d_nsgs_local_solve (fc2d_nsgs.c:212-252), in the working precision
template <typename T>
__device__ __forceinline__ void local_solve(const T* W, T D, const T* q, T mu, T* P) {
  const T Wnn = W[0], Wtn = W[1], Wnt = W[2], Wtt = W[3];
  if (q[0] > 0) {
    P[0] = 0;
    P[1] = 0;
  } else {
    P[0] = -(Wtt * q[0] - Wnt * q[1]) / D;
    P[1] = -(-Wtn * q[0] + Wnn * q[1]) / D;
    const T muPn = mu * P[0];
    if (fabs(P[1]) > muPn) {
      if (P[1] + muPn < 0) {
        P[0] = -q[0] / (Wnn - mu * Wnt);
        P[1] = -mu * P[0];
      } else {
        P[0] = -q[0] / (Wnn + mu * Wnt);
        P[1] = mu * P[0];
      }
    }
  }
}

// Slots of a row loaded together, ahead of their products.
#define FC2D_NB 8

// The static inputs of a contact (its first slots' columns and entries),
// loaded before the barrier that releases its colour.
template <typename T>
struct Row;
template <>
struct Row<float> {
  int p, first, slots;  // the contact, its slab's slots
  int col[FC2D_NB];
  float4 w[FC2D_NB];
  float2 q;
  float4 d;  // diagonal block
  float det, mu;
};
template <>
struct Row<double> {
  int p, first, slots;
  int col[FC2D_NB];
  double2 w[FC2D_NB];  // row `comp` of the blocks
  double q;
};

template <typename T>
__device__ __forceinline__ void load_slots(const Args<T>& a, Row<T>& x, int t0, int lane, int comp) {
#pragma unroll
  for (int k = 0; k < FC2D_NB; k++) {
    x.col[k] = -1;
    if (t0 + k < x.slots) {
      const size_t e = (size_t)(x.first + t0 + k) * 32 + lane;
      x.col[k] = __ldg(&a.scol[e]);
      if constexpr (sizeof(T) == sizeof(float))
        x.w[k] = __ldg(reinterpret_cast<const float4*>(a.sW) + e);
      else
        x.w[k] = __ldg(reinterpret_cast<const double2*>(a.sW) + 2 * e + comp);
    }
  }
}

template <typename T>
__device__ __forceinline__ void load_row(const Args<T>& a, int c, int k, int comp, Row<T>& x) {
  const int2 s = __ldg(&a.slab[__ldg(&a.sp[c]) + (k >> 5)]);
  x.first = s.x;
  x.slots = s.y;
  x.p = __ldg(&a.cptr[c]) + k;
  const size_t p = (size_t)x.p;
  load_slots(a, x, 0, k & 31, comp);
  if constexpr (sizeof(T) == sizeof(float)) {
    x.q = __ldg(reinterpret_cast<const float2*>(a.q) + p);
    x.d = __ldg(reinterpret_cast<const float4*>(a.D) + p);
    x.det = __ldg(&a.det[p]);
    x.mu = __ldg(&a.mu[p]);
  } else {
    x.q = __ldg(&a.q[2 * p + comp]);
  }
}

// A contact of the FP32 sweep on one lane: its neighbours' reactions are
// fetched together, then the products run in the row's order
// (SBM_row_prod_no_diag_2x2: every block on the diagonal is left out).
template <typename RX, typename Team>
__device__ __forceinline__ void contact32(const Args<float>& a, RX& rx, int k, bool act, Row<float>& x, float& x0,
                                          float& x1, float P[2], Team& team) {
  const int p = x.p;
  const float2 old = rx.get(p);
  float ql[2] = {x.q.x, x.q.y};
  for (int t0 = 0;; t0 += FC2D_NB) {
    float2 r[FC2D_NB];
    rx.gather(x.col, p, r);
#pragma unroll
    for (int i = 0; i < FC2D_NB; i++)
      if (x.col[i] >= 0) {
        ql[0] += x.w[i].x * r[i].x;
        ql[1] += x.w[i].z * r[i].x;
        ql[0] += x.w[i].y * r[i].y;
        ql[1] += x.w[i].w * r[i].y;
      }
    if (!rx.any(t0 + FC2D_NB < x.slots)) break;
    load_slots(a, x, t0 + FC2D_NB, k & 31, 0);
  }
  const float W[4] = {x.d.x, x.d.y, x.d.z, x.d.w};
  P[0] = old.x;
  P[1] = old.y;
  local_solve<float>(W, x.det, ql, x.mu, P);
  x0 = old.x - P[0];
  x1 = old.y - P[1];
  if (act) rx.put(p, P[0], P[1], team);
}

// A contact of the FP64 sweep on two lanes, one component each.  The sweep
// is bound by FP64 warp instructions (64 cycles each on an SM quarter whatever
// their lanes do), so the two rows of every product and the two quotients of
// the local solve run side by side; divisions and comparisons are the integer
// forms of fc3dgpu_ieee64.cuh.  The bits are local_solve's.  Every lane of the
// warp calls it; `act` false stores nothing.
template <typename RX, typename Team>
__device__ __forceinline__ void contact64(const Args<double>& a, RX& rx, int k, int comp, bool act,
                                          Row<double>& x, double& dx, double& pn, Team& team) {
  using namespace fc3dgpu;
  const int p = x.p;
  const double2 o = rx.get(p);
  const double old = comp ? o.y : o.x;
  double2 n, t;  // Wnn, Wtn; Wnt, Wtt
  double mu, det;
  auto block = [&]() {
    n = __ldg(reinterpret_cast<const double2*>(a.D) + 2 * (size_t)p);
    t = __ldg(reinterpret_cast<const double2*>(a.D) + 2 * (size_t)p + 1);
    mu = __ldg(&a.mu[p]);
    det = __ldg(&a.det[p]);
  };
  if (Team::flow) block();  // before the wait; the other teams' registers don't hold it
  double y = x.q;
  for (int t0 = 0;; t0 += FC2D_NB) {
    double2 r[FC2D_NB];
    rx.gather(x.col, p, r);
#pragma unroll
    for (int i = 0; i < FC2D_NB; i++)
      if (x.col[i] >= 0) {
        y += x.w[i].x * r[i].x;
        y += x.w[i].y * r[i].y;
      }
    if (!rx.any(t0 + FC2D_NB < x.slots)) break;
    load_slots(a, x, t0 + FC2D_NB, k & 31, comp);
  }
  const double z = __shfl_xor_sync(0xffffffffu, y, 1);
  const double q0 = comp ? z : y, q1 = comp ? y : z;
  if (!Team::flow) block();
  double P = 0.0;
  const bool contact = !ie_positive(q0);
  // P = -(adjugate q) / D, component by component
  const double s = (comp ? -n.y : t.y) * q0 + (comp ? n.x : -t.x) * q1;
  const double f = ie_div(-s, det);
  const double g = __shfl_xor_sync(0xffffffffu, f, 1);
  const double P0 = comp ? g : f, P1 = comp ? f : g;
  if (contact) {
    P = f;
    const double muPn = mu * P0;
    if (ie_lt(muPn, ie_abs(P1))) {
      // slip backward (P1 + mu P0 < 0) or forward
      const bool back = ie_lt(P1, -muPn);
      const double b = back ? n.x - mu * t.x : n.x + mu * t.x;
      const double S0 = ie_div(-q0, b);
      P = comp ? (back ? -mu : mu) * S0 : S0;
    }
  }
  dx = old - P;
  pn = P;
  if (act) rx.put_component(p, comp, P, team);
}

// All colours of one sweep; v gets this thread's sums |r_old - r_new|^2 and
// |r_new|^2.  row: the static inputs of the thread's first contact of colour
// 0, loaded; left loaded for the next sweep.
template <bool REP, typename Team>
__device__ __forceinline__ void sweep_colours(const Args<float>& a, Reactions<float, REP>& rx, int g0, int G,
                                              Row<float>& row, float v[2], Team& team) {
  auto size = [&](int c) { return __ldg(&a.cptr[c + 1]) - __ldg(&a.cptr[c]); };
  int n = size(0), next;
  for (int c = 0; c < a.ncol; c++, n = next) {
    const int cn = c + 1 < a.ncol ? c + 1 : 0;
    next = size(cn);
    float x0 = 0.f, x1 = 0.f, P[2] = {0.f, 0.f};
    for (int k = g0; k < n; k += G) {
      if (k != g0) {
        // the sums of the contact before, in the sweep's order
        v[0] += x0 * x0 + x1 * x1;
        v[1] += P[0] * P[0] + P[1] * P[1];
        load_row(a, c, k, 0, row);
      }
      contact32(a, rx, k, true, row, x0, x1, P, team);
    }
    if (c + 1 < a.ncol) team.arrive();
    if (g0 < next) load_row(a, cn, g0, 0, row);
    if (g0 < n) {
      v[0] += x0 * x0 + x1 * x1;
      v[1] += P[0] * P[0] + P[1] * P[1];
    }
    if (c + 1 < a.ncol) team.wait();
  }
}

template <bool REP, typename Team>
__device__ __forceinline__ void sweep_colours(const Args<double>& a, Reactions<double, REP>& rx, int g0, int G,
                                              Row<double>& row, double v[2], Team& team) {
  const int comp = g0 & 1, h0 = g0 >> 1, H = G >> 1;
  const int lead = (g0 & ~31) >> 1;  // the warp's first contact, present while any of the warp's is
  auto size = [&](int c) { return __ldg(&a.cptr[c + 1]) - __ldg(&a.cptr[c]); };
  int n = size(0), next;
  for (int c = 0; c < a.ncol; c++, n = next) {
    const int cn = c + 1 < a.ncol ? c + 1 : 0;
    next = size(cn);
    double dx = 0.0, pn = 0.0;
    for (int j = 0; lead + j < n; j += H) {
      const bool act = h0 + j < n;
      const int k = act ? h0 + j : lead + j;
      if (j > 0) {
        v[0] += dx * dx;
        v[1] += pn * pn;
      }
      if (j > 0 || !act) load_row(a, c, k, comp, row);
      contact64(a, rx, k, comp, act, row, dx, pn, team);
      if (!act) dx = pn = 0.0;
    }
    if (c + 1 < a.ncol) team.arrive();
    if (h0 < next) load_row(a, cn, h0, comp, row);
    v[0] += dx * dx;
    v[1] += pn * pn;
    if (c + 1 < a.ncol) team.wait();
  }
}

// local_solve with the integer forms of its divisions and comparisons
__device__ __forceinline__ void local_solve64(const double2 n, const double2 t, double det, const double q[2],
                                              double mu, double P[2]) {
  using namespace fc3dgpu;
  if (ie_positive(q[0])) {
    P[0] = P[1] = 0.0;
    return;
  }
  ie_div2(-(t.y * q[0] - t.x * q[1]), -(-n.y * q[0] + n.x * q[1]), ie_den(det), P[0], P[1]);
  const double muPn = mu * P[0];
  if (ie_lt(muPn, ie_abs(P[1]))) {
    const bool back = ie_lt(P[1], -muPn);
    P[0] = ie_div(-q[0], back ? n.x - mu * t.x : n.x + mu * t.x);
    P[1] = (back ? -mu : mu) * P[0];
  }
}

// The FP64 sweep with a contact a lane, where a requested launch leaves a thread
// more than ALONE_FROM contacts of a colour: two lanes a contact then take twice
// the rounds, each with the whole chain of a contact.
template <bool REP, typename Team>
__device__ __forceinline__ void sweep_alone(const Args<double>& a, Reactions<double, REP>& rx, int g0, int G,
                                            double v[2], Team& team) {
  constexpr int NB = 4;  // slots loaded together
  for (int c = 0; c < a.ncol; c++) {
    const int p0 = __ldg(&a.cptr[c]), n = __ldg(&a.cptr[c + 1]) - p0;
    for (int k = g0; k < n; k += G) {
      const int p = p0 + k;
      const int2 s = __ldg(&a.slab[__ldg(&a.sp[c]) + (k >> 5)]);
      const double2 old = rx.get(p), q = __ldg(reinterpret_cast<const double2*>(a.q) + p);
      double y[2] = {q.x, q.y};
      for (int t0 = 0; t0 < s.y; t0 += NB) {
        int col[NB];
        double2 w[NB][2], r[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) {
          const size_t e = (size_t)(s.x + (t0 + i < s.y ? t0 + i : t0)) * 32 + (k & 31);
          col[i] = t0 + i < s.y ? __ldg(&a.scol[e]) : -1;
          w[i][0] = __ldg(reinterpret_cast<const double2*>(a.sW) + 2 * e);
          w[i][1] = __ldg(reinterpret_cast<const double2*>(a.sW) + 2 * e + 1);
        }
        rx.gather(col, p, r);
#pragma unroll
        for (int i = 0; i < NB; i++)
          if (col[i] >= 0) {
            y[0] += w[i][0].x * r[i].x;
            y[1] += w[i][1].x * r[i].x;
            y[0] += w[i][0].y * r[i].y;
            y[1] += w[i][1].y * r[i].y;
          }
      }
      const double2 wn = __ldg(reinterpret_cast<const double2*>(a.D) + 2 * (size_t)p);
      const double2 wt = __ldg(reinterpret_cast<const double2*>(a.D) + 2 * (size_t)p + 1);
      double P[2];
      local_solve64(wn, wt, __ldg(&a.det[p]), y, __ldg(&a.mu[p]), P);
      const double x0 = old.x - P[0], x1 = old.y - P[1];
      v[0] += x0 * x0 + x1 * x1;
      v[1] += P[0] * P[0] + P[1] * P[1];
      rx.put(p, P[0], P[1], team);
    }
    if (c + 1 < a.ncol) team.sync();
  }
}

// ---- the sweeps as dataflow -------------------------------------------------
// What bounds a colour of a large problem is not its contacts but what stands
// between two colours: a barrier over every SM and then the loads it releases.
// Here a warp takes units of a few contacts and waits only for the reactions
// these read, each stored with the number of the sweep that wrote it.  In a
// colour's order a contact reads the new reactions of lower colours and the
// old ones of higher colours; the pattern is symmetric, so a contact of a
// higher colour cannot write its new one before this contact has written its
// own, and a stamp at least the one needed is the one needed.  Granular
// problems, us a sweep by colours and as dataflow: FP64 24.4 and 18.0 at 367
// contacts, 32.0 and 24.7 at 7,002, 32.1 and 27.3 at 28,008, 60.7 and 33.6 at
// 70,020; FP32 10.2 and 7.7, 14.4 and 9.9, 19.8 and 10.4, 21.5 and 11.2.
// What is left is the chain of a colour's longest rows: with a warp a quarter
// an instruction takes eight cycles and an FP64 one 64.

// Polls of a reaction before the back-off, and the back-off (ns).
#define FC2D_FLOW_SPIN 16
#define FC2D_FLOW_SLEEP_NS 100

// The stamped reactions beside the plain ones (which the error evaluation and
// the end of the solve read): in FP32 one 128-bit word (x, y, stamp), in FP64
// one for each component (value, stamp).
template <typename T>
struct FlowReactions {
  using V = typename Vec2<T>::type;
  static constexpr int L = sizeof(T) == sizeof(double) ? 2 : 1;  // words of a reaction
  T* rw;
  T* rs;
  int sweep;
  bool failed;
  unsigned long long spin;
  __device__ __forceinline__ V get(int j) const { return __ldcg(reinterpret_cast<const V*>(rw) + j); }
  __device__ __forceinline__ bool any(bool more) const { return __any_sync(0xffffffffu, more); }
  __device__ __forceinline__ void stamp(int j, V v, int at) const {
    if constexpr (sizeof(T) == sizeof(float)) {
      fc3dgpu::st_word128(rs + 4 * (size_t)j,
                          (unsigned long long)__float_as_uint(v.x) | (unsigned long long)__float_as_uint(v.y) << 32,
                          (unsigned long long)(unsigned)at);
    } else {
      fc3dgpu::st_word128(rs + 4 * (size_t)j, (unsigned long long)__double_as_longlong(v.x), (unsigned long long)at);
      fc3dgpu::st_word128(rs + 4 * (size_t)j + 2, (unsigned long long)__double_as_longlong(v.y),
                          (unsigned long long)at);
    }
  }
  // Waits for the reactions of a row's next slots.  Every poll loads all of
  // them without a branch between two loads (a slot without a column loads the
  // contact's own word), so it costs one memory latency (with a branch a
  // slot a sweep of 28,008 contacts took 15.1 us in FP32, 12.3 without).  A
  // wait that gives up goes on with what is there: the block ends
  // the solve after the sweep.
  template <int N>
  __device__ __forceinline__ void gather(const int (&col)[N], int p, V (&r)[N]) {
    int from[N], need[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
      from[i] = col[i] >= 0 ? col[i] : p;
      need[i] = sweep - (col[i] >= 0 && col[i] < p ? 0 : 1);
    }
    for (unsigned long long n = 0;; n++) {
      unsigned long long w[N][L][2];
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int k = 0; k < L; k++) fc3dgpu::ld_word128(rs + 4 * (size_t)from[i] + 2 * k, w[i][k][0], w[i][k][1]);
      bool all = true;
#pragma unroll
      for (int i = 0; i < N; i++) {
        bool there = true;
#pragma unroll
        for (int k = 0; k < L; k++) there = there && (int)(unsigned)w[i][k][1] >= need[i];
        if constexpr (L == 1) {
          r[i].x = __uint_as_float((unsigned)w[i][0][0]);
          r[i].y = __uint_as_float((unsigned)(w[i][0][0] >> 32));
        } else {
          r[i].x = __longlong_as_double((long long)w[i][0][0]);
          r[i].y = __longlong_as_double((long long)w[i][L - 1][0]);
        }
        all = all && there;
      }
      if (__all_sync(0xffffffffu, all || failed)) break;
      if (n > spin) failed = true;
      if (n > FC2D_FLOW_SPIN) __nanosleep(FC2D_FLOW_SLEEP_NS);
    }
  }
  template <typename Team>
  __device__ __forceinline__ void put(int j, T x0, T x1, Team&) const {
    V v;
    v.x = x0;
    v.y = x1;
    stamp(j, v, sweep);
    __stcg(reinterpret_cast<V*>(rw) + j, v);
  }
  template <typename Team>
  __device__ __forceinline__ void put_component(int j, int comp, T x, Team&) const {
    fc3dgpu::st_word128(rs + 4 * (size_t)j + 2 * comp, (unsigned long long)__double_as_longlong(x),
                        (unsigned long long)sweep);
    __stcg(rw + 2 * (size_t)j + comp, x);
  }
};

// The reactions of the solve's start (FP64) with sweep 0's stamps, and the
// sweep's plain copy.
template <typename T>
__device__ __forceinline__ FlowReactions<T> open_flow(const Args<T>& a, FlowTeam& team) {
  FlowReactions<T> fx{a.rw, a.rs, 0, false, a.spin};
  for (int j = team.rank() * blockDim.x + threadIdx.x; j < a.nc; j += team.size() * blockDim.x) {
    const double2 x = __ldcg(reinterpret_cast<const double2*>(a.r) + j);
    typename Vec2<T>::type v;
    v.x = (T)x.x;
    v.y = (T)x.y;
    fx.stamp(j, v, 0);
    if (sizeof(T) != sizeof(double)) __stcg(reinterpret_cast<typename Vec2<T>::type*>(a.rw) + j, v);
  }
  team.sync_all();
  return fx;
}

// Contacts and this block's units of each colour: unit u of a colour goes to
// block u mod the grid.
struct FlowTable {
  int n[MAXC], mine[MAXC];
  template <typename T>
  __device__ __forceinline__ void fill(const Args<T>& a, const FlowTeam& team) {
    for (int c = threadIdx.x; c < a.ncol; c += blockDim.x) {
      n[c] = a.cptr[c + 1] - a.cptr[c];
      const int units = (n[c] + a.rows - 1) / a.rows, rank = team.rank(), size = team.size();
      mine[c] = rank < units ? (units - rank + size - 1) / size : 0;
    }
    __syncthreads();
  }
};

// One sweep, a block's units in colour order to its warps in turn.  Lane
// groups without a contact repeat the unit's first one without storing it.
template <typename T>
__device__ __forceinline__ void flow_sweep(const Args<T>& a, FlowReactions<T>& fx, const FlowTable& tab, T v[2],
                                           FlowTeam& team) {
  constexpr int L = sizeof(T) == sizeof(double) ? 2 : 1;
  const int lane = threadIdx.x & 31, comp = L == 2 ? lane & 1 : 0, i = lane / L, nw = blockDim.x >> 5;
  int e = threadIdx.x >> 5;  // the warp's next unit among the block's
  for (int c = 0; c < a.ncol; c++) {
    const int n = tab.n[c], mine = tab.mine[c];
    for (; e < mine; e += nw) {
      const int k0 = (team.rank() + e * team.size()) * a.rows;
      const bool act = i < a.rows && k0 + i < n;
      const int k = act ? k0 + i : k0;
      Row<T> row;
      load_row(a, c, k, comp, row);
      if constexpr (L == 2) {
        double dx, pn;
        contact64(a, fx, k, comp, act, row, dx, pn, team);
        if (act) {
          v[0] += dx * dx;
          v[1] += pn * pn;
        }
      } else {
        float x0, x1, P[2];
        contact32(a, fx, k, act, row, x0, x1, P, team);
        if (act) {
          v[0] += x0 * x0 + x1 * x1;
          v[1] += P[0] * P[0] + P[1] * P[1];
        }
      }
    }
    e -= mine;
  }
  if (__syncthreads_or(fx.failed)) team.give_up();
}

// Bring the FP64 reactions into the sweep's copy (replica or FP32 copy in
// HBM); the cluster barrier keeps other blocks from writing into a copy
// before it is filled.
template <typename T, bool REP, typename Team>
__device__ __forceinline__ Reactions<T, REP> open_reactions(const Args<T>& a, typename Vec2<T>::type* smem,
                                                            Team& team) {
  using V = typename Vec2<T>::type;
  Reactions<T, REP> rx{smem, a.rw};
  const double2* r = reinterpret_cast<const double2*>(a.r);
  if (REP) {
    for (int j = threadIdx.x; j < a.nc; j += blockDim.x) {
      const double2 x = __ldcg(r + j);
      V v;
      v.x = (T)x.x;
      v.y = (T)x.y;
      smem[j] = v;
    }
    team.sync_all();
  } else if (sizeof(T) != sizeof(double)) {
    const int g0 = team.rank() * blockDim.x + threadIdx.x, G = team.size() * blockDim.x;
    for (int j = g0; j < a.nc; j += G) {
      const double2 x = __ldcg(r + j);
      V v;
      v.x = (T)x.x;
      v.y = (T)x.y;
      __stcg(reinterpret_cast<V*>(a.rw) + j, v);
    }
    team.sync_all();
  }
  return rx;
}

// Write the sweep's copy back to the FP64 reactions (each block its own
// contacts), then hold every block until no other may still read its
// shared memory.
template <typename T, bool REP, typename Team>
__device__ __forceinline__ void close_reactions(const Args<T>& a, const Reactions<T, REP>& rx, Team& team) {
  if (REP || sizeof(T) != sizeof(double)) {
    const int g0 = team.rank() * blockDim.x + threadIdx.x, G = team.size() * blockDim.x;
    for (int p = g0; p < a.nc; p += G) {
      const typename Vec2<T>::type x = rx.get(p);
      __stcg(reinterpret_cast<double2*>(a.r) + p, make_double2((double)x.x, (double)x.y));
    }
  }
  team.sync_all();
}

// All sweeps of one problem (or of one precision phase of it) in one launch
// of one thread-block cluster or one cooperative grid (the Team).  A colour's
// contacts are spread over the team's threads, one a thread in FP32 and one a
// pair of threads in FP64 (contact k, k + G, ... for place k of G: a contact
// always lands on the same block, so its W row stays in that SM's L1).  What
// bounds a colour is its dependent chain: the rows are stored coalesced
// (read by rows, each lane touched its own lines and a colour of 5,000
// contacts queued on the L1's tags) and loaded before the barrier that
// releases the colour; the light-error terms are summed behind the barrier's
// arrival; above 64 contacts a colour the sweeps go as dataflow (above).  By
// colours, granular problems, us a sweep before and after: FP64 37.0 and 24.4
// at 367 contacts, 48.9 and 32.0 at 7,002, 74.7 and 32.1 at 28,008; FP32 12.0
// and 10.2, 16.2 and 14.4, 25.8 and 19.8.  The hardware cluster barrier
// (release / acquire) separates colours, the barrier of the error reduction
// closing the last one, and the convergence logic runs on the device with the
// same bits in every block.
// The light error's |r|^2 is summed over the new reactions as they are made
// (each contact is updated once per sweep, so it is |r|^2 after the sweep).
// A phase that follows another starts its sweep count, budget and trace
// where the previous one stopped (read from the device, no host round trip).
template <typename T, bool REP, typename Team>
__global__ void __launch_bounds__(Team::flow ? 256 : NT_MAX, 1) k_fc2d_nsgs(const Args<T> a) {
  using V = typename Vec2<T>::type;
  extern __shared__ __align__(16) unsigned char dsm[];
  V* rsm = reinterpret_cast<V*>(dsm);
  __shared__ Reduce<T> R;
  Team team(a);
  if (threadIdx.x == 0) R.calls = 0;
  __syncthreads();
  Reactions<T, REP> rx{nullptr, a.rw};
  FlowReactions<T> fx{};
  __shared__ typename std::conditional<Team::flow, FlowTable, char>::type tab;
  if constexpr (Team::flow) {
    tab.fill(a, team);
    fx = open_flow(a, team);
  } else {
    rx = open_reactions<T, REP>(a, rsm, team);
  }
  const int g0 = team.rank() * blockDim.x + threadIdx.x, G = team.size() * blockDim.x;
  const bool lead = team.rank() == 0 && threadIdx.x == 0;
  const int done = a.before ? (int)a.before[0] : 0;
  const int budget = a.max_iter - done;
  T tolerance = (T)a.tol, err = (T)INFINITY, best = (T)INFINITY;
  int iter = 0, not_conv = 1, since_best = 0;
  Row<T> row;
  if constexpr (!Team::flow && !Team::alone) {
    const int comp = sizeof(T) == sizeof(double) ? g0 & 1 : 0, k = sizeof(T) == sizeof(double) ? g0 >> 1 : g0;
    if (k < a.cptr[1] - a.cptr[0]) load_row(a, 0, k, comp, row);
  }
  while (iter < budget && not_conv) {
    ++iter;
    T v[2] = {0, 0};
    if constexpr (Team::flow) {
      fx.sweep = iter;
      flow_sweep(a, fx, tab, v, team);
    } else if constexpr (Team::alone) {
      sweep_alone(a, rx, g0, G, v, team);
    } else {
      sweep_colours(a, rx, g0, G, row, v, team);
    }
    if constexpr (sizeof(T) == sizeof(double))
      team_sum2(v, R, team, a.part);
    else if constexpr (Team::flow)
      flow_sum<2>(v, R, team, a.part);
    else
      team_sum<2>(v, R, team, a.part);
    if constexpr (Team::grid)
      if (team.dead()) return;
    if constexpr (sizeof(T) == sizeof(double)) {
      const double nr = fc3dgpu::ie_sqrt(v[1]);
      err = fc3dgpu::ie_sqrt(v[0]);
      if (fabs(nr) > DBL_EPSILON) err = fc3dgpu::ie_div(err, nr);
    } else {
      err = sqrt(v[0]);
      const T nr = sqrt(v[1]);
      if (fabs(nr) > (T)DBL_EPSILON) err /= nr;
    }
    if (a.trace && lead && done + iter <= TRACE_CAP) a.trace[done + iter - 1] = (double)err;
    if (a.mode == FP32_PHASE) {
      if (err < best) {
        best = err;
        since_best = 0;
      } else {
        since_best++;
      }
      not_conv = !(err < (T)a.switch_tol) && since_best < a.stall;
    } else if (a.mode == LIGHT) {
      not_conv = !(err < tolerance);  // determine_convergence (fc2d_nsgs.c:147-162)
    } else if (a.mode == FULL_FINAL && err < tolerance) {
      // determine_convergence_with_full_final (fc2d_nsgs.c:187-228)
      not_conv = 0;
      if constexpr (sizeof(T) == sizeof(double)) {
        const double full = full_error<REP>(a, rx, R, team);
        if constexpr (Team::grid)
          if (team.dead()) return;
        if (full > a.tol) {
          tolerance = err / full * a.tol;
          not_conv = 1;
        }
      }
    }
  }
  double final_err = (double)err;
  if constexpr (sizeof(T) == sizeof(double)) {
    if (a.mode == FULL_FINAL) {
      final_err = full_error<REP>(a, rx, R, team);
      not_conv = !(final_err < a.tol);
    } else if (a.mode == NO_EVAL) {
      final_err = INFINITY;  // no branch of the sweep loop evaluates an error (fc2d_nsgs.c:438-448)
      not_conv = 1;
    }
  }
  if constexpr (Team::grid)
    if (team.dead()) return;
  if (lead) {
    a.out[0] = done + iter;
    a.out[1] = final_err;
    a.out[2] = not_conv;
    a.out[3] = (double)err;
  }
  close_reactions<T, REP>(a, rx, team);
}

template <bool REP, typename Team>
__global__ void __launch_bounds__(NT_MAX, 1) k_fc2d_error(const Args<double> a) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ Reduce<double> R;
  Team team(a);
  if (threadIdx.x == 0) R.calls = 0;
  __syncthreads();
  const Reactions<double, REP> rx = open_reactions<double, REP>(a, reinterpret_cast<double2*>(dsm), team);
  const double e = full_error<REP>(a, rx, R, team);
  if (team.rank() == 0 && threadIdx.x == 0) a.out[1] = e;
  close_reactions<double, REP>(a, rx, team);
}

}  // namespace fc2dgpu

// ---------------------------------------------------------------------------
// Context (C-ABI)
// ---------------------------------------------------------------------------
using namespace fc2dgpu;

// A launch: a cluster of cs blocks, or a cooperative grid of `blocks`; the
// reactions in HBM or replicated in shared memory.
struct Shape {
  bool grid = false, rep = false, flow = false;
  bool alone = false;  // FP64: a contact a lane
  int cs = 1, nt = 128, blocks = 1, rows = 1;
};

// Arrays side by side in one allocation; from base nullptr only their length.
struct Pool {
  char* base;
  size_t at;
  template <typename T>
  void take(T*& p, size_t n) {
    p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += (sizeof(T) * n + 255) / 256 * 256;
  }
};

// What a problem sends to the device (Args), with FP32 copies for the first
// phase of a mixed-precision solve.  Filled on the host in one buffer of the
// device's layout, so that it takes one copy.
struct Uploaded {
  int *cptr = nullptr, *rp = nullptr, *col = nullptr, *dpos = nullptr, *sp = nullptr;
  int2* slab = nullptr;
  double *W = nullptr, *det = nullptr, *q = nullptr, *mu = nullptr;
  float *det32 = nullptr, *q32 = nullptr, *mu32 = nullptr;
  void carve(Pool& pool, int nc, size_t nnzb, int ncol, int nslab) {
    pool.take(cptr, ncol + 1);
    pool.take(rp, (size_t)nc + 1);
    pool.take(col, nnzb);
    pool.take(dpos, nc);
    pool.take(sp, ncol + 1);
    pool.take(slab, nslab);
    pool.take(W, 4 * nnzb);
    pool.take(det, nc);
    pool.take(q, 2 * (size_t)nc);
    pool.take(mu, nc);
    pool.take(det32, nc);
    pool.take(q32, 2 * (size_t)nc);
    pool.take(mu32, nc);
  }
};

struct fc2dgpu_ctx : Uploaded {
  int device = 0;
  int cs_req = 0, nt_req = 0;  // launch shape asked for (0 = automatic)
  int rep_req = 0;             // reactions: 0 automatic, 1 in HBM, 2 replicated in shared memory
  Shape s32, s64;              // launch shapes of the current problem's FP32 and FP64 kernels
  int max_colour = 0;          // contacts in the largest colour
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  int nc = 0, ncol = 0;
  bool singular = false;
  double norm_q = 0.0;
  std::vector<int> perm, iperm, colour;
  void* pool = nullptr;  // holds the arrays of Uploaded and the next seven
  size_t pool_bytes = 0;
  int* scol = nullptr;
  double *sW = nullptr, *D = nullptr, *r = nullptr, *u = nullptr;
  float *sW32 = nullptr, *D32 = nullptr, *r32 = nullptr;
  double* rs = nullptr;  // stamped reactions of the dataflow, of either precision (a symmetric block pattern)
  void* work = nullptr;  // holds the next four
  double *trace = nullptr, *out = nullptr, *part = nullptr;
  unsigned* arrived = nullptr;
  unsigned long long spin = SPIN;
  int precision = 1;          // 0 FP32 sweeps + FP64 polish, 1 FP64 sweeps only
  double switch_tol = 0.0;    // FP32 phase stops below this light error (0: max(tol, 1e-6))
  int stall = 64;             // ... or after this many sweeps without a new lowest error
  int sweeps32 = 0, sweeps64 = 0;
  int trace_len = 0;
};

#define K2(x)                                                                             \
  do {                                                                                    \
    cudaError_t e_ = (x);                                                                 \
    if (e_ != cudaSuccess) {                                                              \
      fc3dgpu_set_error("%s:%d %s: %s", __FILE__, __LINE__, #x, cudaGetErrorString(e_)); \
      return NUMERICS_ERR_UNKNOWN;                                                        \
    }                                                                                     \
  } while (0)

// Dataflow above this many contacts in the largest colour, where one block no
// longer holds it at a contact a thread: with 41 contacts a sweep takes 12.6 us
// in one block and 13.5 as dataflow in FP64 (11.5 and 12.5 mixed), with 131 on a
// cluster 24.4 and 18.0 (FP32 10.2 and 7.7).
constexpr int FLOW_FROM = 64;

static void choose_shape(fc2dgpu_ctx* c);

// Whether every block (i, j) has a block (j, i), as often (the dataflow needs
// it).  On the device a row looks itself up in its neighbours' rows, so the work
// goes with the square of a row's length: for rows of up to this many blocks.
// Reading the answer back takes 40 us, in which the host looks at some thousand
// blocks (fc2dgpu_ctx_set_problem on the host and on the device, ms: 367 contacts
// 0.62 and 0.65, 3,303 0.92 and 0.87, 7,002 1.29 and 1.14).
constexpr int SYMMETRIC_ROWS = 64;
constexpr int SYMMETRIC_FROM = 8192;  // blocks

__global__ void k_one_sided(int nc, const int* __restrict__ rp, const int* __restrict__ col, int* __restrict__ one_sided) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nc) return;
  auto count = [&](int row, int of) {
    int n = 0;
    for (int k = rp[row]; k < rp[row + 1]; k++) n += col[k] == of;
    return n;
  };
  for (int k = rp[p]; k < rp[p + 1]; k++)
    if (count(col[k], p) != count(p, col[k])) *one_sided = 1;
}

// On the host for longer rows and few blocks: the columns' rows in ascending order, which a
// transposition gives, against the rows' sorted columns, which a second one
// gives.
static bool symmetric_pattern(int nc, const int* rp, const int* col) {
  auto transpose = [&](const int* p, const int* x, std::vector<int>& tp, std::vector<int>& t) {
    tp.assign(nc + 1, 0);
    for (int k = 0; k < p[nc]; k++) tp[x[k] + 1]++;
    for (int j = 0; j < nc; j++) tp[j + 1] += tp[j];
    t.resize(p[nc]);
    std::vector<int> at(tp.begin(), tp.end() - 1);
    for (int i = 0; i < nc; i++)
      for (int k = p[i]; k < p[i + 1]; k++) t[at[x[k]]++] = i;
  };
  std::vector<int> tp, t, sp, sorted;
  transpose(rp, col, tp, t);
  if (!std::equal(tp.begin(), tp.end(), rp)) return false;
  transpose(tp.data(), t.data(), sp, sorted);
  return t == sorted;
}

static void free_problem(fc2dgpu_ctx* c) {
  if (c->pool) cudaFree(c->pool);
  c->pool = nullptr;
  c->pool_bytes = 0;
  c->nc = 0;
}

extern "C" void fc2dgpu_ctx_destroy(fc2dgpu_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  free_problem(c);
  if (c->work) cudaFree(c->work);
  for (auto& e : c->ev)
    if (e) cudaEventDestroy(e);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

extern "C" fc2dgpu_ctx* fc2dgpu_ctx_create(int device) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
    cudaGetLastError();
    fc3dgpu_set_error("fc2dgpu_ctx_create: no CUDA device %d", device);
    return nullptr;
  }
  if (cudaSetDevice(device) != cudaSuccess) {
    fc3dgpu_set_error("fc2dgpu_ctx_create: cudaSetDevice(%d) failed", device);
    return nullptr;
  }
  fc2dgpu_ctx* c = new fc2dgpu_ctx();
  c->device = device;
  auto carve = [&](Pool p) {
    p.take(c->trace, TRACE_CAP);
    p.take(c->out, 9);
    p.take(c->part, 2 * GRID_MAX * 4);
    p.take(c->arrived, 1);
    return p.at;
  };
  bool ok = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaEventCreate(&c->ev[0]) == cudaSuccess && cudaEventCreate(&c->ev[1]) == cudaSuccess &&
            cudaMalloc(&c->work, carve(Pool{nullptr, 0})) == cudaSuccess;
  if (ok) {
    carve(Pool{static_cast<char*>(c->work), 0});
    ok = cudaMemsetAsync(c->out, 0, sizeof(double) * 9, c->stream) == cudaSuccess;
  }
  if (!ok) {
    fc3dgpu_set_error("fc2dgpu_ctx_create: set-up failed (%s)", cudaGetErrorString(cudaGetLastError()));
    fc2dgpu_ctx_destroy(c);
    return nullptr;
  }
  return c;
}

// The sweeps' coalesced copy of the rows (Args::slab), one thread a row.  Built
// here from the uploaded rows: on the host, with an upload each in both
// precisions, the layout took 12.7 ms at 70,020 contacts for 6.4 now (7,002: 1.68
// and 1.17).
__global__ void k_slab_rows(int ncol, const int* __restrict__ cptr, const int* __restrict__ sp,
                            const int2* __restrict__ slab, const int* __restrict__ rp, const int* __restrict__ col,
                            const int* __restrict__ dpos, const double* __restrict__ W, int* __restrict__ scol,
                            double* __restrict__ sW, float* __restrict__ sW32, double* __restrict__ D,
                            float* __restrict__ D32) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= sp[ncol]) return;
  int c = 0;
  while (sp[c + 1] <= b) c++;
  const int p = cptr[c] + (b - sp[c]) * 32 + lane;
  const int2 s = slab[b];
  auto put = [&](size_t e, int j, double a00, double a01, double a10, double a11) {
    scol[e] = j;
    reinterpret_cast<double2*>(sW)[2 * e] = make_double2(a00, a01);
    reinterpret_cast<double2*>(sW)[2 * e + 1] = make_double2(a10, a11);
    reinterpret_cast<float4*>(sW32)[e] = make_float4((float)a00, (float)a01, (float)a10, (float)a11);
  };
  int t = 0;
  if (p < cptr[c + 1]) {
    for (int k = rp[p]; k < rp[p + 1]; k++) {
      const double* w = W + 4 * (size_t)k;
      if (col[k] != p) put((size_t)(s.x + t++) * 32 + lane, col[k], w[0], w[2], w[1], w[3]);
    }
    const double* d = W + 4 * (size_t)(rp[p] + dpos[p]);
    for (int i = 0; i < 4; i++) {
      D[4 * (size_t)p + i] = d[i];
      D32[4 * (size_t)p + i] = (float)d[i];
    }
  }
  for (; t < s.y; t++) put((size_t)(s.x + t) * 32 + lane, -1, 0.0, 0.0, 0.0, 0.0);
}

extern "C" int fc2dgpu_ctx_set_problem(fc2dgpu_ctx* c, int nc, const int64_t* rowptr, const int64_t* colidx,
                                       const double* blocks, const double* q, const double* mu, int colour_kind) {
  if (!c || nc <= 0 || !rowptr || !colidx || !blocks || !q || !mu) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: invalid argument");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  const int64_t nnzb = rowptr[nc];
  if (rowptr[0] != 0 || nnzb < nc || nnzb > INT32_MAX) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: bad row pointer");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  std::vector<int> dposo(nc, -1);
  for (int i = 0; i < nc; i++) {
    if (rowptr[i + 1] < rowptr[i]) {
      fc3dgpu_set_error("fc2dgpu_ctx_set_problem: row pointer decreases at %d", i);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
    for (int64_t k = rowptr[i]; k < rowptr[i + 1]; k++) {
      if (colidx[k] < 0 || colidx[k] >= nc) {
        fc3dgpu_set_error("fc2dgpu_ctx_set_problem: column index %lld out of range", (long long)colidx[k]);
        return NUMERICS_ERR_INVALID_ARGUMENT;
      }
      if (colidx[k] == i && dposo[i] < 0) dposo[i] = (int)(k - rowptr[i]);
    }
    if (dposo[i] < 0) {
      fc3dgpu_set_error("fc2dgpu_ctx_set_problem: contact %d has no diagonal block", i);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
  }
  for (int i = 0; i < nc; i++)
    if (!(mu[i] >= 0.0) || isinf(mu[i])) {
      fc3dgpu_set_error("fc2dgpu_ctx_set_problem: mu[%d] = %g is not a friction coefficient", i, mu[i]);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
  // colouring of the conflict graph (the device Jones-Plassmann colouring)
  std::vector<int32_t> colour(nc);
  const int ncol = fc3dgpu_colour(nc, rowptr, colidx, colour_kind, colour.data());
  if (ncol < 0) return ncol;
  if (ncol > MAXC) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: %d colours (at most %d)", ncol, MAXC);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (cudaSetDevice(c->device) != cudaSuccess) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: cudaSetDevice failed");
    return NUMERICS_ERR_UNKNOWN;
  }
  c->nc = 0;
  c->colour.assign(colour.begin(), colour.end());
  c->perm.resize(nc);
  std::iota(c->perm.begin(), c->perm.end(), 0);
  std::stable_sort(c->perm.begin(), c->perm.end(), [&](int x, int y) { return colour[x] < colour[y]; });
  c->iperm.resize(nc);
  for (int p = 0; p < nc; p++) c->iperm[c->perm[p]] = p;
  // the rows' slabs by colour (Args::slab)
  std::vector<int> size(ncol, 0);
  for (int i = 0; i < nc; i++) size[colour[i]]++;
  c->max_colour = *std::max_element(size.begin(), size.end());
  int nslab = 0;
  for (int n : size) nslab += (n + 31) / 32;
  Uploaded h;
  Pool measure = {nullptr, 0};
  h.carve(measure, nc, nnzb, ncol, nslab);
  const size_t sent = measure.at;
  const std::unique_ptr<char[]> host(new (std::nothrow) char[sent]);
  if (!host) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: out of host memory");
    return NUMERICS_ERR_MEMORY;
  }
  Pool pool = {host.get(), 0};
  h.carve(pool, nc, nnzb, ncol, nslab);
  h.cptr[0] = h.sp[0] = 0;
  for (int k = 0; k < ncol; k++) {
    h.cptr[k + 1] = h.cptr[k] + size[k];
    h.sp[k + 1] = h.sp[k] + (size[k] + 31) / 32;
  }
  bool singular = false;
  size_t slots = 0;
  int longest = 0;
  h.rp[0] = 0;
  for (int k = 0; k < ncol; k++)
    for (int b = h.sp[k]; b < h.sp[k + 1]; b++) {
      int most = 0;  // blocks off the diagonal of the slab's longest row
      for (int p = h.cptr[k] + 32 * (b - h.sp[k]); p < std::min(h.cptr[k] + 32 * (b + 1 - h.sp[k]), h.cptr[k + 1]); p++) {
        const int i = c->perm[p];
        const int64_t k0 = rowptr[i], k1 = rowptr[i + 1];
        int off = 0;
        for (int64_t s = k0; s < k1; s++) {
          const size_t at = (size_t)h.rp[p] + (size_t)(s - k0);
          h.col[at] = c->iperm[colidx[s]];
          off += colidx[s] != i;
          for (int e = 0; e < 4; e++) h.W[4 * at + e] = blocks[4 * s + e];
        }
        h.rp[p + 1] = h.rp[p] + (int)(k1 - k0);
        longest = std::max(longest, (int)(k1 - k0));
        most = std::max(most, off);
        h.dpos[p] = dposo[i];
        const double* d = &blocks[4 * (k0 + dposo[i])];
        h.det[p] = d[0] * d[3] - d[1] * d[2];
        // of the rounded block, in FP32
        h.det32[p] = (float)d[0] * (float)d[3] - (float)d[1] * (float)d[2];
        if (h.det[p] < DBL_EPSILON) singular = true;
        for (int e = 0; e < 2; e++) {
          h.q[2 * (size_t)p + e] = q[2 * (size_t)i + e];
          h.q32[2 * (size_t)p + e] = (float)q[2 * (size_t)i + e];
        }
        h.mu[p] = mu[i];
        h.mu32[p] = (float)mu[i];
      }
      h.slab[b] = make_int2((int)slots, most);
      slots += most;
    }
  double s2 = 0.0;
  for (int64_t k = 0; k < 2LL * nc; k++) s2 += q[k] * q[k];
  c->norm_q = sqrt(s2);
  // the device's arrays, in the allocation of the problem before where that is
  // of about the size
  int* one_sided = nullptr;
  const bool look = c->max_colour > FLOW_FROM;  // for dataflow
  auto carve = [&](Pool p) {
    c->carve(p, nc, nnzb, ncol, nslab);
    p.take(c->scol, slots * 32);
    p.take(c->sW, slots * 128);
    p.take(c->sW32, slots * 128);
    p.take(c->D, 4 * (size_t)nc);
    p.take(c->D32, 4 * (size_t)nc);
    p.take(c->rs, look ? 4 * (size_t)nc : 0);
    // zero from here on
    p.take(c->r, 2 * (size_t)nc);
    p.take(c->u, 2 * (size_t)nc);
    p.take(c->r32, 2 * (size_t)nc);
    p.take(one_sided, 1);
    return p.at;
  };
  const size_t bytes = carve(Pool{nullptr, 0});
  cudaError_t e = cudaSuccess;
  if (bytes > c->pool_bytes || bytes < c->pool_bytes / 2) {
    free_problem(c);
    e = cudaMalloc(&c->pool, bytes);
    c->pool_bytes = e == cudaSuccess ? bytes : 0;
    if (e != cudaSuccess) c->pool = nullptr;
  }
  int mismatch = 0;
  const bool on_device = longest <= SYMMETRIC_ROWS && nnzb >= SYMMETRIC_FROM;
  if (e == cudaSuccess) {
    cudaStream_t st = c->stream;
    carve(Pool{static_cast<char*>(c->pool), 0});
    e = cudaMemcpyAsync(c->pool, host.get(), sent, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->r, 0, (size_t)((char*)(one_sided + 1) - (char*)c->r), st);
    k_slab_rows<<<(nslab * 32 + 255) / 256, 256, 0, st>>>(ncol, c->cptr, c->sp, c->slab, c->rp, c->col, c->dpos, c->W,
                                                          c->scol, c->sW, c->sW32, c->D, c->D32);
    if (look && on_device) {
      k_one_sided<<<(nc + 255) / 256, 256, 0, st>>>(nc, c->rp, c->col, one_sided);
      if (e == cudaSuccess) e = cudaMemcpyAsync(&mismatch, one_sided, sizeof(int), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    const cudaError_t done = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = done;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    free_problem(c);
    fc3dgpu_set_error("fc2dgpu_ctx_set_problem: %s", cudaGetErrorString(e));
    return NUMERICS_ERR_UNKNOWN;
  }
  if (!look || mismatch || (!on_device && !symmetric_pattern(nc, h.rp, h.col))) c->rs = nullptr;
  c->nc = nc;
  c->ncol = ncol;
  c->singular = singular;
  choose_shape(c);
  return 0;
}

extern "C" int fc2dgpu_ctx_set_q_mu(fc2dgpu_ctx* c, const double* q, const double* mu) {
  if (!c || !q || !mu || c->nc == 0) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_q_mu: invalid argument");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  const int nc = c->nc;
  for (int i = 0; i < nc; i++)
    if (!(mu[i] >= 0.0) || isinf(mu[i])) {
      fc3dgpu_set_error("fc2dgpu_ctx_set_q_mu: mu[%d] = %g is not a friction coefficient", i, mu[i]);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
  std::vector<double> qp(2 * (size_t)nc), mup(nc);
  double s2 = 0.0;
  for (int64_t k = 0; k < 2LL * nc; k++) s2 += q[k] * q[k];
  for (int i = 0; i < nc; i++) {
    const size_t p = (size_t)c->iperm[i];
    qp[2 * p] = q[2 * i];
    qp[2 * p + 1] = q[2 * i + 1];
    mup[p] = mu[i];
  }
  K2(cudaSetDevice(c->device));
  K2(copy_to_device(c->q, qp.data(), sizeof(double) * qp.size(), c->stream));
  K2(copy_to_device(c->mu, mup.data(), sizeof(double) * mup.size(), c->stream));
  const std::vector<float> q32(qp.begin(), qp.end()), mu32(mup.begin(), mup.end());
  K2(copy_to_device(c->q32, q32.data(), sizeof(float) * q32.size(), c->stream));
  K2(copy_to_device(c->mu32, mu32.data(), sizeof(float) * mu32.size(), c->stream));
  c->norm_q = sqrt(s2);
  return 0;
}

extern "C" int fc2dgpu_ctx_set_r(fc2dgpu_ctx* c, const double* r) {
  if (!c || !r || c->nc == 0) return NUMERICS_ERR_INVALID_ARGUMENT;
  std::vector<double> rp(2 * (size_t)c->nc);
  for (int i = 0; i < c->nc; i++) {
    rp[2 * (size_t)c->iperm[i]] = r[2 * i];
    rp[2 * (size_t)c->iperm[i] + 1] = r[2 * i + 1];
  }
  K2(cudaSetDevice(c->device));
  K2(copy_to_device(c->r, rp.data(), sizeof(double) * rp.size(), c->stream));
  return 0;
}

// Launch shape: a cluster of up to CS_MAX blocks.  The sweep is bound by
// the latency of each colour's dependent chain (loads, FP64 divisions,
// barrier) and by the FP64 pipes (about two FP64 operations per clock per SM
// on this part), so a colour with more contacts is spread over more SMs;
// blocks of up to NT_MAX threads keep each thread on one or two contacts per
// colour.  The reactions are replicated in every block's shared memory when
// 16 bytes per contact fit (up to about 13,000 contacts), else kept in HBM.
static cudaLaunchConfig_t config(fc2dgpu_ctx* c, int cs, int nt, size_t smem, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(cs, 1, 1);
  cfg.blockDim = dim3(nt, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

static size_t rep_bytes(const fc2dgpu_ctx* c) { return sizeof(double2) * (size_t)c->nc; }

// Kernel attributes a launch of this shape needs (cluster size above the
// portable 8, dynamic shared memory above 48 KiB).
template <typename K>
static cudaError_t prepare(K kernel, int cs, size_t smem) {
  cudaError_t e = cudaSuccess;
  if (cs > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess && smem > 0) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e;
}

// Whether a cluster of cs blocks of nt threads of the sweep kernel (the
// larger of the two kernels) can be resident on this device.
static bool cluster_fits(fc2dgpu_ctx* c, int cs, int nt, bool rep) {
  const size_t smem = rep ? rep_bytes(c) : 0;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = config(c, cs, nt, smem, attr);
  int n = 0;
  cudaError_t e = rep ? prepare(k_fc2d_nsgs<double, true, ClusterTeam>, cs, smem) : prepare(k_fc2d_nsgs<double, false, ClusterTeam>, cs, smem);
  if (e == cudaSuccess)
    e = rep ? cudaOccupancyMaxActiveClusters(&n, k_fc2d_nsgs<double, true, ClusterTeam>, &cfg)
            : cudaOccupancyMaxActiveClusters(&n, k_fc2d_nsgs<double, false, ClusterTeam>, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n > 0;
}

// A colour with more contacts than a full cluster has threads (16 x 512)
// goes to a cooperative grid over every SM instead (a barrier over all of them
// instead of the cluster's 0.3 us; the FP64 pipes of all SMs).
constexpr int GRID_FROM = CS_MAX * NT_MAX;
// In FP64 the FP64 units of a cluster's SMs bound a colour from far fewer
// contacts (cluster and grid, us a sweep: 41.3 and 32.0 with 2,401 contacts in
// the largest colour, 54.1 and 32.1 with 4,828; with 514 the cluster's 25.6
// against 37.8 on the grid).
constexpr int GRID64_FROM = 1000;

// Contacts of the largest colour a thread from which FP64 contacts are one
// lane's.  ms for 40 sweeps on two lanes and on one, by contacts a thread: 1.2
// (2,048 threads) 2.25 and 2.47, 2.5 (77,824) 7.21 and 7.45; 6.2 (77,824) 15.0 and
// 14.7, 4.7 (512) 4.48 and 3.78, 4.7 (2,048) 6.17 and 5.63, 12 (8,192) 24.7 and 22.2,
// 19 (128) 14.7 and 11.4, 76 (128) 60.1 and 45.3.
constexpr int ALONE_FROM = 4;

static Shape grid_shape(fc2dgpu_ctx* c, int nt, int lanes) {
  Shape s;
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  // FP64: the largest colour over all SMs, one pass each
  if (nt <= 0) nt = lanes == 1 ? 256 : std::min(256, std::max(32, (lanes * c->max_colour / std::max(sms, 1) + 31) / 32 * 32));
  nt = std::min(std::max(nt / 32 * 32, 32), NT_MAX);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fc2d_nsgs<double, false, GridTeam>, nt, 0);
  const int resident = std::max(1, std::min(per_sm * sms, GRID_MAX));
  s.grid = true;
  s.nt = nt;
  s.blocks = std::max(1, std::min((lanes * c->max_colour + nt - 1) / nt, resident));
  return s;
}

// Units of as few contacts as give every SM quarter one of an average colour;
// a block an SM, of eight warps where the largest colour has more units than
// quarters, else of four.
static Shape flow_shape(fc2dgpu_ctx* c, int most) {
  Shape s;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  const long long quarters = 4LL * c->ncol * sms;
  s.grid = s.flow = true;
  s.rows = (int)std::min<long long>(most, std::max(1LL, (c->nc + quarters - 1) / quarters));
  const int units = (c->max_colour + s.rows - 1) / s.rows;
  s.nt = units > 4 * sms ? 256 : 128;
  s.blocks = std::max(1, std::min((units + s.nt / 32 - 1) / (s.nt / 32), std::min(sms, GRID_MAX)));
  return s;
}

static void choose_blocks(fc2dgpu_ctx* c);
static void choose_shape(fc2dgpu_ctx* c) {
  if (c->rs && c->cs_req == 0 && c->nt_req == 0 && c->rep_req == 0) {
    c->s32 = flow_shape(c, 32);
    c->s64 = flow_shape(c, 16);
    return;
  }
  choose_blocks(c);
  c->s64.alone = c->max_colour > (long long)ALONE_FROM * (c->s64.grid ? c->s64.blocks : c->s64.cs) * c->s64.nt;
}

static void choose_blocks(fc2dgpu_ctx* c) {
  if (c->cs_req < 0 || (c->cs_req == 0 && c->rep_req != 2 && c->max_colour > GRID_FROM)) {
    c->s32 = grid_shape(c, c->nt_req, 1);
    c->s64 = c->cs_req < 0 ? c->s32 : grid_shape(c, c->nt_req, 2);
    return;
  }
  Shape s;
  int cs = c->cs_req, nt = c->nt_req;
  if (cs <= 0) {
    const int want = (c->max_colour + 63) / 64;  // about 64 contacts per SM and colour
    cs = 1;
    while (cs < want && cs < CS_MAX) cs *= 2;
  }
  cs = std::min(std::max(cs, 1), CS_MAX);
  if (nt <= 0) nt = std::min(NT_MAX, std::max(32, ((c->max_colour + cs - 1) / cs + 31) / 32 * 32));
  nt = std::min(std::max(nt / 32 * 32, 32), NT_MAX);
  // a replicated copy costs one distributed shared-memory store per block of
  // the cluster for each update: it pays for clusters of up to 4 blocks
  bool rep = c->rep_req == 2 || (c->rep_req == 0 && rep_bytes(c) <= REP_MAX_BYTES && cs <= 4);
  if (rep && c->rep_req == 0 && !cluster_fits(c, cs, nt, true)) rep = false;
  if (c->cs_req <= 0)
    while (cs > 1 && !cluster_fits(c, cs, nt, rep)) cs /= 2;
  s.cs = cs;
  s.nt = nt;
  s.rep = rep;
  c->s32 = c->s64 = s;
  // FP64 takes two threads a contact
  if (c->nt_req == 0) {
    const int nt2 = std::min(NT_MAX, 2 * nt);
    if (cluster_fits(c, cs, nt2, rep)) c->s64.nt = nt2;
  }
  if (c->cs_req == 0 && c->rep_req == 0 && c->max_colour > GRID64_FROM) c->s64 = grid_shape(c, c->nt_req, 2);
}

template <typename K, typename A>
static cudaError_t launch_grid(fc2dgpu_ctx* c, const Shape& s, K kernel, const A& a) {
  void* params[] = {(void*)&a};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3(s.blocks), dim3(s.nt), params, 0, c->stream);
}

template <typename K, typename A>
static cudaError_t launch(fc2dgpu_ctx* c, const Shape& s, K kernel, const A& a, size_t smem) {
  cudaError_t e = prepare(kernel, s.cs, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = config(c, s.cs, s.nt, smem, attr);
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

extern "C" int fc2dgpu_ctx_set_launch(fc2dgpu_ctx* c, int cluster_blocks, int threads, int reactions) {
  if (!c || cluster_blocks < -1 || cluster_blocks > CS_MAX || threads < 0 || threads > NT_MAX ||
      (threads && threads % 32) || reactions < 0 || reactions > 2 || (cluster_blocks < 0 && reactions == 2)) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_launch: cluster of 0..%d blocks (-1: cooperative grid, reactions in HBM), 0 or "
                      "32..%d threads (multiple of 32), reactions 0, 1 or 2", CS_MAX, NT_MAX);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (reactions == 2 && (c->nc == 0 || rep_bytes(c) > REP_MAX_BYTES)) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_launch: %d contacts do not fit a shared-memory copy", c->nc);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (cluster_blocks > 0) {
    const bool rep = reactions == 2 || (reactions == 0 && c->nc > 0 && rep_bytes(c) <= REP_MAX_BYTES);
    if (cudaSetDevice(c->device) != cudaSuccess || !cluster_fits(c, cluster_blocks, threads ? threads : NT_MAX, rep)) {
      fc3dgpu_set_error("fc2dgpu_ctx_set_launch: a cluster of %d blocks of %d threads does not fit this device",
                        cluster_blocks, threads ? threads : NT_MAX);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
  }
  c->cs_req = cluster_blocks;
  c->nt_req = threads;
  c->rep_req = reactions;
  if (c->nc > 0) choose_shape(c);
  return 0;
}

extern "C" int fc2dgpu_ctx_launch_shape(fc2dgpu_ctx* c, int* cluster_blocks, int* threads, int* reactions) {
  if (!c) return NUMERICS_ERR_INVALID_ARGUMENT;
  const Shape& s = c->precision == 0 ? c->s32 : c->s64;
  if (cluster_blocks) *cluster_blocks = s.grid ? -s.blocks : s.cs;
  if (threads) *threads = s.nt;
  if (reactions) *reactions = s.rep ? 2 : 1;
  return 0;
}

static Args<double> args64(const fc2dgpu_ctx* c) {
  Args<double> a;
  memset(&a, 0, sizeof(a));
  a.nc = c->nc;
  a.ncol = c->ncol;
  a.cptr = c->cptr;
  a.rp = c->rp;
  a.col = c->col;
  a.dpos = c->dpos;
  a.W = c->W;
  a.sp = c->sp;
  a.slab = c->slab;
  a.scol = c->scol;
  a.sW = c->sW;
  a.D = c->D;
  a.det = c->det;
  a.q = c->q;
  a.mu = c->mu;
  a.r = c->r;
  a.rw = c->r;
  a.u = c->u;
  a.norm_q = c->norm_q;
  a.trace = c->trace;
  a.out = c->out;
  a.part = c->part;
  a.rs = c->rs;
  a.arrived = c->arrived;
  a.fail = c->out + 8;
  a.spin = c->spin;
  return a;
}

static Args<float> args32(const fc2dgpu_ctx* c) {
  Args<float> a;
  memset(&a, 0, sizeof(a));
  a.nc = c->nc;
  a.ncol = c->ncol;
  a.cptr = c->cptr;
  a.rp = c->rp;
  a.col = c->col;
  a.dpos = c->dpos;
  a.sp = c->sp;
  a.slab = c->slab;
  a.scol = c->scol;
  a.sW = c->sW32;
  a.D = c->D32;
  a.det = c->det32;
  a.q = c->q32;
  a.mu = c->mu32;
  a.r = c->r;
  a.rw = c->r32;
  a.u = c->u;
  a.norm_q = c->norm_q;
  a.trace = c->trace;
  a.out = c->out + 4;
  a.part = c->part;
  a.rs = reinterpret_cast<float*>(c->rs);
  a.arrived = c->arrived;
  a.fail = c->out + 8;
  a.spin = c->spin;
  return a;
}

extern "C" int fc2dgpu_ctx_set_precision(fc2dgpu_ctx* c, int precision, double switch_tol, int stall_window) {
  if (!c || precision < 0 || precision > 1 || !(switch_tol >= 0.0) || stall_window < 0) {
    fc3dgpu_set_error("fc2dgpu_ctx_set_precision: precision 0 or 1, switch_tol >= 0, stall_window >= 0");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  c->precision = precision;
  c->switch_tol = switch_tol;
  c->stall = stall_window > 0 ? stall_window : 64;
  return 0;
}

extern "C" int fc2dgpu_ctx_last_sweeps(fc2dgpu_ctx* c, int* sweeps32, int* sweeps64) {
  if (!c) return NUMERICS_ERR_INVALID_ARGUMENT;
  if (sweeps32) *sweeps32 = c->sweeps32;
  if (sweeps64) *sweeps64 = c->sweeps64;
  return 0;
}

// The error of a launch whose waits gave up.
static int gave_up(fc2dgpu_ctx* c, const char* who) {
  K2(cudaMemsetAsync(c->out, 0, sizeof(double) * 9, c->stream));
  fc3dgpu_set_error("%s: a wait reached its poll limit", who);
  return NUMERICS_ERR_UNKNOWN;
}

extern "C" int fc2dgpu_ctx_spin_limit(fc2dgpu_ctx* c, unsigned long long polls) {
  if (!c) return NUMERICS_ERR_INVALID_ARGUMENT;
  c->spin = polls ? polls : SPIN;
  return 0;
}

extern "C" int fc2dgpu_ctx_compute_error(fc2dgpu_ctx* c, double norm_q, double* error) {
  if (!c || c->nc == 0 || !error) {
    fc3dgpu_set_error("fc2dgpu_ctx_compute_error: invalid argument");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  K2(cudaSetDevice(c->device));
  Args<double> a = args64(c);
  a.norm_q = norm_q;
  const Shape& s = c->s64;
  if (s.grid) K2(cudaMemsetAsync(c->arrived, 0, sizeof(unsigned), c->stream));
  K2(s.grid  ? launch_grid(c, s, k_fc2d_error<false, GridTeam>, a)
     : s.rep ? launch(c, s, k_fc2d_error<true, ClusterTeam>, a, rep_bytes(c))
             : launch(c, s, k_fc2d_error<false, ClusterTeam>, a, 0));
  double out[9];
  K2(cudaMemcpyAsync(out, c->out, sizeof(out), cudaMemcpyDeviceToHost, c->stream));
  K2(cudaStreamSynchronize(c->stream));
  if (out[8] != 0.0) return gave_up(c, "fc2dgpu_ctx_compute_error");
  *error = out[1];
  return 0;
}

extern "C" int fc2dgpu_ctx_solve(fc2dgpu_ctx* c, double tol, int max_iter, int error_evaluation, int* iters,
                                 double* error, int* info, double* ms) {
  if (!c || c->nc == 0) {
    fc3dgpu_set_error("fc2dgpu_ctx_solve: no problem");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (max_iter < 0) {
    fc3dgpu_set_error("fc2dgpu_ctx_solve: negative iteration budget");
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (c->singular) {
    // as fc2d_nsgs: a diagonal block with a determinant below DBL_EPSILON
    if (iters) *iters = 0;
    if (error) *error = INFINITY;
    if (info) *info = 1;
    if (ms) *ms = 0.0;
    c->trace_len = 0;
    return 0;
  }
  K2(cudaSetDevice(c->device));
  Args<double> a = args64(c);
  a.tol = tol;
  a.max_iter = max_iter;
  a.mode = error_evaluation == SICONOS_FRICTION_3D_NSGS_ERROR_EVALUATION_LIGHT_WITH_FULL_FINAL ? FULL_FINAL
           : error_evaluation == SICONOS_FRICTION_3D_NSGS_ERROR_EVALUATION_LIGHT                ? LIGHT
                                                                                               : NO_EVAL;
  // mixed precision: FP32 sweeps first (for the two modes that stop on an
  // error), then the FP64 sweeps of the reference's loop from their iterate,
  // on the budget and trace position the FP32 phase leaves (read on the
  // device: both launches go out back to back)
  const bool mixed = c->precision == 0 && a.mode != NO_EVAL && max_iter > 0;
  K2(cudaEventRecord(c->ev[0], c->stream));
  if (mixed) {
    Args<float> b = args32(c);
    b.tol = tol;
    b.max_iter = max_iter;
    b.mode = FP32_PHASE;
    b.switch_tol = c->switch_tol > 0.0 ? c->switch_tol : std::max(tol, 1e-6);
    b.stall = c->stall;
    const Shape& s = c->s32;
    b.rows = s.rows;
    if (s.grid) K2(cudaMemsetAsync(c->arrived, 0, sizeof(unsigned), c->stream));
    K2(s.flow  ? launch_grid(c, s, k_fc2d_nsgs<float, false, FlowTeam>, b)
       : s.grid ? launch_grid(c, s, k_fc2d_nsgs<float, false, GridTeam>, b)
       : s.rep ? launch(c, s, k_fc2d_nsgs<float, true, ClusterTeam>, b, sizeof(float2) * (size_t)c->nc)
               : launch(c, s, k_fc2d_nsgs<float, false, ClusterTeam>, b, 0));
    a.before = c->out + 4;
  }
  const Shape& s = c->s64;
  a.rows = s.rows;
  if (s.grid) K2(cudaMemsetAsync(c->arrived, 0, sizeof(unsigned), c->stream));
  if (s.alone)
    K2(s.grid  ? launch_grid(c, s, k_fc2d_nsgs<double, false, GridAlone>, a)
       : s.rep ? launch(c, s, k_fc2d_nsgs<double, true, ClusterAlone>, a, rep_bytes(c))
               : launch(c, s, k_fc2d_nsgs<double, false, ClusterAlone>, a, 0));
  else
    K2(s.flow  ? launch_grid(c, s, k_fc2d_nsgs<double, false, FlowTeam>, a)
       : s.grid ? launch_grid(c, s, k_fc2d_nsgs<double, false, GridTeam>, a)
       : s.rep ? launch(c, s, k_fc2d_nsgs<double, true, ClusterTeam>, a, rep_bytes(c))
               : launch(c, s, k_fc2d_nsgs<double, false, ClusterTeam>, a, 0));
  K2(cudaEventRecord(c->ev[1], c->stream));
  double out[9];
  K2(cudaMemcpyAsync(out, c->out, sizeof(out), cudaMemcpyDeviceToHost, c->stream));
  K2(cudaStreamSynchronize(c->stream));
  if (out[8] != 0.0) return gave_up(c, "fc2dgpu_ctx_solve");
  float t = 0.f;
  cudaEventElapsedTime(&t, c->ev[0], c->ev[1]);
  if (iters) *iters = (int)out[0];
  if (error) *error = out[1];
  if (info) *info = (int)out[2];
  if (ms) *ms = t;
  c->sweeps32 = mixed ? (int)out[4] : 0;
  c->sweeps64 = (int)out[0] - c->sweeps32;
  c->trace_len = std::min((int)out[0], TRACE_CAP);
  return 0;
}

extern "C" int fc2dgpu_ctx_get_r_u(fc2dgpu_ctx* c, double* r, double* u) {
  if (!c || c->nc == 0) return NUMERICS_ERR_INVALID_ARGUMENT;
  K2(cudaSetDevice(c->device));
  std::vector<double> rp(2 * (size_t)c->nc), up(2 * (size_t)c->nc);
  K2(copy_to_host(rp.data(), c->r, sizeof(double) * rp.size(), c->stream));
  K2(copy_to_host(up.data(), c->u, sizeof(double) * up.size(), c->stream));
  for (int i = 0; i < c->nc; i++) {
    const size_t p = (size_t)c->iperm[i];
    if (r) {
      r[2 * i] = rp[2 * p];
      r[2 * i + 1] = rp[2 * p + 1];
    }
    if (u) {
      u[2 * i] = up[2 * p];
      u[2 * i + 1] = up[2 * p + 1];
    }
  }
  return 0;
}

extern "C" int fc2dgpu_ctx_colours(fc2dgpu_ctx* c, int32_t* colour) {
  if (!c || c->nc == 0) return NUMERICS_ERR_INVALID_ARGUMENT;
  if (colour) memcpy(colour, c->colour.data(), sizeof(int32_t) * c->nc);
  return c->ncol;
}

extern "C" int fc2dgpu_ctx_trace(fc2dgpu_ctx* c, double* out, int cap) {
  if (!c) return -1;
  const int n = std::min(cap, c->trace_len);
  if (n <= 0 || !out) return 0;
  K2(cudaSetDevice(c->device));
  K2(copy_to_host(out, c->trace, sizeof(double) * n, c->stream));
  return n;
}
