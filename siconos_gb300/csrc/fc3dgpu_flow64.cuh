// The FP64 sweep as dataflow, three lanes a contact.
//
// What bounds an FP64 sweep by colours: a colour takes as long as its slowest
// block (a contact that needs the PLI loop and a second Newton takes twice a
// usual one), and an SM's other quarters idle meanwhile: 48 us a colour on a
// 41,000-contact lattice for a mean of 26 us of work in a block.  Here a warp
// takes units of up to ten contacts (fc3dgpu_coop64.cuh) and waits only for the
// reactions they read, as the FP32 dataflow does (fc3dgpu_flow.cuh gives the
// argument that every contact reads exactly the sequential sweep's values;
// the block pattern is symmetric here too).  Each colour's units are dealt
// over all blocks, so every SM quarter has work of each colour.  us a sweep by colours and as
// dataflow (lattices of n contacts, 6 colours):
//   42: 130, 85    2,800: 244, 138    11,600: 263, 190    40,935: 296, 236
//   68,688: 408, 305    96,780: 453, 392    125,840: 483, 475    163,584: 541, 594
// Beyond FC3D_FLOW64_MAX contacts a colour and block the sweeps go by colours:
// the FP64 pipe is then full either way and one lane a contact needs it less.
//
// A stamped reaction is 32 bytes, two 128-bit words that are each stored and
// loaded as one access and each carry the sweep: (r0, low half of r1, sweep)
// and (r2, high half of r1, sweep).  A reader takes a reaction when both words
// show the sweep it needs.  The plain reactions are stored beside them for the
// error evaluation.
#pragma once
#include "fc3dgpu_coop64.cuh"
#include "fc3dgpu_word128.cuh"

namespace fc3dgpu {

// Polls of a reaction before the back-off, and the back-off (ns).
#define FC3D_FLOW64_SPIN 16
#define FC3D_FLOW64_SLEEP_NS 100

// The reaction in the two words w; false before sweep `need` has written it.
__device__ __forceinline__ bool take_stamped64(const unsigned long long w[4], int need, double x[3]) {
  x[0] = __longlong_as_double((long long)w[0]);
  x[1] = __longlong_as_double((long long)((w[1] & 0xffffffffull) | (w[3] << 32)));
  x[2] = __longlong_as_double((long long)w[2]);
  return (int)(w[1] >> 32) >= need && (int)(w[3] >> 32) >= need;
}
__device__ __forceinline__ bool ld_stamped64(const double* rs, int p, int need, double x[3]) {
  unsigned long long w[4];
  ld_word128(rs + 4 * (size_t)p, w[0], w[1]);
  ld_word128(rs + 4 * (size_t)p + 2, w[2], w[3]);
  return take_stamped64(w, need, x);
}
// Word `w` (0 or 1) of the stamped reaction p
__device__ __forceinline__ void st_stamped64(double* rs, int p, int w, const double x[3], int stamp) {
  const unsigned long long r1 = (unsigned long long)__double_as_longlong(x[1]), s = (unsigned long long)(unsigned)stamp << 32;
  st_word128(rs + 4 * (size_t)p + 2 * w, (unsigned long long)__double_as_longlong(w ? x[2] : x[0]),
             (w ? r1 >> 32 : r1 & 0xffffffffull) | s);
}

// The unit of rows [p0, p1) of a colour, at most FC3D_COOP_GROUPS, in sweep
// `sweep`; false when a wait gave up.
__device__ __forceinline__ bool flow64_unit(const SweepArgs<double>& a, int p0, int p1, int sweep, double ltol,
                                            double& dr2, double& rr2) {
  const int lane = threadIdx.x & 31;
  const bool spare = lane >= 3 * FC3D_COOP_GROUPS;
  CoopLane c;
  const int g = spare ? 0 : lane / 3;
  c.base = 3 * g;
  c.i = lane - (spare ? 3 * FC3D_COOP_GROUPS : c.base);
  // groups without a row repeat the unit's first without storing it
  int p = p0 + g;
  const bool have = !spare && p < p1 && __ldg(&a.perm[p]) >= 0;
  const unsigned haves = __ballot_sync(0xffffffffu, have);
  if (!haves) return true;
  const int lead = __shfl_sync(0xffffffffu, p, __ffs(haves) - 1);
  if (!have) p = lead;
  const int sl = p / FC3D_SLAB, k = p % FC3D_SLAB;
  const long long base = a.slab_off[sl];
  const int ns = a.slab_nslot[sl];
  const int nsmax = __reduce_max_sync(0xffffffffu, ns);
  CoopProblem P;
#pragma unroll
  for (int e = 0; e < 9; e++) P.M[e] = __ldg(&a.D[((size_t)sl * 9 + e) * FC3D_SLAB + k]);
  P.m0 = c.i == 0 ? P.M[0] : (c.i == 1 ? P.M[1] : P.M[2]);
  P.m1 = c.i == 0 ? P.M[3] : (c.i == 1 ? P.M[4] : P.M[5]);
  P.m2 = c.i == 0 ? P.M[6] : (c.i == 1 ? P.M[7] : P.M[8]);
  P.mu = __ldg(&a.mu[(size_t)sl * FC3D_SLAB + k]);
  P.rhoN = __ldg(&a.rho[((size_t)sl * 2) * FC3D_SLAB + k]);
  P.rhoT = __ldg(&a.rho[((size_t)sl * 2 + 1) * FC3D_SLAB + k]);
  P.rho_i = c.i == 0 ? P.rhoN : P.rhoT;
  double rpli = __ldcg(&a.rpli[p]);
  const double o = __ldcg(&a.r[(size_t)p * FC3D_RSTRIDE + c.i]);
  double acc = a.q[((size_t)sl * 3 + c.i) * FC3D_SLAB + k];
  bool ok = true;
  constexpr int CH = 5;
  for (int t0 = 0; t0 < nsmax && ok; t0 += CH) {
    int pj[CH];
    double wv[CH][3], rv[CH][3];
#pragma unroll
    for (int t = 0; t < CH; t++) {
      const size_t s = (size_t)(base + (t0 + t < ns ? t0 + t : 0));
      pj[t] = t0 + t < ns ? __ldg(&a.col[s * FC3D_SLAB + k]) : a.npad;
      const double* wp = a.W + (s * 9 + c.i) * FC3D_SLAB + k;
#pragma unroll
      for (int e = 0; e < 3; e++) wv[t][e] = t0 + t < ns ? __ldg(&wp[3 * e * FC3D_SLAB]) : 0.0;
    }
    // (a second block on the diagonal reads the row's own last reaction)
    unsigned late = 0;
#pragma unroll
    for (int t = 0; t < CH; t++)
      late |= (ld_stamped64(a.rs, pj[t], sweep - (pj[t] >= p ? 1 : 0), rv[t]) ? 0u : 1u) << t;
    unsigned long long polls = 0;
    while (late) {
      if (++polls > a.spin_limit) {
        atomicOr(a.status, 1);
        ok = false;
        break;
      }
      if (polls > FC3D_FLOW64_SPIN) __nanosleep(FC3D_FLOW64_SLEEP_NS);
      // a poll's loads are predicated, without a branch between them, so it
      // costs one memory latency (40,935 contacts: 257 us a sweep with
      // branches, 242 without, 236 with five slots at once in place of six)
      unsigned long long w[CH][4];
#pragma unroll
      for (int t = 0; t < CH; t++) {
        ld_word128_if(late >> t & 1u, a.rs + 4 * (size_t)pj[t], w[t][0], w[t][1]);
        ld_word128_if(late >> t & 1u, a.rs + 4 * (size_t)pj[t] + 2, w[t][2], w[t][3]);
      }
#pragma unroll
      for (int t = 0; t < CH; t++)
        if ((late >> t & 1u) && take_stamped64(w[t], sweep - (pj[t] >= p ? 1 : 0), rv[t])) late &= ~(1u << t);
    }
    // the lanes left the wait one by one: together again, and all of them leave
    // the loop when one gave up
    ok = __all_sync(0xffffffffu, ok);
#pragma unroll
    for (int t = 0; t < CH; t++)
      if (t0 + t < ns) {
        acc += wv[t][0] * rv[t][0];
        acc += wv[t][1] * rv[t][1];
        acc += wv[t][2] * rv[t][2];
      }
  }
  if (!ok) return false;
  P.q = acc;
  const bool off = ie_lt(-DBL_EPSILON, coop_get(acc, c.base));  // take-off
  const bool act = have && !off;
  double rn = o, residual = 0.0;
  CoopCount work = {0, 0, 0, false};
  if (coop_any(act)) residual = coop_local_solve(c, P, act, a, ltol, rn, rpli, work);
  if (off) {
    rn = 0.0;
    residual = 0.0;
  }
  if (a.relax) rn = a.omega * rn + (1.0 - a.omega) * o;
  const bool discard = a.filter && (!finite64(residual) || residual > 1.0);
  const double keep = discard ? o : rn;
  double x[3];
  coop_all(c, keep, x);
  if (have && c.i < 2) st_stamped64(a.rs, p, c.i, x, sweep);
  if (have) a.r[(size_t)p * FC3D_RSTRIDE + c.i] = keep;
  const double d = o - rn;
  const double d2 = coop_sum(c, d * d), k2 = coop_sum(c, keep * keep);
  if (have && c.i == 0) {
    if (!off) a.rpli[p] = rpli;
    dr2 += d2;
    rr2 += k2;
    if (a.counters && !off) {
      atomicAdd(&a.counters[0], (unsigned long long)work.newton);
      atomicAdd(&a.counters[1], (unsigned long long)work.pli);
      atomicAdd(&a.counters[2], (unsigned long long)work.ls);
      atomicAdd(&a.counters[3], 1ULL);
      atomicMax(&a.counters[4], (unsigned long long)work.newton);
    }
  }
  return true;
}

// Rows of a unit: what gives every SM quarter a unit of an average colour, so
// that few contacts share one warp's control flow (a warp runs as long as its
// slowest contact): 2,800 contacts in units of ten 202 us a sweep, of one 140;
// two units a quarter are 11 % slower at 40,935.
__device__ __forceinline__ int flow64_rows(const int* sptr, int ncol, int size) {
  const long long n = (long long)(sptr[ncol] - sptr[0]) * FC3D_SLAB, per = (long long)ncol * size * 4;
  return (int)min((long long)FC3D_COOP_GROUPS, max(1LL, (n + per - 1) / per));
}

// One sweep over the colours whose slabs are sptr[c] .. sptr[c + 1), by block
// `rank` of `size`: unit u of `rows` rows of a colour goes to block u mod
// size, a block's units in colour order to its warps in turn (in the order of
// the rows' costs, as the sweep by colours takes them, a sweep of 40,935 was 3
// % slower, of 68,688 3 % faster).  False when a wait gave up (the same value
// in every thread of the block).
__device__ __forceinline__ bool flow64_sweep(const SweepArgs<double>& a, const int* sptr, int ncol, int rows, int rank,
                                             int size, int sweep, double ltol, double& dr2, double& rr2) {
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  bool ok = true;
  int e = w;  // the warp's next unit among the block's
  for (int c = 0; c < ncol && ok; c++) {
    const int r0 = sptr[c] * FC3D_SLAB, r1 = sptr[c + 1] * FC3D_SLAB;
    const int units = (r1 - r0 + rows - 1) / rows;
    const int mine = rank < units ? (units - rank + size - 1) / size : 0;
    for (; e < mine && ok; e += nw) {
      const int p0 = r0 + (rank + e * size) * rows;
      ok = flow64_unit(a, p0, min(r1, p0 + rows), sweep, ltol, dr2, rr2);
    }
    e -= mine;
  }
  return !__syncthreads_or(!ok);
}

}  // namespace fc3dgpu
