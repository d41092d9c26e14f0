// The rolling-friction one-contact Newton on five lanes a contact.
//
// What bounds it: on one lane a Newton iteration is a chain of about 600 FP64
// operations and 30 divisions and roots, and GB300's FP64 unit takes one warp
// instruction in 64 to 76 cycles whatever its lanes do (see
// fc3dgpu_ieee64.cuh), so a colour costs that chain times up to 9 iterations
// even for one contact.  Here lane i of a group of five holds component i of
// every vector and row i of every matrix, six contacts a warp: the products
// with 5x5 matrices, the elimination's row updates and the Jacobian's rows
// run side by side (about 155 FP64 instructions an iteration), divisions,
// roots and comparisons run on the integer pipes, the point an iteration ends
// at is the one the next starts from, and products with the structural zeros
// of the velocity matrix (which can only change the sign of a zero) are left
// out.  FP64 sweep by colours, one lane -> five lanes a contact, copies of
// the rockfall problem: 547 -> 161 us at 21 contacts, 892 -> 259 at 2,100,
// 1,015 -> 507 at 21,000, 3,898 -> 3,009 at 210,000.  The FP32 sweeps stay on
// one lane: the exchanges cost what they save there (83 and 86 us at 21
// contacts, 147 and 224 at 21,000).
//
// The control flow is the same for the whole warp: loops run until its last
// contact is done, finished contacts keep their values, and the collectives
// are full-warp shuffles and votes.  Every value is formed by the operations
// and in the order of the reference (cited in rfc3dgpu.cu at the one-lane
// form), so the bits are the same.
#pragma once
#include "fc3dgpu_ieee64.cuh"

namespace rfc3dgpu {

#define RFC3D_COOP_GROUPS 6  // contacts of a warp (lanes 30 and 31 idle)

using fc3dgpu::ie_abs;
using fc3dgpu::ie_div;
using fc3dgpu::ie_le;
using fc3dgpu::ie_lt;
using fc3dgpu::ie_sqrt;

// The lane's place: component i of the group whose first lane is `base`.
struct RLane {
  int i, base;
};

__device__ __forceinline__ double rget(double x, int lane) {
  return __shfl_sync(0xffffffffu, x, lane);
}
__device__ __forceinline__ bool rany(bool p) { return __any_sync(0xffffffffu, p); }
__device__ __forceinline__ void rall(const RLane& c, double x, double out[5]) {
#pragma unroll
  for (int k = 0; k < 5; k++) out[k] = rget(x, c.base + k);
}
// the components summed in order
__device__ __forceinline__ double rsum(const RLane& c, double x) {
  double a[5];
  rall(c, x, a);
  return a[0] + a[1] + a[2] + a[3] + a[4];
}
// the norms of components 1, 2 (n12) and 3, 4 (n34)
__device__ __forceinline__ void rnorms(const RLane& c, double x, double& n12, double& n34) {
  const double sq = x * x;
  const int t = c.base + (c.i >= 3 ? 3 : 1);
  const double n = ie_sqrt(rget(sq, t) + rget(sq, t + 1));
  n12 = rget(n, c.base + 1);
  n34 = rget(n, c.base + 3);
}

struct RProblem {
  double M[25];  // the whole diagonal block, column-major
  double q;      // component i
  double mu, mur, rho;
  double d1, d2, d3;  // mur^2 + mu^2 + 1, mu^2 + 1, mur^2 + 1
  double k1, k2, k3;  // 1 / (1 + mu^2 + mur^2), 1 / (1 + mu^2), 1 / (1 + mur^2)
};

__device__ __forceinline__ void rconstants(RProblem& P) {
  const double mu2 = P.mu * P.mu, mur2 = P.mur * P.mur;
  P.d1 = mur2 + mu2 + 1.0;
  P.d2 = mu2 + 1.0;
  P.d3 = mur2 + 1.0;
  P.k1 = ie_div(1.0, 1.0 + mu2 + mur2);
  P.k2 = ie_div(1.0, 1.0 + mu2);
  P.k3 = ie_div(1.0, 1.0 + mur2);
}

// row i of M times x, onto q
__device__ __forceinline__ double rvelocity(const RLane& c, const RProblem& P, double r) {
  double x[5], v = P.q;
  rall(c, r, x);
#pragma unroll
  for (int j = 0; j < 5; j++) {
    const double m = c.i == 0 ? P.M[5 * j]
                         : (c.i == 1 ? P.M[5 * j + 1]
                                     : (c.i == 2 ? P.M[5 * j + 2] : (c.i == 3 ? P.M[5 * j + 3] : P.M[5 * j + 4])));
    v += m * x[j];
  }
  return v;
}

enum { RZ_DUAL = 0, RZ_INSIDE, RZ_OUT };

// A point: velocity v, natural map F and what its gradient shares.
struct RPoint {
  double v, F, RV;
  double nVT, nOT;      // norms of the velocity's tangent and rolling parts
  double nT, nM, rv0;   // norms and first component of RV
  int zone;
};

// natural_map without gradient
__device__ __forceinline__ void rpoint(const RLane& c, const RProblem& P, double r, RPoint& p) {
  rnorms(c, p.v, p.nVT, p.nOT);
  const double t0 = p.v + P.mu * p.nVT + P.mur * p.nOT;
  p.RV = r - P.rho * (c.i == 0 ? t0 : p.v);
  rnorms(c, p.RV, p.nT, p.nM);
  p.rv0 = rget(p.RV, c.base);
  const double mT = P.mu * p.nT, mM = P.mur * p.nM, a = mT + mM;
  const bool dual = ie_le(a, -p.rv0);
  const bool inside = ie_le(p.nT, P.mu * p.rv0) && ie_le(p.nM, P.mur * p.rv0);
  p.zone = dual ? RZ_DUAL : (inside ? RZ_INSIDE : RZ_OUT);
  double F = p.RV;
  const bool out = p.zone == RZ_OUT;
  if (rany(out)) {
    // the projection's regions in the reference's order
    double t = ie_div(a + p.rv0, P.d1);
    const bool both = out && ie_lt(P.mu * t, p.nT) && ie_lt(P.mur * t, p.nM);
    bool fric = false, roll = false;
    if (rany(out && !both)) {
      const double t2 = ie_div(mT + p.rv0, P.d2);
      fric = out && !both && ie_lt(P.mu * t2, p.nT) && ie_le(p.nM, P.mur * t2);
      if (fric) t = t2;
      if (rany(out && !both && !fric)) {
        const double t3 = ie_div(mM + p.rv0, P.d3);
        roll = out && !both && !fric && ie_le(p.nT, P.mu * t3) && ie_lt(P.mur * t3, p.nM);
        if (roll) t = t3;
      }
    }
    const bool tang = c.i == 1 || c.i == 2;
    const bool mine = c.i > 0 && (both || (fric && tang) || (roll && !tang));
    const double x = ie_div((c.i <= 2 ? P.mu : P.mur) * t * p.RV, mine ? (c.i <= 2 ? p.nT : p.nM) : 1.0);
    if (mine) F = x;
    if (c.i == 0 && (both || fric || roll)) F = t;
  }
  p.F = r - (dual ? 0.0 : F);
}

// Row i of -(A M + B), the Newton matrix at p
__device__ __forceinline__ void rmatrix(const RLane& c, const RProblem& P, const RPoint& p, double G[5]) {
  const int i = c.i;
  const bool tang = i == 1 || i == 2;
  // first row of the velocity matrix D (the other rows are rho on the diagonal)
  const double nv = i <= 2 ? p.nVT : p.nOT;
  const bool flat = ie_le(nv, 0.0);
  double s = ie_div(p.v, i == 0 || flat ? 1.0 : nv);
  if (flat) s = i == 1 || i == 3 ? 1.0 : 0.0;
  const double d = i == 0 ? P.rho : P.rho * (i <= 2 ? P.mu : P.mur) * s;
  double D[5];
  rall(c, d, D);
  double a[5], b[5];
  if (p.zone == RZ_DUAL) {
#pragma unroll
    for (int j = 0; j < 5; j++) {
      a[j] = 0.0;
      b[j] = i == j ? 1.0 : 0.0;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 5; j++) {
      a[j] = i == 0 ? D[j] : (i == j ? P.rho : 0.0);
      b[j] = 0.0;
    }
  }
  const bool out = p.zone == RZ_OUT;
  if (rany(out)) {
    // the subdifferential H of the projection at RV
    const double mT = P.mu * p.nT, mM = P.mur * p.nM;
    const double a1 = mT + mM + p.rv0, b1 = p.rv0 + mT, c1 = mM + p.rv0;
    double t = a1 * P.k1;
    const bool both = ie_lt(P.mu * t, p.nT) && ie_lt(P.mur * t, p.nM);
    t = b1 * P.k2;
    const bool fric = !both && ie_lt(P.mu * t, p.nT) && ie_le(p.nM, P.mur * t);
    t = c1 * P.k3;
    const bool roll = !both && !fric && ie_le(p.nT, P.mu * t) && ie_lt(P.mur * t, p.nM);
    const double k = both ? P.k1 : (fric ? P.k2 : P.k3);
    const bool mine = i > 0 && (both || (fric && tang) || (roll && !tang));
    const double g = (i <= 2 ? P.mu : P.mur) * k;
    const double n = out && mine ? (i <= 2 ? p.nT : p.nM) : 1.0;
    const double sr = ie_div(p.RV, n), gn = ie_div(g, n);
    const double h0 = g * sr;
    const double ci = both ? (i <= 2 ? p.rv0 + mM : b1) : p.rv0;
    const double add = both ? a1 : (fric ? b1 : c1);
    double S[5];
    rall(c, sr, S);
    const double sA = i <= 2 ? S[1] : S[3], sB = i <= 2 ? S[2] : S[4];
    const double hii = gn * (-ci * sr * sr + add), hip = gn * (-ci * sA * sB);
    const double w = h0 * P.mur;
    const double w1 = rget(w, c.base + 1), w2 = rget(w, c.base + 2);
    const double x1 = (i == 2 ? w2 : w1) * (i == 4 ? S[4] : S[3]), x2 = (i == 1 ? w1 : w2) * (i == 3 ? S[3] : S[4]);
    // row i of H
    double h[5];
    const bool some = both || fric || roll;
    h[0] = i == 0 ? (some ? k : 0.0) : (mine ? h0 : 0.0);
    const double col = mine ? h0 : 0.0;
    const double one = some && !mine ? 1.0 : 0.0;  // the other pair's rows are the identity
    h[1] = tang ? (mine ? (i == 1 ? hii : hip) : (i == 1 ? one : 0.0)) : (i > 0 && both ? x1 : 0.0);
    h[2] = tang ? (mine ? (i == 2 ? hii : hip) : (i == 2 ? one : 0.0)) : (i > 0 && both ? x2 : 0.0);
    h[3] = i >= 3 ? (mine ? (i == 3 ? hii : hip) : (i == 3 ? one : 0.0)) : (tang && both ? x1 : 0.0);
    h[4] = i >= 3 ? (mine ? (i == 4 ? hii : hip) : (i == 4 ? one : 0.0)) : (tang && both ? x2 : 0.0);
#pragma unroll
    for (int j = 1; j < 5; j++) {
      const double y = rget(col, c.base + j);
      if (i == 0) h[j] = y;
    }
#pragma unroll
    for (int j = 0; j < 5; j++) {
      const double x = j == 0 ? h[0] * P.rho : h[0] * D[j] + h[j] * P.rho;
      const double y = i == j ? 1.0 - h[j] : -h[j];
      if (out) {
        a[j] = x;
        b[j] = y;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 5; j++)
    G[j] = -((a[0] * P.M[5 * j] + a[1] * P.M[5 * j + 1] + a[2] * P.M[5 * j + 2] + a[3] * P.M[5 * j + 3] +
              a[4] * P.M[5 * j + 4]) +
             b[j]);
}

// gepp5 of the system with rows G: component i of the solution, or of F as it
// is on a tiny pivot
__device__ __forceinline__ double rsolve(const RLane& c, const double G[5], double F) {
  double A[5], x = F;
#pragma unroll
  for (int j = 0; j < 5; j++) A[j] = G[j];
  bool tiny = false;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    // the pivot of column k: the first largest entry of rows k and below
    double piv = rget(A[k], c.base + k), best = ie_abs(piv);
    int at = k;
#pragma unroll
    for (int l = k + 1; l < 5; l++) {
      const double e = rget(A[k], c.base + l), m = ie_abs(e);
      if (ie_lt(best, m)) {
        best = m;
        piv = e;
        at = l;
      }
    }
    if (ie_lt(best, 1e-16)) tiny = true;
    if (k == 4) break;
    if (rany(at != k)) {
      const int src = c.base + (c.i == k ? at : (c.i == at ? k : c.i));
#pragma unroll
      for (int j = k; j < 5; j++) A[j] = rget(A[j], src);
      x = rget(x, src);
    }
    const bool below = c.i > k;
    const double f = ie_div(below ? A[k] : 0.0, tiny ? 1.0 : piv);
#pragma unroll
    for (int j = k + 1; j < 5; j++) {
      const double y = A[j] - f * rget(A[j], c.base + k);
      if (below) A[j] = y;
    }
    const double y = x - f * rget(x, c.base + k);
    if (below) x = y;
  }
  const double Aii = c.i == 0 ? A[0] : (c.i == 1 ? A[1] : (c.i == 2 ? A[2] : (c.i == 3 ? A[3] : A[4])));
  const double den = tiny ? 1.0 : Aii;
  double prod[5];
#pragma unroll
  for (int k = 4; k >= 0; k--) {
    double t = x;
    if (k < 4) {
      double s = prod[k + 1];
#pragma unroll
      for (int j = k + 2; j < 5; j++) s += prod[j];
      t = x - s;
    }
    const double xk = rget(ie_div(t, den), c.base + k);
    if (c.i == k) x = xk;
    prod[k] = A[k] * xk;
  }
  return tiny ? F : x;
}

// local_nsn of one contact a group (`act` false leaves a group out): r is
// component i of its reaction.
__device__ __forceinline__ void rlocal_solve(const RLane& c, RProblem& P, bool act, double eps, double tol, int itermax,
                                             double& r) {
  rconstants(P);
  const double nq = ie_sqrt(rsum(c, P.q * P.q));
  const bool has = ie_lt(eps, nq);
  const double inv = ie_div(1.0, has ? nq : 1.0);
  const double rel = has ? inv : 1.0;
  RPoint p;
  p.v = rvelocity(c, P, r);
  rpoint(c, P, r, p);
  double res = ie_sqrt(rsum(c, p.F * p.F)) * rel;
  bool run = act && !ie_lt(res, tol);
  for (int it = 1; it < itermax && rany(run); it++) {
    double G[5];
    rmatrix(c, P, p, G);
    const double dR = rsolve(c, G, p.F);
    const double rn = r + dR;
    RPoint t;
    t.v = rvelocity(c, P, rn);
    rpoint(c, P, rn, t);
    // the reference's residual after a step cubes the third component
    double f2 = t.F * t.F;
    const double f3 = f2 * t.F;
    if (c.i == 2) f2 = f3;
    const double e2 = rsum(c, f2) * rel;
    const double x = ie_sqrt(ie_lt(0.0, e2) ? e2 : 0.0);
    if (run) {
      const double old = res;
      r = rn;
      p = t;
      res = x;
      if (ie_lt(res, tol) || ie_lt(ie_abs(res - old), eps)) run = false;
    }
  }
}

}  // namespace rfc3dgpu
