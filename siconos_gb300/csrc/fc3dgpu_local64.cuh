// The one-contact solver in FP64: the steps, branches and rounding of
// fc3dgpu_local.cuh (the reference's hybrid solver, cited there), arranged for
// GB300's FP64 rate.
//
// What bounds it: the FP64 unit of an SM quarter takes one warp instruction
// in 64 (fma) to 76 cycles, whatever the number of active lanes and without
// overlap, comparisons included; every other pipe is idle meanwhile.  So the
// time of a local solve is its count of FP64 instructions, and
//   - divisions, square roots and comparisons run on the integer pipes
//     (fc3dgpu_ieee64.cuh: the same bits);
//   - a value the reference computes twice from the same operands in the same
//     order is computed once: the velocity, Alart-Curnier function and |F|^2
//     of an accepted line-search point are those of the next iterate; the
//     line search's A M + B is the Newton matrix; the gradient shares the
//     function's terms; |q| and 1/|q| serve the whole solve;
//   - a comparison that only decides something (is the residual below the
//     tolerance, does the contact slip, is the step accepted) is decided in
//     FP32 from squares when it is clear there by a margin far above the FP32
//     error, and in the reference's form otherwise: the same decision, without
//     its root and quotient;
//   - products with entries of A and B that are zero by construction (the
//     whole of rows 1 and 2 in the sticking case but one entry each) are left
//     out: they can only change the sign of a zero;
//   - the natural-map error of the incoming reaction is evaluated only when
//     the Newton result does not meet the tolerance, the one case that reads
//     it (under 1 contact in 100 on the sphere lattices).
// One Newton iteration of a sticking contact takes 68 FP64 adds and multiplies
// where the plain form takes about 430 FP64 instructions.
#pragma once
#include "fc3dgpu_ieee64.cuh"
#include "fc3dgpu_local.cuh"

namespace fc3dgpu {

// Division and square root of the Newton and PLI steps: exact, or the seeded
// ones of the opt-in fast polish.
#ifdef FC3D_FAST_F64
struct LDen {
  double b;
};
__device__ __forceinline__ LDen lden(double b) { return LDen{b}; }
__device__ __forceinline__ double ldiv64(double a, const LDen& d) { return ldiv<double>(a, d.b); }
__device__ __forceinline__ void ldiv64x2(double a0, double a1, const LDen& d, double& q0, double& q1) {
  q0 = ldiv<double>(a0, d.b);
  q1 = ldiv<double>(a1, d.b);
}
__device__ __forceinline__ double lsqrt64(double x) { return dsqrt<double>(x); }
#else
using LDen = IeDen;
__device__ __forceinline__ LDen lden(double b) { return ie_den(b); }
__device__ __forceinline__ double ldiv64(double a, const LDen& d) { return ie_div(a, d); }
__device__ __forceinline__ void ldiv64x2(double a0, double a1, const LDen& d, double& q0, double& q1) {
  ie_div2(a0, a1, d, q0, q1);
}
__device__ __forceinline__ double lsqrt64(double x) { return ie_sqrt(x); }
#endif
__device__ __forceinline__ double ldiv64(double a, double b) { return ldiv64(a, lden(b)); }

template <>
__device__ __forceinline__ void project_cone<double>(double r[3], double mu) {
  const double normT = ie_sqrt(r[1] * r[1] + r[2] * r[2]);
  if (ie_le(mu * normT, -r[0])) {
    r[0] = 0;
    r[1] = 0;
    r[2] = 0;
  } else if (!ie_le(normT, mu * r[0])) {
    r[0] = ie_div(mu * normT + r[0], mu * mu + 1.0);
    const double t = mu * r[0];
    ie_div2(t * r[1], t * r[2], ie_den(normT), r[1], r[2]);
  }
}

template <>
__device__ __forceinline__ double unitary_error2<double>(const double r[3], const double u[3], double mu) {
  double w[3];
  w[0] = r[0] - u[0] - mu * ie_sqrt(u[1] * u[1] + u[2] * u[2]);
  w[1] = r[1] - u[1];
  w[2] = r[2] - u[2];
  project_cone<double>(w, mu);
  w[0] = r[0] - w[0];
  w[1] = r[1] - w[1];
  w[2] = r[2] - w[2];
  return w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
}

// solve3x3 with the quotients by one pivot sharing its reciprocal
template <>
__device__ __forceinline__ int solve3x3<double>(const double a[9], double b[3]) {
  const double E = DBL_EPSILON;
  const double aa0 = ie_abs(a[0]), aa1 = ie_abs(a[1]), aa2 = ie_abs(a[2]);
  const bool c01 = ie_le_pos(aa1, aa0), c02 = ie_le_pos(aa2, aa0), c12 = ie_le_pos(aa2, aa1);
  const int p1 = c01 ? (c02 ? 0 : 2) : (c12 ? 1 : 2);
  // pivot row l, the other two m and n in ascending order
  const int m = p1 == 0 ? 1 : 0;
  const double l0 = p1 == 0 ? a[0] : (p1 == 1 ? a[1] : a[2]), m0 = m ? a[1] : a[0], n0 = p1 == 2 ? a[1] : a[2];
  const double l1 = p1 == 0 ? a[3] : (p1 == 1 ? a[4] : a[5]), m1 = m ? a[4] : a[3], n1 = p1 == 2 ? a[4] : a[5];
  const double l2 = p1 == 0 ? a[6] : (p1 == 1 ? a[7] : a[8]), m2 = m ? a[7] : a[6], n2 = p1 == 2 ? a[7] : a[8];
  const double bl = p1 == 0 ? b[0] : (p1 == 1 ? b[1] : b[2]), b1 = m ? b[1] : b[0], b2 = p1 == 2 ? b[1] : b[2];
  if (ie_le_pos(ie_abs(l0), E)) return 1;
  const LDen d0 = lden(l0);
  double f1, f2;
  ldiv64x2(m0, n0, d0, f1, f2);
  const double lm1 = m1 - f1 * l1, lm2 = m2 - f1 * l2, ln1 = n1 - f2 * l1, ln2 = n2 - f2 * l2;
  const double bm = b1 - f1 * bl, bn = b2 - f2 * bl;
  const bool mn = ie_le_pos(ie_abs(ln1), ie_abs(lm1));
  const double u1 = mn ? lm1 : ln1, u2 = mn ? lm2 : ln2, ub = mn ? bm : bn;  // second pivot row
  const double w1 = mn ? ln1 : lm1, w2 = mn ? ln2 : lm2, wb = mn ? bn : bm;
  if (ie_lt_pos(ie_abs(u1), E)) return 1;
  const LDen d1 = lden(u1);
  const double f = ldiv64(w1, d1);
  const double s2 = ldiv64(wb - f * ub, w2 - f * u2);
  const double s1 = ldiv64(ub - u2 * s2, d1);
  b[0] = ldiv64(bl - s1 * l1 - s2 * l2, d0);
  b[1] = s1;
  b[2] = s2;
  return 0;
}

// A point of the Newton iteration: the velocity v = M r + q, the
// Alart-Curnier function F there and the terms its gradient shares.
struct AcPoint {
  double v[3];
  double F[3];
  double FF;                // |F|^2
  double RVT, RVS, TT, SS;  // r_T - rhoT v_T and its squares
  double RV1;               // 1 / |r_T - rhoT v_T| (slip)
  double Radius;
  bool contact;  // r_n - rhoN v_n > 0
  int zone;      // 0 stick, 1 slip, 2 no contact, 3 undefined (NaN)
};

__device__ __forceinline__ void velocity64(const LocalProblem<double>& L, const double r[3], double v[3]) {
  v[0] = L.q[0];
  v[1] = L.q[1];
  v[2] = L.q[2];
  mvp3x3<double>(L.M, r, v);
}

// FP32 margins of the decisions below: the operands' relative errors are
// under 2^-21, a decision taken is off by 1e-4 or more.
#define FC3D_CLEAR 1e-4f

// sqrt(s) against Radius: 0 clearly below (stick), 1 not decided or slip, 2
// Radius is +0, where s itself can be compared in place of the root.
__device__ __forceinline__ int slip_clear(double s, double Radius) {
  if (ie_bits(Radius) == 0) return 2;
  const float sf = ie_float(s), rf = ie_float(Radius);
  return rf > 1e-15f && rf < 1e15f && sf < (1.f - FC3D_CLEAR) * rf * rf && ie_positive(Radius) ? 0 : 1;
}
// The zone of RV = |r_T - rhoT v_T| (>= 0 or NaN) against Radius: 0 stick,
// 1 slip, 2 no contact, 3 undefined
__device__ __forceinline__ int slip_zone(double RV, double Radius) {
  if ((int64_t)ie_bits(Radius) < 0) return ie_nan(RV) || ie_nan(Radius) ? 3 : (ie_le(RV, Radius) ? 0 : 2);
  return ie_le_pos(RV, Radius) ? 0 : (ie_lt_pos(Radius, RV) ? (ie_positive(Radius) ? 1 : 2) : 3);
}

// The squared limit (tol |q|)^2 of the local residual and error in FP32;
// plain is false where it says nothing (|q| near epsilon, out of range).
struct LocalLimit {
  float lim2;
  bool plain;
};
__device__ __forceinline__ LocalLimit local_limit(double qq, double tol) {
  const float q2 = ie_float(qq), t = ie_float(tol);
  LocalLimit l;
  l.lim2 = (t * q2) * t;
  l.plain = q2 > 1e-30f && t < 0.5f && l.lim2 > 1e-36f && l.lim2 < 1e30f;
  return l;
}
// sqrt(x2) / |q| < tol: 1 clearly, 0 clearly not, -1 not decided
__device__ __forceinline__ int below_limit(const LocalLimit& l, double x2) {
  const float x = ie_float(x2);
  if (!l.plain) return -1;
  return x < (1.f - 100.f * FC3D_CLEAR) * l.lim2 ? 1 : (x > (1.f + 100.f * FC3D_CLEAR) * l.lim2 ? 0 : -1);
}

// The Goldstein-Price test 0.9 dq <= slope <= 0.1 dq of a first trial
// (alpha = 1) in FP32: d approximates dq within 4e-6 S.  Bit 0: the left
// part holds, bit 1: the right part; -1 not decided.
__device__ __forceinline__ int search_clear(float slope, float d, float S) {
  const float m = 4e-6f * S + 1e-5f * fabsf(slope);
  const float a = slope - 0.9f * d, b = 0.1f * d - slope;
  if (!(S > 1e-30f && S < 1e30f && fabsf(a) > m && fabsf(b) > m)) return -1;
  return (a > 0.f ? 1 : 0) | (b > 0.f ? 2 : 0);
}

// ac_std without gradient at (r, p.v).  F[1] and F[2] keep their values in
// the undefined zone, as there.
__device__ __forceinline__ void ac_eval64(const LocalProblem<double>& L, const double r[3], AcPoint& p) {
  const double pn = L.rhoN * p.v[0], pt = L.rhoT * p.v[1], ps = L.rhoT * p.v[2];
  const double RVN = r[0] - pn;
  p.RVT = r[1] - pt;
  p.RVS = r[2] - ps;
  p.TT = p.RVT * p.RVT;
  p.SS = p.RVS * p.RVS;
  const double s = p.TT + p.SS;
  p.contact = ie_positive(RVN);
  p.Radius = 0;
  p.F[0] = r[0];
  if (p.contact) {
    p.Radius = L.mu * RVN;
    p.F[0] = pn;
  }
  const int clear = slip_clear(s, p.Radius);
  if (clear == 0) {
    p.zone = 0;
  } else {
    const double RV = clear == 2 ? s : lsqrt64(s);  // (no contact: the sign of either)
    p.zone = slip_zone(RV, p.Radius);
    if (p.zone == 1) p.RV1 = ldiv64(1.0, RV);
  }
  if (p.zone == 0) {
    p.F[1] = pt;
    p.F[2] = ps;
  } else if (p.zone == 1) {
    p.F[1] = r[1] - p.Radius * p.RVT * p.RV1;
    p.F[2] = r[2] - p.Radius * p.RVS * p.RV1;
  } else if (p.zone == 2) {
    p.F[1] = r[1];
    p.F[2] = r[2];
  }
  p.FF = p.F[0] * p.F[0] + p.F[1] * p.F[1] + p.F[2] * p.F[2];
}

// Rows 1 and 2 of the gradients A (with respect to u) and B (r) of a slip
// point; both keep their values in the undefined zone, as there.
struct AcGrad {
  double A1, A2, A4, A7, A8, B1, B2, B4, B7, B8;
};

// G = A M + B at p
__device__ __forceinline__ void ac_matrix64(const LocalProblem<double>& L, const AcPoint& p, AcGrad& g, double G[9]) {
  const double* M = L.M;
#pragma unroll
  for (int j = 0; j < 3; j++) G[3 * j] = p.contact ? L.rhoN * M[3 * j] : (j == 0 ? 1.0 : 0.0);
  if (p.zone == 0) {
    g.A1 = g.A2 = g.A7 = 0;
    g.A4 = g.A8 = L.rhoT;
    g.B1 = g.B2 = g.B4 = g.B7 = g.B8 = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      G[1 + 3 * j] = L.rhoT * M[1 + 3 * j];
      G[2 + 3 * j] = L.rhoT * M[2 + 3 * j];
    }
  } else if (p.zone == 2) {
    g.A1 = g.A2 = g.A4 = g.A7 = g.A8 = 0;
    g.B1 = g.B2 = g.B7 = 0;
    g.B4 = g.B8 = 1;
    G[1] = G[2] = G[5] = G[7] = 0;
    G[4] = G[8] = 1;
  } else {
    if (p.zone == 1) {
      const double RV1 = p.RV1, RV3 = RV1 * RV1 * RV1;
      const double GTT = RV1 - p.TT * RV3, GTS = -p.RVT * p.RVS * RV3, GSS = RV1 - p.SS * RV3;
      const double mr = L.mu * L.rhoN;
      g.A1 = mr * p.RVT * RV1;
      g.A2 = mr * p.RVS * RV1;
      g.A4 = GTT * L.rhoT * p.Radius;
      g.A7 = GTS * L.rhoT * p.Radius;
      g.A8 = GSS * L.rhoT * p.Radius;
      g.B1 = -L.mu * p.RVT * RV1;
      g.B2 = -L.mu * p.RVS * RV1;
      g.B4 = 1.0 - GTT * p.Radius;
      g.B7 = -GTS * p.Radius;
      g.B8 = 1.0 - GSS * p.Radius;
    } else {
      g.A1 = g.A2 = g.B1 = g.B2 = 0;
    }
    const double Bt[3] = {g.B1, g.B4, g.B7}, Bs[3] = {g.B2, g.B7, g.B8};
#pragma unroll
    for (int j = 0; j < 3; j++) {
      G[1 + 3 * j] = (g.A1 * M[3 * j] + g.A4 * M[1 + 3 * j] + g.A7 * M[2 + 3 * j]) + Bt[j];
      G[2 + 3 * j] = (g.A2 * M[3 * j] + g.A7 * M[1 + 3 * j] + g.A8 * M[2 + 3 * j]) + Bs[j];
    }
  }
}

// |q| and 1 / |q| as newton_damped uses them
struct LocalNorm {
  double qq;    // |q|^2
  LocalLimit lim;
};
__device__ __forceinline__ double local_nrel(const LocalNorm& m) {
  const double nq = lsqrt64(m.qq);
  return ie_lt_pos(DBL_EPSILON, nq) ? ldiv64(1.0, nq) : 1.0;
}
__device__ __forceinline__ bool residual_below(const LocalNorm& m, double FF, double tol) {
  const int c = below_limit(m.lim, FF);
  return c >= 0 ? c != 0 : ie_lt(lsqrt64(FF) * local_nrel(m), tol);
}

// Damped Newton from r; p holds the velocity at r on entry and the point at
// the final r on exit (its residual is sqrt(p.FF) / |q|).
__device__ __forceinline__ void newton_damped64(LocalProblem<double>& L, double r[3], AcPoint& p,
                                                const LocalNorm& nm) {
  const double E = DBL_EPSILON;
  const double m1 = 0.1, m2 = 0.9, inf = 1e20;
  AcGrad g = {};
  p.F[0] = p.F[1] = p.F[2] = 0;
  ac_eval64(L, r, p);
  if (residual_below(nm, p.FF, L.tol)) return;
  for (int inew = 1; inew < L.newton_max; ++inew) {
    L.n_newton++;
    double G[9], dR[3] = {p.F[0], p.F[1], p.F[2]};
    ac_matrix64(L, p, g, G);
    {
      double Gm[9];
#pragma unroll
      for (int e = 0; e < 9; e++) Gm[e] = -G[e];
      // a singular matrix: no step, and the residual stands
      if (solve3x3<double>(Gm, dR)) break;
    }
    // Goldstein-Price line search on |F|^2 / 2: dq its slope along dR
    const double F0[3] = {p.F[0], p.F[1], p.F[2]}, FF0 = p.FF;
    float df = 0.f, Sf = 0.f;
    {
      const float x0 = ie_float_signed(dR[0]), x1 = ie_float_signed(dR[1]), x2 = ie_float_signed(dR[2]);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const float f = ie_float_signed(F0[i]);
        const float a = f * ie_float_signed(G[i]) * x0, b = f * ie_float_signed(G[i + 3]) * x1,
                    d = f * ie_float_signed(G[i + 6]) * x2;
        df += a + b + d;
        Sf += fabsf(a) + fabsf(b) + fabsf(d);
      }
    }
    double alpha = 1, amin = 0, amax = inf;
    double rt[3];
    bool accepted = false;
    for (int it = 0; it < L.ls_max; it++) {
      L.n_ls++;
      // the first trial's step is dR itself
      const bool one = it == 0;
#pragma unroll
      for (int i = 0; i < 3; i++) rt[i] = r[i] + (one ? dR[i] : alpha * dR[i]);
      velocity64(L, rt, p.v);
      ac_eval64(L, rt, p);
      const double D = p.FF - FF0;
      int ok = one ? search_clear(0.5f * ie_float_signed(D), df, Sf) : -1;
      if (ok < 0) {
        double gd[3];
#pragma unroll
        for (int i = 0; i < 3; i++) gd[i] = G[i] * dR[0] + G[i + 3] * dR[1] + G[i + 6] * dR[2];
        const double dq = F0[0] * gd[0] + F0[1] * gd[1] + F0[2] * gd[2];
        double slope = 0.5 * p.FF - 0.5 * FF0;
        if (!one) slope = ldiv64(slope, alpha);
        ok = (ie_le(m2 * dq, slope) ? 1 : 0) | (ie_le(slope, m1 * dq) ? 2 : 0);
      }
      if (ok == 3) {
        accepted = true;
        break;
      }
      if (!(ok & 1))
        amin = alpha;
      else
        amax = alpha;
      if (ie_lt(alpha, inf))
        alpha = 0.5 * (amin + amax);
      else
        alpha = 10 * alpha;
    }
    if (accepted) {
      r[0] = rt[0];
      r[1] = rt[1];
      r[2] = rt[2];
    } else {
#pragma unroll
      for (int i = 0; i < 3; i++) r[i] = r[i] + alpha * dR[i];
      velocity64(L, r, p.v);
      ac_eval64(L, r, p);
    }
    if (residual_below(nm, p.FF, L.tol)) return;
    // |dR| is at least its largest component
    if (ie_lt(ie_abs(dR[0]), 10 * E) && ie_lt(ie_abs(dR[1]), 10 * E) && ie_lt(ie_abs(dR[2]), 10 * E) &&
        ie_lt(lsqrt64(dR[0] * dR[0] + dR[1] * dR[1] + dR[2] * dR[2]), 10 * E))
      return;
  }
}

// local_error <= tol without evaluating it, for a point clearly inside the
// cone: the projection there is the identity, so the error's components are
// v_N + mu |v_T| and v_T, each to a few units of the last place of r.
__device__ __forceinline__ bool error_clear(const LocalLimit& l, float r0, float rt, float v0, float vt, float mu) {
  const float B = v0 + (mu + 1.f) * vt + 1e-15f * (r0 + rt);
  return l.plain && r0 > 1e-30f && v0 + (mu + 2.f) * vt < 1e-3f * r0 && vt < 1e-3f * mu * r0 &&
         mu < 1e3f && rt < 0.99f * mu * r0 &&
         B * B < 0.5f * l.lim2;
}

// local_error with the velocity v = M r + q given; e2 its square times |q|^2
__device__ __forceinline__ double local_error64(const LocalNorm& m, double e2) {
  double e = lsqrt64(e2);
  const double nq = lsqrt64(m.qq);
  if (ie_lt_pos(DBL_EPSILON, nq)) e = ldiv64(e, nq);
  return e;
}

// The PLI loop; v holds the velocity at r on entry and on exit.
__device__ __forceinline__ void pli_solve64(LocalProblem<double>& L, double r[3], double v[3]) {
  const double mu = L.mu;
  double rho = L.rho_pli, rho_k = rho;
  double localerror = 1, localerror_k;
  const double tau = 2.0 / 3.0, tauinv = 3.0 / 2.0, Lc = 0.9, Lmin = 0.3;
  int localiter = 0;
  while (ie_lt(L.tol, localerror) && (localiter < L.pli_max)) {
    localiter++;
    L.n_pli++;
    localerror_k = localerror;
    const double r_k[3] = {r[0], r[1], r[2]}, v_k[3] = {v[0], v[1], v[2]};
    int ls = 0;
    bool success = false;
    double ra1 = 0, a2 = 0;
    rho_k = ldiv64(rho, tau);
    const double normUT = lsqrt64(v_k[1] * v_k[1] + v_k[2] * v_k[2]);
    const double vn = v_k[0] + mu * normUT;
    while (!success && (ls < 10)) {
      rho_k = rho_k * tau;
      r[0] = r_k[0] - rho_k * vn;
      r[1] = r_k[1] - rho_k * v_k[1];
      r[2] = r_k[2] - rho_k * v_k[2];
      project_cone<double>(r, mu);
      velocity64(L, r, v);
      const double a0 = v_k[0] - v[0], a1 = v_k[1] - v[1], b2 = v_k[2] - v[2];
      ra1 = rho_k * lsqrt64(a0 * a0 + a1 * a1 + b2 * b2);
      const double c0 = r_k[0] - r[0], c1 = r_k[1] - r[1], c2 = r_k[2] - r[2];
      a2 = lsqrt64(c0 * c0 + c1 * c1 + c2 * c2);
      success = ie_le(ra1, Lc * a2);
      ls++;
    }
    localerror = unitary_error2<double>(r, v, mu);
    if (ie_lt(ra1, Lmin * a2) && ie_lt(localerror, localerror_k))
      rho = rho_k * tauinv;
    else
      rho = rho_k;
  }
  L.rho_pli = rho;
  L.residual = localerror;
}

__device__ __forceinline__ bool finite64(double x) {
  return ((uint32_t)(ie_bits(x) >> 52) & 0x7ffu) != 0x7ffu;
}

// local_solve of fc3dgpu_local.cuh
template <>
__device__ __forceinline__ void local_solve<double>(LocalProblem<double>& L, double r[3]) {
  if (ie_lt(-DBL_EPSILON, L.q[0])) {
    r[0] = 0;
    r[1] = 0;
    r[2] = 0;
    L.residual = 0;
    return;
  }
  LocalNorm nm;
  nm.qq = L.q[0] * L.q[0] + L.q[1] * L.q[1] + L.q[2] * L.q[2];
  nm.lim = local_limit(nm.qq, L.tol);
  double rb[3] = {r[0], r[1], r[2]};
  AcPoint p;
  velocity64(L, r, p.v);
  double cur = 0;          // natural-map error of rb, once known
  // pass 0: Newton; pass 1, when its result is not good enough: PLI, then
  // Newton again from the better reaction
  for (int pass = 0;; pass++) {
    if (pass == 1) {
      pli_solve64(L, r, p.v);
      const double e = local_error64(nm, unitary_error2<double>(r, p.v, L.mu));
      if (finite64(L.residual) && (ie_le(e, L.tol) || ie_le(e, cur))) {
        cur = e;
        rb[0] = r[0];
        rb[1] = r[1];
        rb[2] = r[2];
      } else {
        r[0] = rb[0];
        r[1] = rb[1];
        r[2] = rb[2];
        velocity64(L, r, p.v);
      }
      if (ie_lt(cur, L.tol)) break;
    }
    newton_damped64(L, r, p, nm);
    L.slip = p.zone == 1;
    if (L.mode == 1) {
      // damped Newton alone: a non-finite result keeps the incoming reaction
      if (!(finite64(r[0]) && finite64(r[1]) && finite64(r[2]))) {
        r[0] = rb[0];
        r[1] = rb[1];
        r[2] = rb[2];
      }
      L.residual = lsqrt64(p.FF) * local_nrel(nm);
      return;
    }
    // the residual sqrt(p.FF) / |q| is finite with p.FF
    const bool good = finite64(p.FF);
    if (good) {
      const float vt = ie_float(p.v[1]) + ie_float(p.v[2]), rt = ie_float(r[1]) + ie_float(r[2]);
      const float r0 = ie_float_signed(r[0]);
      if (error_clear(nm.lim, r0, rt, ie_float(p.v[0]), vt, ie_float(L.mu))) {
        cur = 0;  // met: below the tolerance, the value is not used
        break;
      }
    }
    const double e2 = unitary_error2<double>(r, p.v, L.mu);
    if (good && below_limit(nm.lim, e2) == 1) {
      cur = 0;
      break;
    }
    const double e = local_error64(nm, e2);
    if (good && ie_le(e, L.tol)) {
      cur = e;
      break;
    }
    if (pass == 0) {
      double vb[3];
      velocity64(L, rb, vb);
      cur = local_error64(nm, unitary_error2<double>(rb, vb, L.mu));
    }
    if (good && ie_le(e, cur)) {
      cur = e;
      rb[0] = r[0];
      rb[1] = r[1];
      rb[2] = r[2];
    } else {
      r[0] = rb[0];
      r[1] = rb[1];
      r[2] = rb[2];
      velocity64(L, r, p.v);
    }
    // a NaN error ends the solve as a met tolerance does
    if (pass == 1 || !ie_le(L.tol, cur) || ie_le(cur, L.tol)) break;
  }
  L.residual = cur;
}

}  // namespace fc3dgpu
