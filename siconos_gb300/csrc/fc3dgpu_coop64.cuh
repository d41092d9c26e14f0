// The FP64 one-contact solver on three lanes a contact.
//
// What bounds it: as in fc3dgpu_local64.cuh an FP64 warp instruction costs 64
// to 76 cycles of its SM quarter whatever its lanes do.  When a colour has
// fewer contacts than the SM quarters have lanes, one contact a lane leaves
// lanes (and whole quarters) idle while the longest local solve runs; here
// lane i of a group of three holds component i of every vector and row i of
// every matrix, ten contacts a warp, so a Newton iteration takes 40 FP64
// instructions (57 with a slipping contact in the warp) instead of 68 (128).
// The control flow is the same for the whole warp, loops running until its
// last contact is done: an instruction of a finished contact costs nothing,
// and the exchanges are plain full-warp shuffles.
//
// Every value is formed by the operations and in the order of
// fc3dgpu_local64.cuh, so the bits are the same.
#pragma once
#include "fc3dgpu_local64.cuh"

namespace fc3dgpu {

#define FC3D_COOP_GROUPS 10  // contacts of a warp (lanes 30 and 31 idle)

// The lane's place: component i of the group whose first lane is `base`.
struct CoopLane {
  int i, base;
};

__device__ __forceinline__ double coop_get(double x, int lane) { return __shfl_sync(0xffffffffu, x, lane); }
__device__ __forceinline__ void coop_all(const CoopLane& c, double x, double out[3]) {
  out[0] = coop_get(x, c.base);
  out[1] = coop_get(x, c.base + 1);
  out[2] = coop_get(x, c.base + 2);
}
// (x_0 + x_1) + x_2
__device__ __forceinline__ double coop_sum(const CoopLane& c, double x) {
  double a[3];
  coop_all(c, x, a);
  return a[0] + a[1] + a[2];
}
// sqrt(x_1^2 + x_2^2) from the squares
__device__ __forceinline__ double coop_norm_t(const CoopLane& c, double sq) {
  return coop_get(sq, c.base + 1) + coop_get(sq, c.base + 2);
}
__device__ __forceinline__ bool coop_any(bool p) { return __any_sync(0xffffffffu, p); }

struct CoopProblem {
  double M[9];  // the whole diagonal block
  double m0, m1, m2;  // its row i
  double q;     // component i
  double mu, rho_i, rhoN, rhoT;  // rho_i: rhoN for component 0, rhoT for 1 and 2
};

__device__ __forceinline__ double coop_velocity(const CoopLane& c, const CoopProblem& P, double r) {
  double x[3];
  coop_all(c, r, x);
  return P.q + P.m0 * x[0] + P.m1 * x[1] + P.m2 * x[2];
}

// project_cone<double>, component i
__device__ __forceinline__ double coop_project(const CoopLane& c, double w, double mu) {
  const double normT = ie_sqrt(coop_norm_t(c, w * w));
  const double w0 = coop_get(w, c.base), mn = mu * normT;
  const bool zero = ie_le(mn, -w0);
  const bool out = !zero && !ie_le(normT, mu * w0);
  if (coop_any(out)) {
    const double x0 = ie_div(mn + w0, mu * mu + 1.0);
    const double xt = ie_div(mu * x0 * w, out ? normT : 1.0);
    if (out) w = c.i == 0 ? x0 : xt;
  }
  return zero ? 0.0 : w;
}

// unitary_error2<double>
__device__ __forceinline__ double coop_error2(const CoopLane& c, double r, double u, double mu) {
  const double nt = mu * ie_sqrt(coop_norm_t(c, u * u));
  double w = r - u;
  if (c.i == 0) w = w - nt;
  w = r - coop_project(c, w, mu);
  return coop_sum(c, w * w);
}

// AcPoint, component i
struct CoopPoint {
  double v, F, FF;
  double RV, sq;  // r - rho v and its square
  double RV1, Radius;
  bool contact;
  int zone;
};

__device__ __forceinline__ void coop_eval(const CoopLane& c, const CoopProblem& P, double r, CoopPoint& p) {
  const double pv = P.rho_i * p.v;
  p.RV = r - pv;
  p.sq = p.RV * p.RV;
  const double RVN = coop_get(p.RV, c.base);
  const double s = coop_norm_t(c, p.sq);
  p.contact = ie_positive(RVN);
  p.Radius = p.contact ? P.mu * RVN : 0.0;
  const int clear = slip_clear(s, p.Radius);
  p.zone = 0;
  double RV = s;
  if (coop_any(clear == 1)) {
    const double x = lsqrt64(s);
    if (clear == 1) RV = x;
  }
  if (clear != 0) p.zone = slip_zone(RV, p.Radius);
  double F = p.zone == 0 ? pv : (p.zone == 2 ? r : p.F);
  if (coop_any(p.zone == 1)) {
    const double RV1 = ldiv64(1.0, p.zone == 1 ? RV : 1.0);
    const double Fs = r - p.Radius * p.RV * RV1;
    if (p.zone == 1) {
      p.RV1 = RV1;
      F = Fs;
    }
  }
  p.F = c.i == 0 ? (p.contact ? pv : r) : F;
  p.FF = coop_sum(c, p.F * p.F);
}

// Row i of the gradients A and B (columns 0, i and the other tangent j);
// kept in the undefined zone.
struct CoopGrad {
  double A0, Ai, Aj, B0, Bi, Bj;
};

// Row i of G = A M + B
__device__ __forceinline__ void coop_matrix(const CoopLane& c, const CoopProblem& P, const CoopPoint& p, CoopGrad& g,
                                            double G[3]) {
  const bool n = c.i == 0;
  if (coop_any(p.zone == 1 || p.zone == 3)) {
    const double RV1 = p.RV1, RV3 = RV1 * RV1 * RV1;
    const double Gii = RV1 - p.sq * RV3;
    const double Gij = -coop_get(p.RV, c.base + 1) * coop_get(p.RV, c.base + 2) * RV3;
    const double A0 = P.mu * P.rhoN * p.RV * RV1, B0 = -P.mu * p.RV * RV1;
    const double Ai = Gii * P.rhoT * p.Radius, Aj = Gij * P.rhoT * p.Radius;
    const double Bi = 1.0 - Gii * p.Radius, Bj = -Gij * p.Radius;
    if (p.zone == 1) {
      g.A0 = A0;
      g.Ai = Ai;
      g.Aj = Aj;
      g.B0 = B0;
      g.Bi = Bi;
      g.Bj = Bj;
    } else {
      g.A0 = g.B0 = 0;
      if (p.zone == 0) {
        g.Ai = P.rhoT;
        g.Aj = g.Bi = g.Bj = 0;
      } else if (p.zone == 2) {
        g.Ai = g.Aj = g.Bj = 0;
        g.Bi = 1;
      }
    }
    // columns of A and B in order; row 0 is (rhoN, 0, 0) and 0, or 0 and (1, 0, 0)
    const double a0 = n ? (p.contact ? P.rhoN : 0.0) : g.A0, b0 = n ? (p.contact ? 0.0 : 1.0) : g.B0;
    const double a1 = n ? 0.0 : (c.i == 1 ? g.Ai : g.Aj), a2 = n ? 0.0 : (c.i == 1 ? g.Aj : g.Ai);
    const double b1 = n ? 0.0 : (c.i == 1 ? g.Bi : g.Bj), b2 = n ? 0.0 : (c.i == 1 ? g.Bj : g.Bi);
    G[0] = (a0 * P.M[0] + a1 * P.M[1] + a2 * P.M[2]) + b0;
    G[1] = (a0 * P.M[3] + a1 * P.M[4] + a2 * P.M[5]) + b1;
    G[2] = (a0 * P.M[6] + a1 * P.M[7] + a2 * P.M[8]) + b2;
  } else {
    // every contact of the warp sticks or separates: rho_i times row i of M,
    // or row i of the identity
    const bool unit = n ? !p.contact : p.zone == 2;
    const double g0 = P.rho_i * P.m0, g1 = P.rho_i * P.m1, g2 = P.rho_i * P.m2;
    G[0] = unit ? (c.i == 0 ? 1.0 : 0.0) : g0;
    G[1] = unit ? (c.i == 1 ? 1.0 : 0.0) : g1;
    G[2] = unit ? (c.i == 2 ? 1.0 : 0.0) : g2;
    g.A0 = g.B0 = 0;
    g.Ai = unit ? 0.0 : P.rhoT;
    g.Aj = g.Bj = 0;
    g.Bi = unit ? 1.0 : 0.0;
  }
}

// solve3x3<double> of the system with rows -G, right-hand side F (component
// i each); x: the whole solution in every lane.  True when singular.
__device__ __forceinline__ bool coop_solve(const CoopLane& c, const double G[3], double F, double x[3]) {
  const double E = DBL_EPSILON;
  const double a0 = -G[0], a1 = -G[1], a2 = -G[2];
  double col[3];
  coop_all(c, a0, col);
  const double aa0 = ie_abs(col[0]), aa1 = ie_abs(col[1]), aa2 = ie_abs(col[2]);
  const bool c01 = ie_le_pos(aa1, aa0), c02 = ie_le_pos(aa2, aa0), c12 = ie_le_pos(aa2, aa1);
  const int p1 = c01 ? (c02 ? 0 : 2) : (c12 ? 1 : 2);
  const int pl = c.base + p1, pm = c.base + (p1 == 0 ? 1 : 0), pn = c.base + (p1 == 2 ? 1 : 2);
  const double l0 = p1 == 0 ? col[0] : (p1 == 1 ? col[1] : col[2]);
  const double l1 = coop_get(a1, pl), l2 = coop_get(a2, pl), bl = coop_get(F, pl);
  const LDen d0 = lden(l0);
  const double f0 = ldiv64(a0, d0);
  const double e1 = a1 - f0 * l1, e2 = a2 - f0 * l2, eb = F - f0 * bl;
  const double lm1 = coop_get(e1, pm), lm2 = coop_get(e2, pm), bm = coop_get(eb, pm);
  const double ln1 = coop_get(e1, pn), ln2 = coop_get(e2, pn), bn = coop_get(eb, pn);
  const bool mn = ie_le_pos(ie_abs(ln1), ie_abs(lm1));
  const double u1 = mn ? lm1 : ln1, u2 = mn ? lm2 : ln2, ub = mn ? bm : bn;
  const double w1 = mn ? ln1 : lm1, w2 = mn ? ln2 : lm2, wb = mn ? bn : bm;
  const LDen d1 = lden(u1);
  const double f = ldiv64(w1, d1);
  x[2] = ldiv64(wb - f * ub, w2 - f * u2);
  x[1] = ldiv64(ub - u2 * x[2], d1);
  x[0] = ldiv64(bl - x[1] * l1 - x[2] * l2, d0);
  return ie_le_pos(ie_abs(l0), E) || ie_lt_pos(ie_abs(u1), E);
}

// Work of one local solve, as LocalProblem's counters.
struct CoopCount {
  int newton, pli, ls;
  bool slip;  // the last Newton ended at a slipping point
};

// residual_below, the exact form only when some group of `act` needs it
__device__ __forceinline__ bool coop_below(const LocalNorm& m, bool act, double FF, double tol) {
  const int k = below_limit(m.lim, FF);
  bool below = k == 1;
  if (coop_any(act && k < 0)) {
    const double nq = lsqrt64(m.qq);
    const bool has = ie_lt_pos(DBL_EPSILON, nq);
    const double inv = ldiv64(1.0, has ? nq : 1.0);
    const bool exact = ie_lt(lsqrt64(FF) * inv, tol);
    if (k < 0) below = exact;
  }
  return below;
}

// newton_damped64 for the groups with `act`; the others keep r and p.
__device__ __forceinline__ void coop_newton(const CoopLane& c, const CoopProblem& P, bool act, int newton_max,
                                            int ls_max, double tol, const LocalNorm& nm, double& r, CoopPoint& p,
                                            CoopCount& n) {
  const double E = DBL_EPSILON;
  const double m1 = 0.1, m2 = 0.9, inf = 1e20;
  CoopGrad g = {};
  {
    CoopPoint t = p;
    t.F = 0;
    coop_eval(c, P, r, t);
    if (act) p = t;
  }
  // (collectives never stand behind a lane's own condition)
  const bool below0 = coop_below(nm, act, p.FF, tol);
  bool run = act && !below0;
  for (int inew = 1; inew < newton_max && coop_any(run); ++inew) {
    if (run) n.newton++;
    double G[3], x[3];
    coop_matrix(c, P, p, g, G);
    if (coop_solve(c, G, p.F, x)) run = false;
    const double dR = c.i == 0 ? x[0] : (c.i == 1 ? x[1] : x[2]);
    float df, Sf;
    {
      const float f = ie_float_signed(p.F);
      const float a = f * ie_float_signed(G[0]) * ie_float_signed(x[0]),
                  b = f * ie_float_signed(G[1]) * ie_float_signed(x[1]),
                  d = f * ie_float_signed(G[2]) * ie_float_signed(x[2]);
      const float e = a + b + d, S = fabsf(a) + fabsf(b) + fabsf(d);
      df = __shfl_sync(0xffffffffu, e, c.base) + __shfl_sync(0xffffffffu, e, c.base + 1) +
           __shfl_sync(0xffffffffu, e, c.base + 2);
      Sf = __shfl_sync(0xffffffffu, S, c.base) + __shfl_sync(0xffffffffu, S, c.base + 1) +
           __shfl_sync(0xffffffffu, S, c.base + 2);
    }
    double alpha = 1, amin = 0, amax = inf;
    CoopPoint t = p;   // the trial point
    double rt = r;
    bool pending = run;  // still searching
    for (int it = 0; it < ls_max && coop_any(pending); it++) {
      if (pending) n.ls++;
      const double ra = r + (it == 0 ? dR : alpha * dR);
      CoopPoint s = t;
      s.v = coop_velocity(c, P, ra);
      coop_eval(c, P, ra, s);
      const double D = s.FF - p.FF;
      int ok = it == 0 ? search_clear(0.5f * ie_float_signed(D), df, Sf) : -1;
      if (coop_any(pending && ok < 0)) {
        const double dq = coop_sum(c, p.F * (G[0] * x[0] + G[1] * x[1] + G[2] * x[2]));
        double slope = 0.5 * s.FF - 0.5 * p.FF;
        if (it > 0) slope = ldiv64(slope, alpha);
        if (ok < 0) ok = (ie_le(m2 * dq, slope) ? 1 : 0) | (ie_le(slope, m1 * dq) ? 2 : 0);
      }
      if (pending) {
        t = s;
        rt = ra;
        if (ok == 3) {
          pending = false;
        } else {
          if (!(ok & 1))
            amin = alpha;
          else
            amax = alpha;
          if (ie_lt(alpha, inf))
            alpha = 0.5 * (amin + amax);
          else
            alpha = 10 * alpha;
        }
      }
    }
    if (coop_any(pending)) {
      // no trial accepted: the last step length, evaluated
      const double ra = r + alpha * dR;
      CoopPoint s = t;
      s.v = coop_velocity(c, P, ra);
      coop_eval(c, P, ra, s);
      if (pending) {
        t = s;
        rt = ra;
      }
    }
    if (run) {
      r = rt;
      p = t;
    }
    const bool below = coop_below(nm, run, p.FF, tol);
    run = run && !below;
    const bool small = ie_lt(ie_abs(x[0]), 10 * E) && ie_lt(ie_abs(x[1]), 10 * E) && ie_lt(ie_abs(x[2]), 10 * E);
    if (coop_any(run && small) && small && ie_lt(lsqrt64(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]), 10 * E))
      run = false;
  }
}

// local_error64 from the squared error
__device__ __forceinline__ double coop_local_error(const LocalNorm& m, double e2) {
  const double e = lsqrt64(e2), nq = lsqrt64(m.qq);
  const bool has = ie_lt_pos(DBL_EPSILON, nq);
  const double en = ldiv64(e, has ? nq : 1.0);
  return has ? en : e;
}

// pli_solve64 for the groups with `act`
__device__ __forceinline__ void coop_pli(const CoopLane& c, const CoopProblem& P, bool act, int pli_max, double tol,
                                         double& rho, double& r, double& v, double& res, CoopCount& n) {
  double localerror = 1;
  const double tau = 2.0 / 3.0, tauinv = 3.0 / 2.0, Lc = 0.9, Lmin = 0.3;
  bool run = act && ie_lt(tol, localerror);
  for (int iter = 0; iter < pli_max && coop_any(run); iter++) {
    if (run) n.pli++;
    const double r_k = r, v_k = v, before = localerror;
    double rho_k = ldiv64(rho, tau);
    const double nt = P.mu * lsqrt64(coop_norm_t(c, v_k * v_k));
    const double vn = c.i == 0 ? v_k + nt : v_k;
    bool search = run;
    double ra1 = 0, a2 = 0;
    for (int ls = 0; ls < 10 && coop_any(search); ls++) {
      const double rk = rho_k * tau;
      const double rn = coop_project(c, r_k - rk * vn, P.mu);
      const double vv = coop_velocity(c, P, rn);
      const double dv = v_k - vv, dr = r_k - rn;
      const double x1 = rk * lsqrt64(coop_sum(c, dv * dv)), x2 = lsqrt64(coop_sum(c, dr * dr));
      if (search) {
        rho_k = rk;
        r = rn;
        v = vv;
        ra1 = x1;
        a2 = x2;
        search = !ie_le(ra1, Lc * a2);
      }
    }
    const double e = coop_error2(c, r, v, P.mu);
    const double up = rho_k * tauinv;
    if (run) {
      localerror = e;
      rho = ie_lt(ra1, Lmin * a2) && ie_lt(localerror, before) ? up : rho_k;
    }
    run = run && ie_lt(tol, localerror);
  }
  if (act) res = localerror;
}

// local_solve<double> (mode 0, no take-off) of one contact a group: P.q the
// local q, r the reaction (component i each), rho_pli its PLI step; `act`
// false leaves a group out.  Returns the local residual (0 stands for one
// below the tolerance).
template <typename Args>
__device__ __forceinline__ double coop_local_solve(const CoopLane& c, const CoopProblem& P, bool act, const Args& a,
                                                   double tol, double& r, double& rho_pli, CoopCount& n) {
  LocalNorm nm;
  nm.qq = coop_sum(c, P.q * P.q);
  nm.lim = local_limit(nm.qq, tol);
  double rb = r, cur = 0, res = 0;
  CoopPoint p = {};
  p.v = coop_velocity(c, P, r);
  // pass 0: Newton; 1: PLI; 2: Newton again (the last two for the contacts
  // that the first does not solve)
  bool more = act;
  for (int pass = 0; pass < 3 && coop_any(more); pass++) {
    bool good, met = false;
    if (pass == 1) {
      coop_pli(c, P, more, a.pli_max, tol, rho_pli, r, p.v, res, n);
      good = finite64(res);
    } else {
      coop_newton(c, P, more, a.newton_max, a.ls_max, tol, nm, r, p, n);
      if (more) n.slip = p.zone == 1;
      good = finite64(p.FF);
      const float vi = ie_float(p.v), ri = ie_float_signed(r);
      const float v0 = __shfl_sync(0xffffffffu, vi, c.base), r0 = __shfl_sync(0xffffffffu, ri, c.base);
      const float vt = __shfl_sync(0xffffffffu, vi, c.base + 1) + __shfl_sync(0xffffffffu, vi, c.base + 2);
      const float rt = fabsf(__shfl_sync(0xffffffffu, ri, c.base + 1)) + fabsf(__shfl_sync(0xffffffffu, ri, c.base + 2));
      met = good && error_clear(nm.lim, r0, rt, v0, vt, ie_float(P.mu));
    }
    if (coop_any(more && !met)) {
      const double e2 = coop_error2(c, r, p.v, P.mu);
      if (!met && pass != 1) met = good && below_limit(nm.lim, e2) == 1;
      if (coop_any(more && !met)) {
        const double e = coop_local_error(nm, e2);
        const bool low = good && ie_le(e, tol);
        if (coop_any(more && !met)) {
          const double vb = coop_velocity(c, P, rb);
          if (pass == 0 && coop_any(more && !met && !low)) {
            const double eb = coop_local_error(nm, coop_error2(c, rb, vb, P.mu));
            cur = eb;
          }
          if (more && !met) {
            if (low || (good && ie_le(e, cur))) {
              cur = e;
              rb = r;
            } else {
              r = rb;
              p.v = vb;
            }
            // a NaN error ends the solve as a met tolerance does
            if (pass == 0 ? !ie_le(tol, cur) || ie_le(cur, tol) : pass == 1 && ie_lt(cur, tol)) more = false;
          }
        }
      }
    }
    if (met) {
      if (more) cur = 0;
      more = false;
    }
  }
  return cur;
}

}  // namespace fc3dgpu
