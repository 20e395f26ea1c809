// k_adi.cuh -- the diagonalised ADI operator arc2d with pentadiagonal line
// inversions (src/lhs.f:817-1057 with lhsinv :1536-1816 and pentadag
// :1819-1873; ilhs = 2) or the upwind-split tridiagonal ones (lhsinv_up
// :1333-1533; ilhs = 3).
//
// The reference converts q to primitive variables in place, multiplies s by
// T_xi^-1, inverts a scalar pentadiagonal system per j-line and variable,
// multiplies by N^-1, inverts per k-line, multiplies by T_eta and converts
// q back.  Here q is never rewritten: the primitive values and every
// per-cell factor are kept in scratch arrays (cell-parallel kernels) and the
// rows of the line systems are assembled per cell in gather form
// (adi_row_cell).  A line has three systems, since variables 1 and 2 share
// one matrix; each is solved with pentadag's recurrences for its one or two
// right-hand sides, 32 lines along j by a CTA through staged tiles
// (k_lines.cuh), a line along k by one thread.  In FP64 the conservative round
// trip of q (:853-860, :1047-1054) is applied at the end so q leaves with the
// reference's bits.
#pragma once
#include "dev_common.cuh"
#include "k_lines.cuh"
#include "launch.h"

namespace ot2d {

// scratch arrays of one slice (stride S.wstride).  Rows of the line systems
// (adi_row_cell): A_RB / A_RD one array per system; pentadiagonal (ilhs 2)
// A_RA, A_RE, A_RC shared by the systems; tridiagonal (ilhs 3) A_RA = 0 =
// A_RE and the diagonals of the three systems in A_RA, A_RE, A_RC.  A_EM: per
// system the second super-diagonal of pentadag's forward sweep (the first
// replaces A_RD); A_DN, the dissipation's diagonal, is used before it.
enum ADIw { A_P = 0, A_QX, A_QY, A_CX, A_CY, A_UV, A_VN, A_GE, A_U, A_V, A_E, A_D2P, A_RA, A_RE, A_RC,
            A_RB, A_RD = A_RB + 3, A_EM = A_RD + 3, A_N = A_EM + 3, A_DN = A_EM };
static_assert(A_N <= ADI_NSCRATCH, "ADI scratch layout");

__device__ __forceinline__ bool adi_slice(const ot2d_params& p) { return p.ilhs == 2 || p.ilhs == 3; }

// line view of direction dir (0: j lines, m = j, n = k; 1: k lines, m = k, n = j)
__device__ __forceinline__ int64_t adi_at(int jd, int dir, int m, int n) { return dir == 0 ? at(jd, m, n) : at(jd, n, m); }

// bSq = Mp**2/(bt - Mp**2 (bt-1)) of cell o (arc2d_precon, lhsinv)
template <class R>
__device__ __forceinline__ R adi_bsq(const Slice<R>& S, int64_t o) {
  const R btv = S.bt ? S.bt[o] : (R)1.;
  return S.k_mp2 / by(btv - S.k_mp2 * (btv - (R)1));
}

// s *= tscale when `scale` (step.f:141-148), primitive variables (:853-860) and the
// T_xi^-1 multiplication with its per-cell factors (:863-917), on every
// cell of js-1..je+1 x ks-1..ke+1
template <class R>
__device__ void adi_txi_cell(const Slice<R>& S, const ot2d_params& p, int j, int k, int scale) {
  const int64_t o = at(S.jd, j, k), qs = S.qs, ws = S.wstride;
  const R gm1 = S.k_gm1, ggm1 = S.k_ggm1;
  const R q1 = S.q[o], J = S.q[(p.nq - 1) * qs + o];
  const R dj = (R)1.0 / by(q1);
  const R uu = S.q[qs + o] * dj, vv = S.q[2 * qs + o] * dj, e = S.q[3 * qs + o] * dj;
  const R rho = q1 * J;
  R s1 = S.s[o], s2 = S.s[qs + o], s3 = S.s[2 * qs + o], s4 = S.s[3 * qs + o];
  if (scale) {
    const R ts = S.tscale[o];
    s1 = s1 * ts; s2 = s2 * ts; s3 = s3 * ts; s4 = s4 * ts;
  }
  const R uv2 = (R)0.5 * (uu * uu + vv * vv);
  const R cjkl = root(ggm1 * (e - uv2));
  const R c2i = (R)1.0 / by(cjkl * cjkl);
  S.w[A_P * ws + o] = (e - uv2) * gm1 * rho;
  R rj1 = S.xx[o], rj2 = S.xy[o];
  const R ugc = S.ug ? S.ug[o] : (R)0, vgc = S.vg ? S.vg[o] : (R)0;
  // arc2d_precon (:1116, :1125) takes the contravariant velocities relative
  // to the grid before storing them; arc2d (:874-876) subtracts afterwards
  const bool pre = S.k_mp2 >= (R)0;
  const R qq1 = pre ? rj1 * (uu - ugc) + rj2 * (vv - vgc) : rj1 * uu + rj2 * vv;
  S.w[A_QX * ws + o] = pre ? qq1 : qq1 - (rj1 * ugc + rj2 * vgc);
  const R rr1 = root(sq(rj1) + sq(rj2));
  rj1 = rj1 / by(rr1); rj2 = rj2 / by(rr1);
  const R rk1 = S.yx[o], rk2 = S.yy[o];
  if (pre) {
    S.w[A_QY * ws + o] = rk1 * (uu - ugc) + rk2 * (vv - vgc);
  } else {
    const R qq2 = rk1 * uu + rk2 * vv;
    S.w[A_QY * ws + o] = qq2 - (rk1 * ugc + rk2 * vgc);
  }
  const R rr2 = root(sq(rk1) + sq(rk2));
  S.w[A_UV * ws + o] = uv2;
  S.w[A_CX * ws + o] = cjkl * rr1;
  S.w[A_CY * ws + o] = cjkl * rr2;
  S.w[A_VN * ws + o] = (S.k_rmue + S.turmu[o]) / by(S.k_rey * rho);
  S.w[A_GE * ws + o] = S.k_gamma * e - gm1 * uv2;
  S.w[A_U * ws + o] = uu; S.w[A_V * ws + o] = vv; S.w[A_E * ws + o] = e;
  R a1 = s2 * uu + s3 * vv - s4;
  a1 = a1 * gm1 * c2i;
  a1 = a1 + s1 * ((R)1.0 - uv2 * gm1 * c2i);
  const R a2 = (rj1 * vv - rj2 * uu) * s1 + rj2 * s2 - rj1 * s3;
  R a3 = uv2 * s1 - s2 * uu - s3 * vv + s4;
  a3 = a3 * gm1 * c2i;
  S.s[o] = a1;
  S.s[qs + o] = a2;
  if (pre) {
    // arc2d_precon :1141-1164: the preconditioned acoustic eigenvectors
    const R bSq = adi_bsq(S, o), omb = (R)1. - bSq;
    const R cx = cjkl * rr1;
    const R X = root((omb * qq1) * (omb * qq1) + (R)4. * bSq * cx * cx) / by(rr1);
    const R Y = (R)0.5 * (omb * qq1 / by(rr1) + X);
    const R Z = (R)0.5 * (omb * qq1 / by(rr1) - X);
    const R qqmxt = qq1 + ugc * rj1 * rr1 + vgc * rj2 * rr1;
    R a4 = qqmxt * s1 / by(rr1) - rj1 * s2 - rj2 * s3;
    a4 = a4 * bSq;
    S.s[2 * qs + o] = -(Z * a3 + a4) / by(X);
    S.s[3 * qs + o] = (Y * a3 + a4) / by(X);
    return;
  }
  const R a4 = qq1 * s1 / by(rr1) - rj1 * s2 - rj2 * s3;
  S.s[2 * qs + o] = (R)0.5 * (a3 - a4 / by(cjkl));
  S.s[3 * qs + o] = (R)0.5 * (a3 + a4 / by(cjkl));
}

// spectral-radius diagonal of lhsinv (:1587-1596): d[0] = diag(m,1) =
// diag(m,2), d[1] = diag(m,3), d[2] = diag(m,4), d[3] = diag(m,nq)
template <class R>
__device__ __forceinline__ void adi_diag(const Slice<R>& S, const ot2d_params& p, int dir, int64_t o, R* d) {
  const int64_t ws = S.wstride;
  const R Mp = (R)p.Mp;
  const R btv = S.bt ? S.bt[o] : (R)1.;
  const R bSq = (Mp * Mp) / by(btv - (Mp * Mp) * (btv - (R)1));
  const R qv = S.w[(dir == 0 ? A_QX : A_QY) * ws + o], cv = S.w[(dir == 0 ? A_CX : A_CY) * ws + o];
  const R X = root(((R)1. - bSq) * qv * (((R)1. - bSq) * qv) + (R)4. * bSq * cv * cv);
  d[0] = qv;
  d[1] = (R)0.5 * ((bSq + (R)1.) * qv + X);
  d[2] = (R)0.5 * ((bSq + (R)1.) * qv - X);
  d[3] = (R)0.5 * ((bSq + (R)1.) * fabs(qv) + X) / by(S.q[(int64_t)(p.nq - 1) * S.qs + o]);
}

// pressure switch of line direction dir (:919-935, :977-993): interior of
// the line, 0 at its two ends; and diag(m,nq) of lhsinv
template <class R>
__device__ __forceinline__ void adi_d2p_cell(const Slice<R>& S, const ot2d_params& p, int dir, int m, int n, int ms,
                                             int me) {
  const int jd = S.jd; const int64_t ws = S.wstride;
  const R* P = S.w + A_P * ws;
  R v = (R)0;
  if (m > ms && m < me) {
    const R pp = P[adi_at(jd, dir, m + 1, n)], pc = P[adi_at(jd, dir, m, n)], pm = P[adi_at(jd, dir, m - 1, n)];
    v = fabs(pp - (R)2. * pc + pm);
    v = v / by(fabs(pp + (R)2. * pc + pm));
  }
  const int64_t o = adi_at(jd, dir, m, n);
  S.w[A_D2P * ws + o] = v;
  R d[4];
  adi_diag(S, p, dir, o, d);
  S.w[A_DN * ws + o] = d[3];
}

template <class R>
struct AdiRow { R a, b, c, d, e; };

// a product rounded on its own (the compiler must not fuse it with the
// addition that follows)
__device__ __forceinline__ float adi_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double adi_mul(double a, double b) { return __dmul_rn(a, b); }

// Dissipation coefficients atmp..etmp of lhsinv (:1655-1732) at line
// position m, times J (:1734-1740); the entries the reference leaves
// unassigned (both line ends, and the ones its end-point formulas skip) are
// 0.  Requires lines of at least 8 points.
template <class R>
__device__ __forceinline__ AdiRow<R> adi_coef(const Slice<R>& S, const ot2d_params& p, int dir, int m, int n, int ms,
                                              int me) {
  const int jd = S.jd; const int64_t ws = S.wstride, qs = S.qs;
  const R dis2 = (R)10.0, dis4 = (R)0.1;
  R g[5], dn[5];   // positions m-2 .. m+2
  for (int t = 0; t < 5; ++t) {
    const int mm = m - 2 + t;
    if (mm < ms || mm > me) { g[t] = (R)0; dn[t] = (R)0; continue; }
    const int64_t oo = adi_at(jd, dir, mm, n);
    g[t] = S.w[A_D2P * ws + oo];
    dn[t] = S.w[A_DN * ws + oo];
  }
  auto G = [&](int dm) { return g[dm + 2]; };
  auto D = [&](int dm) { return dn[dm + 2]; };
  R at = (R)0, bt = (R)0, ct = (R)0, dt = (R)0, et = (R)0;
  if (m == me - 1) {
    const R c2 = ((G(0))) * dis2, c2m = (R)0.5 * ((G(0) + G(-1))) * dis2;
    const R c4 = (dis4 - fmin2(dis4, (R)1. * c2)), c4m = (dis4 - fmin2(dis4, (R)1. * c2m));
    const R c4m2 = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(-2) + G(-1))));
    ct = +((D(-1) + D(0)) * ((R)3. * c4m + c2m) + (R)2. * (D(0)) * ((R)2. * c4 + c2));
    dt = -((D(-2) + D(-1)) * c4m2 + (D(0) + D(-1)) * ((R)3. * c4m + c2m));
    et = (D(-1) + D(-2)) * c4m2;
  } else if (m == me - 2) {
    const R c2 = (R)0.5 * ((G(0) + G(1))) * dis2, c2m = (R)0.5 * ((G(0) + G(-1))) * dis2;
    const R c4p = (dis4 - fmin2(dis4, (R)1. * dis2 * (G(1))));
    const R c4 = (dis4 - fmin2(dis4, (R)1. * c2)), c4m = (dis4 - fmin2(dis4, (R)1. * c2m));
    const R c4m2 = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(-2) + G(-1))));
    bt = -((R)2. * (D(1)) * c4p + (D(1) + D(0)) * ((R)3. * c4 + c2));
    ct = ((D(-1) + D(0)) * ((R)3. * c4m + c2m) + (D(1) + D(0)) * ((R)2. * c4 + c2));
    dt = -((D(-2) + D(-1)) * c4m2 + (D(0) + D(-1)) * ((R)3. * c4m + c2m));
    et = (D(-1) + D(-2)) * c4m2;
  } else if (m == ms + 1) {
    const R c2 = (R)0.5 * ((G(0) + G(1))) * dis2, c2m = ((G(0))) * dis2;
    const R c4p = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(2) + G(1))));
    const R c4 = (dis4 - fmin2(dis4, (R)1. * c2)), c4m = (dis4 - fmin2(dis4, (R)1. * c2m));
    at = (D(1) + D(2)) * c4p;
    bt = -((D(2) + D(1)) * c4p + (D(1) + D(0)) * ((R)3. * c4 + c2));
    ct = ((R)2. * (D(0)) * ((R)2. * c4m + c2m) + (D(1) + D(0)) * ((R)3. * c4 + c2));
  } else if (m == ms + 2) {
    const R c2 = (R)0.5 * ((G(0) + G(1))) * dis2, c2m = (R)0.5 * ((G(0) + G(-1))) * dis2;
    const R c4p = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(2) + G(1))));
    const R c4 = (dis4 - (R)1. * fmin2(dis4, c2)), c4m = (dis4 - fmin2(dis4, (R)1. * c2m));
    const R c4m2 = (dis4 - fmin2(dis4, (R)1. * dis2 * (G(-1))));
    at = (D(1) + D(2)) * c4p;
    bt = -((D(2) + D(1)) * c4p + (D(1) + D(0)) * ((R)3. * c4 + c2));
    ct = ((D(-1) + D(0)) * ((R)3. * c4m + c2m) + (D(1) + D(0)) * ((R)3. * c4 + c2));
    dt = -(((R)2. * D(-1)) * c4m2 + (D(0) + D(-1)) * ((R)3. * c4m + c2m));
  } else if (m >= ms + 3 && m <= me - 3) {
    const R c2 = (R)0.5 * ((G(0) + G(1))) * dis2, c2m = (R)0.5 * ((G(0) + G(-1))) * dis2;
    const R c4p = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(2) + G(1))));
    const R c4 = (dis4 - fmin2(dis4, (R)1. * c2)), c4m = (dis4 - fmin2(dis4, (R)1. * c2m));
    const R c4m2 = (dis4 - fmin2(dis4, (R).5 * dis2 * (G(-2) + G(-1))));
    at = (D(1) + D(2)) * c4p;
    bt = -((D(2) + D(1)) * c4p + (D(1) + D(0)) * ((R)3. * c4 + c2));
    ct = +((D(-1) + D(0)) * ((R)3. * c4m + c2m) + (D(1) + D(0)) * ((R)3. * c4 + c2));
    dt = -((D(-2) + D(-1)) * c4m2 + (D(0) + D(-1)) * ((R)3. * c4m + c2m));
    et = (D(-1) + D(-2)) * c4m2;
  }
  const int64_t o = adi_at(jd, dir, m, n);
  const R J = S.q[(int64_t)(p.nq - 1) * qs + o];
  return {adi_mul(at, J), adi_mul(bt, J), adi_mul(ct, J), adi_mul(dt, J), adi_mul(et, J)};
}

// The five scaled bands a1..e1 of lhsinv (:1742-1785) for system sys (0:
// variables 1 and 2, 1: variable 3, 2: variable 4) at line position m; cf:
// adi_coef of the position, dg: adi_diag
template <class R>
__device__ __forceinline__ AdiRow<R> adi_row(const Slice<R>& S, const ot2d_params& p, int dir, int sys, int m, int n,
                                            int ms, int me, const AdiRow<R>& cf, const R* dg) {
  const int jd = S.jd; const int64_t ws = S.wstride, qs = S.qs;
  const int64_t o = adi_at(jd, dir, m, n);
  const R* ts = S.tscale;
  const R di = dg[sys];
  R v1 = (R)0, v2 = (R)0, v3 = (R)0;
  if (m > ms && m < me) {
    const R* xn = dir == 0 ? S.xx : S.yx;
    const R* yn = dir == 0 ? S.xy : S.yy;
    const R* Jq = S.q + (int64_t)(p.nq - 1) * qs;
    const int64_t op = adi_at(jd, dir, m + 1, n), om = adi_at(jd, dir, m - 1, n);
    const R vnu = S.w[A_VN * ws + o];
    v1 = (xn[o] * xn[o] + yn[o] * yn[o]) / by(Jq[o]);
    v1 = v1 + (xn[op] * xn[op] + yn[op] * yn[op]) / by(Jq[op]);
    v1 = v1 * Jq[o] * vnu;
    v3 = (xn[o] * xn[o] + yn[o] * yn[o]) / by(Jq[o]);
    v3 = v3 + (xn[om] * xn[om] + yn[om] * yn[om]) / by(Jq[om]);
    v3 = v3 * Jq[o] * vnu;
    v2 = (R)0.5 * (v1 + v3);
  }
  AdiRow<R> r;
  auto T = [&](int mm) { return ts[adi_at(jd, dir, mm, n)]; };
  if (p.ilhs == 3) {
    // lhsinv_up (lhs.f:1387-1501): upwind split eigenvalues, tridiagonal
    const R* xn = dir == 0 ? S.xx : S.yx;
    const R* yn = dir == 0 ? S.xy : S.yy;
    const R eps = (R)0.05 * root(sq(xn[o]) + sq(yn[o]));
    const R fac = (R)1.05;
    const R dpl = (R)0.5 * (di + fac * root(sq(di) + sq(eps)));
    const R dmi = (R)0.5 * (di - fac * root(sq(di) + sq(eps)));
    r.a = (R)0.; r.b = (R)0.; r.c = (R)0.; r.d = (R)0.; r.e = (R)0.;
    r.b = r.b - dpl;
    r.d = r.d + dmi;
    r.c = r.c + dpl - dmi;
    r.b = r.b - (R)0.5 * v1;
    r.c = r.c + v2;
    r.d = r.d - (R)0.5 * v3;
    r.b = (m <= me - 1) ? r.b * T(m + 1) : r.b * T(m);
    r.d = (m >= ms + 1) ? r.d * T(m - 1) : r.d * T(m);
    r.c = r.c * T(m) + (R)1.0;
    return r;
  }
  r = cf;
  r.b = r.b - di * (R)0.5;
  r.d = r.d + di * (R)0.5;
  r.b = r.b - (R)0.5 * v1;
  r.c = r.c + v2;
  r.d = r.d - (R)0.5 * v3;
  r.a = (m <= me - 2) ? r.a * T(m + 2) : r.a * T(m);
  r.b = (m <= me - 1) ? r.b * T(m + 1) : r.b * T(m);
  r.d = (m >= ms + 1) ? r.d * T(m - 1) : r.d * T(m);
  r.e = (m >= ms + 2) ? r.e * T(m - 2) : r.e * T(m);
  r.c = r.c * T(m) + (R)1.0;
  return r;
}

// The rows of the three systems at line position m, for the recurrences of
// adi_forward: a step takes a(m-2), b(m-1), c(m), d(m+1) and e(m+2) of the
// reference's rows, so each is stored where it is used, with 0 where a step
// takes none (its end rows ms and me are no part of the system).  The two end
// positions correct the right-hand sides next to them (:1787-1797).
template <class R>
__device__ void adi_row_cell(const Slice<R>& S, const ot2d_params& p, int dir, int m, int n, int ms, int me) {
  const int64_t ws = S.wstride, qs = S.qs;
  const bool tri = p.ilhs == 3;
  auto put = [&](int arr, int mm, R v) { S.w[arr * ws + adi_at(S.jd, dir, mm, n)] = v; };
  AdiRow<R> cf{(R)0, (R)0, (R)0, (R)0, (R)0};
  if (!tri) cf = adi_coef(S, p, dir, m, n, ms, me);
  R dg[4];
  adi_diag(S, p, dir, adi_at(S.jd, dir, m, n), dg);
  for (int sys = 0; sys < 3; ++sys) {
    const AdiRow<R> r = adi_row(S, p, dir, sys, m, n, ms, me, cf, dg);
    if (m == ms || m == me) {
      const int mi = m == ms ? ms + 1 : me - 1;
      const R x = m == ms ? r.b : r.d;
      for (int v = sys ? sys + 1 : 0; v < (sys ? sys + 2 : 2); ++v) {
        R* sv = S.s + (int64_t)v * qs;
        const int64_t oi = adi_at(S.jd, dir, mi, n);
        sv[oi] = sv[oi] - x * sv[adi_at(S.jd, dir, m, n)] / by(r.c);
      }
      if (m == ms) put(A_RB + sys, ms + 1, (R)0);
      else put(A_RD + sys, me - 1, (R)0);
      if (!tri && sys == 0) {
        if (m == ms) { put(A_RA, ms + 1, (R)0); put(A_RA, ms + 2, (R)0); }
        else { put(A_RE, me - 1, (R)0); put(A_RE, me - 2, (R)0); }
      }
      continue;
    }
    if (m < me - 1) put(A_RB + sys, m + 1, r.b);
    if (m > ms + 1) put(A_RD + sys, m - 1, r.d);
    if (tri) {
      put(sys == 0 ? A_RA : (sys == 1 ? A_RE : A_RC), m, r.c);
    } else if (sys == 0) {
      put(A_RC, m, r.c);
      if (m < me - 2) put(A_RA, m + 2, r.a);
      if (m > ms + 2) put(A_RE, m - 2, r.e);
    }
  }
}

// pentadag's forward recurrences (:1819-1873) for NF right-hand sides: one
// row in, the modified super-diagonals (d, e) and right-hand sides (f) out
template <class R, int NF>
struct AdiForward {
  R Dp = (R)0, Dc = (R)0, Ec = (R)0, En = (R)0, f1[NF], f2[NF];
  __device__ __forceinline__ AdiForward() {
#pragma unroll
    for (int v = 0; v < NF; ++v) f1[v] = f2[v] = (R)0;
  }
  __device__ __forceinline__ void step(R a, R b, R c, R& d, R& e, R* f) {
    const R d2 = (b - a * Dp);
    const R d0 = (R)1. / by(c - d2 * Dc - a * Ec);
#pragma unroll
    for (int v = 0; v < NF; ++v) {
      f[v] = (f[v] - d2 * f1[v] - a * f2[v]) * d0;
      f2[v] = f1[v]; f1[v] = f[v];
    }
    d = (d - d2 * En) * d0;
    e = e * d0;
    Dp = Dc; Dc = d; Ec = En; En = e;
  }
};
// ... and its back substitution
template <class R, int NF>
struct AdiBackward {
  R f1[NF], f2[NF];
  __device__ __forceinline__ AdiBackward() {
#pragma unroll
    for (int v = 0; v < NF; ++v) f1[v] = f2[v] = (R)0;
  }
  __device__ __forceinline__ void step(R d, R e, R* f) {
#pragma unroll
    for (int v = 0; v < NF; ++v) {
      f[v] = f[v] - d * f1[v] - e * f2[v];
      f2[v] = f1[v]; f1[v] = f[v];
    }
  }
};

// System sys of 32 lines along j (rows k0 .. k0+31 of the mesh) by a CTA of
// JL_THREADS threads through staged tiles.  Arrays: a, b, c, d, e, f (f of
// variable 2 too); the forward pass stores d, e and f.  TRI: a = e = 0.
template <class R, bool TRI, int NF>
__device__ void adi_solve_j(const Slice<R>& S, const ot2d_params& p, int sys, int k0, R* sm) {
  const int64_t ws = S.wstride;
  R* w = S.w;
  const int var = sys ? sys + 1 : 0;
  R* const f = S.s + (int64_t)var * S.qs;
  constexpr int NA = TRI ? 3 + NF : 5 + NF, ND = TRI ? 2 : 3;   // d is array ND, then e, then f
  R* src[NA];
  R* dst[NA];
  if (TRI) {
    src[0] = w + (A_RB + sys) * ws;
    src[1] = w + (sys == 0 ? A_RA : (sys == 1 ? A_RE : A_RC)) * ws;
  } else {
    src[0] = w + A_RA * ws; src[1] = w + (A_RB + sys) * ws; src[2] = w + A_RC * ws;
    src[ND + 1] = w + A_RE * ws;
  }
  src[ND] = w + (A_RD + sys) * ws;
#pragma unroll
  for (int v = 0; v < NF; ++v) src[NA - NF + v] = f + (int64_t)v * S.qs;
#pragma unroll
  for (int a = 0; a < NA; ++a) dst[a] = src[a];
  if (!TRI) dst[ND + 1] = w + (A_EM + sys) * ws;
  constexpr unsigned OUT = ((1u << NA) - 1) & ~((1u << ND) - 1), RHS = ((1u << NF) - 1) << (NA - NF);
  AdiForward<R, NF> F;
  AdiBackward<R, NF> B;
  jl_solve<R, NA, OUT, OUT, RHS>(
      src, dst, S.jd, p.jbeg, p.jend, k0, min(32, S.kd - k0 + 1), sm,
      [&](R* t, int) {
        R f_[NF], e = TRI ? (R)0 : t[(ND + (TRI ? 0 : 1)) * JL_TILE];
#pragma unroll
        for (int v = 0; v < NF; ++v) f_[v] = t[(NA - NF + v) * JL_TILE];
        R d = t[ND * JL_TILE];
        F.step(TRI ? (R)0 : t[0], t[(ND - 2) * JL_TILE], t[(ND - 1) * JL_TILE], d, e, f_);
        t[ND * JL_TILE] = d;
        if (!TRI) t[(ND + 1) * JL_TILE] = e;
#pragma unroll
        for (int v = 0; v < NF; ++v) t[(NA - NF + v) * JL_TILE] = f_[v];
      },
      [&](R* t, int) {
        R f_[NF];
#pragma unroll
        for (int v = 0; v < NF; ++v) f_[v] = t[(NA - NF + v) * JL_TILE];
        B.step(t[ND * JL_TILE], TRI ? (R)0 : t[(ND + (TRI ? 0 : 1)) * JL_TILE], f_);
#pragma unroll
        for (int v = 0; v < NF; ++v) t[(NA - NF + v) * JL_TILE] = f_[v];
      });
}

// System sys of the line along k at column j, one thread: rows a chunk ahead
template <class R, bool TRI, int NF>
__device__ void adi_solve_k(const Slice<R>& S, const ot2d_params& p, int sys, int j) {
  constexpr int U = sizeof(R) == 4 ? 8 : 4;
  const int64_t ws = S.wstride;
  const int ks = p.kbeg, ke = p.kend, jd = S.jd;
  const int var = sys ? sys + 1 : 0;
  R* f = S.s + (int64_t)var * S.qs;
  const R* ga = S.w + A_RA * ws;
  const R* gb = S.w + (A_RB + sys) * ws;
  const R* gc = S.w + (TRI ? (sys == 0 ? A_RA : (sys == 1 ? A_RE : A_RC)) : A_RC) * ws;
  const R* ge = S.w + A_RE * ws;
  R* gd = S.w + (A_RD + sys) * ws;
  R* gem = S.w + (A_EM + sys) * ws;
  {
    AdiForward<R, NF> F;
    AdiRow<R> nr[U];
    R nf[U][NF];
    auto load = [&](int k0) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u <= ke) {
          const int64_t o = at(jd, j, k0 + u);
          nr[u] = {TRI ? (R)0 : ga[o], gb[o], gc[o], gd[o], TRI ? (R)0 : ge[o]};
#pragma unroll
          for (int v = 0; v < NF; ++v) nf[u][v] = f[(int64_t)v * S.qs + o];
        }
    };
    load(ks);
    for (int k0 = ks; k0 <= ke; k0 += U) {
      AdiRow<R> rr[U];
      R rf[U][NF];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        rr[u] = nr[u];
#pragma unroll
        for (int v = 0; v < NF; ++v) rf[u][v] = nf[u][v];
      }
      if (k0 + U <= ke) load(k0 + U);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u <= ke) {
          const int64_t o = at(jd, j, k0 + u);
          R d = rr[u].d, e = rr[u].e;
          F.step(rr[u].a, rr[u].b, rr[u].c, d, e, rf[u]);
          gd[o] = d;
          if (!TRI) gem[o] = e;
#pragma unroll
          for (int v = 0; v < NF; ++v) f[(int64_t)v * S.qs + o] = rf[u][v];
        }
    }
  }
  AdiBackward<R, NF> B;
  R nd[U], ne[U], nf[U][NF];
  auto load = [&](int k0) {   // positions k0, k0-1, ...
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k0 - u >= ks) {
        const int64_t o = at(jd, j, k0 - u);
        nd[u] = gd[o];
        ne[u] = TRI ? (R)0 : gem[o];
#pragma unroll
        for (int v = 0; v < NF; ++v) nf[u][v] = f[(int64_t)v * S.qs + o];
      }
  };
  load(ke);
  for (int k0 = ke; k0 >= ks; k0 -= U) {
    R rd[U], re[U], rf[U][NF];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rd[u] = nd[u]; re[u] = ne[u];
#pragma unroll
      for (int v = 0; v < NF; ++v) rf[u][v] = nf[u][v];
    }
    if (k0 - U >= ks) load(k0 - U);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k0 - u >= ks) {
        B.step(rd[u], re[u], rf[u]);
#pragma unroll
        for (int v = 0; v < NF; ++v) f[(int64_t)v * S.qs + at(jd, j, k0 - u)] = rf[u][v];
      }
  }
}

// N^-1 multiplication (:948-975)
template <class R>
__device__ void adi_ninv_cell(const Slice<R>& S, const ot2d_params& p, int j, int k) {
  const int64_t o = at(S.jd, j, k), qs = S.qs, ws = S.wstride;
  const R cjkl = root(S.k_ggm1 * (S.w[A_E * ws + o] - S.w[A_UV * ws + o]));
  const R rj1 = S.xx[o], rj2 = S.xy[o], rr1 = root(rj1 * rj1 + rj2 * rj2);
  const R rk1 = S.yx[o], rk2 = S.yy[o], rr2 = root(rk1 * rk1 + rk2 * rk2);
  const R a1 = (rj1 * rk1 + rj2 * rk2) / by(rr1) / by(rr2);
  const R a2 = (rj1 * rk2 - rj2 * rk1) / by(rr1) / by(rr2);
  const R s2 = S.s[qs + o], s3 = S.s[2 * qs + o], s4 = S.s[3 * qs + o];
  if (S.k_mp2 >= (R)0) {
    // arc2d_precon :1207-1231
    const R bSq = adi_bsq(S, o), omb = (R)1.0 - bSq;
    const R qx = S.w[A_QX * ws + o], qy = S.w[A_QY * ws + o], cx = S.w[A_CX * ws + o], cy = S.w[A_CY * ws + o];
    const R X = root((omb * qx) * (omb * qx) + (R)4. * bSq * cx * cx) / by(rr1);
    const R Y = (R)0.5 * (omb * qx / by(rr1) + X);
    const R Z = (R)0.5 * (omb * qx / by(rr1) - X);
    const R X1 = root((omb * qy) * (omb * qy) + (R)4. * bSq * cy * cy) / by(rr2);
    const R Y1 = (R)0.5 * (omb * qy / by(rr2) + X1);
    const R Z1 = (R)0.5 * (omb * qy / by(rr2) - X1);
    S.s[qs + o] = a1 * s2 + (Y * s3 + Z * s4) * a2 / by(bSq);
    S.s[2 * qs + o] = -(a2 * bSq * s2 - (Y * a1 - Z1) * s3 - (Z * a1 - Z1) * s4) / by(X1);
    S.s[3 * qs + o] = (a2 * bSq * s2 - (Y * a1 - Y1) * s3 - (Z * a1 - Y1) * s4) / by(X1);
    return;
  }
  const R a4 = a1 * s2 + (cjkl * s3 - cjkl * s4) * a2;
  const R a5 = (R)-0.5 * (a2 * s2 / by(cjkl) - (a1 + (R)1) * s3 + (a1 - (R)1) * s4);
  const R a6 = (R)0.5 * (a2 * s2 / by(cjkl) - (a1 - (R)1) * s3 + (a1 + (R)1) * s4);
  S.s[qs + o] = a4; S.s[2 * qs + o] = a5; S.s[3 * qs + o] = a6;
}

// T_eta multiplication (:1005-1034), the unsteady rotation term of
// :1036-1045, and (FP64) the conservative round trip of q (:1047-1054)
template <class R>
__device__ void adi_teta_cell(const Slice<R>& S, const ot2d_params& p, int j, int k) {
  const int64_t o = at(S.jd, j, k), qs = S.qs, ws = S.wstride;
  const R uu = S.w[A_U * ws + o], vv = S.w[A_V * ws + o], uv = S.w[A_UV * ws + o], ge = S.w[A_GE * ws + o];
  const R cjkl = root(S.k_ggm1 * (S.w[A_E * ws + o] - uv));
  R rk1 = S.yx[o], rk2 = S.yy[o];
  const R ugc = S.ug ? S.ug[o] : (R)0, vgc = S.vg ? S.vg[o] : (R)0;
  const bool pre = S.k_mp2 >= (R)0;
  const R qq2 = pre ? S.w[A_QY * ws + o] : S.w[A_QY * ws + o] + (rk1 * ugc + rk2 * vgc);
  const R rr2 = root(rk1 * rk1 + rk2 * rk2);
  rk1 = rk1 / by(rr2); rk2 = rk2 / by(rr2);
  const R s1 = S.s[o], s2 = S.s[qs + o], s3 = S.s[2 * qs + o], s4 = S.s[3 * qs + o];
  const R a1 = s1 + s3 + s4;
  R a2, a3, a4;
  if (pre) {
    // arc2d_precon :1264-1298
    const R bSq = adi_bsq(S, o), omb = (R)1. - bSq, cy = S.w[A_CY * ws + o];
    const R X = root((omb * qq2) * (omb * qq2) + (R)4. * bSq * cy * cy) / by(rr2);
    const R Y = (R)0.5 * (omb * qq2 / by(rr2) + X);
    const R Z = (R)0.5 * (omb * qq2 / by(rr2) - X);
    const R qqmxt = qq2 + ugc * rk1 * rr2 + vgc * rk2 * rr2;
    a2 = uu * s1 + rk2 * s2 + (uu + rk1 * Y / by(bSq)) * s3;
    a2 = a2 + (uu + rk1 * Z / by(bSq)) * s4;
    a3 = vv * s1 - rk1 * s2 + (vv + rk2 * Y / by(bSq)) * s3;
    a3 = a3 + (vv + rk2 * Z / by(bSq)) * s4;
    a4 = uv * s1 + (rk2 * uu - rk1 * vv) * s2;
    a4 = a4 + (ge + Y * qqmxt / by(rr2) / by(bSq)) * s3;
    a4 = a4 + (ge + Z * qqmxt / by(rr2) / by(bSq)) * s4;
  } else {
    a2 = uu * s1 + rk2 * s2 + (uu + rk1 * cjkl) * s3;
    a2 = a2 + (uu - rk1 * cjkl) * s4;
    a3 = vv * s1 - rk1 * s2 + (vv + rk2 * cjkl) * s3;
    a3 = a3 + (vv - rk2 * cjkl) * s4;
    a4 = uv * s1 + (rk2 * uu - rk1 * vv) * s2;
    a4 = a4 + (ge + cjkl * qq2 / by(rr2)) * s3;
    a4 = a4 + (ge - cjkl * qq2 / by(rr2)) * s4;
  }
  R o2 = a2, o3 = a3;
  if (p.iunst == 2) {
    const R tsr = S.tscale[o] * (R)p.rotf;
    const R d = (R)1.0 + sq(S.tscale[o] * (R)p.rotf);
    o2 = (a2 + tsr * a3) / by(d);
    o3 = (a3 - tsr * a2) / by(d);
  }
  S.s[o] = a1; S.s[qs + o] = o2; S.s[2 * qs + o] = o3; S.s[3 * qs + o] = a4;
  if constexpr (sizeof(R) == sizeof(double)) {
    double* q = S.q64;
    const double q1 = q[o], J = q[(int64_t)(p.nq - 1) * qs + o];
    const double dj = 1.0 / by(q1);
    const double u = q[qs + o] * dj, v = q[2 * qs + o] * dj, e = q[3 * qs + o] * dj;
    const double q1n = (q1 * J) / by(J);
    q[o] = q1n;
    q[qs + o] = u * q1n;
    q[2 * qs + o] = v * q1n;
    q[3 * qs + o] = e * q1n;
  }
}

}  // namespace ot2d
