// k_lusgs.cuh -- LU-SGS hyperplane operator ilu2d (src/lhs.f:470-814).
//
// The reference sweeps i+j hyperplanes; cell (j,k) of the forward sweep
// needs the already-updated s(j-1,k) and s(j,k-1) (backward: j+1, k+1).
// GB300 design:
//  1. k_lu_prep (fully parallel): every interior cell computes what the
//     sweeps need from it -- its scaled residual, tscale/2, the diagonal d
//     and the primitive / metric / spectral-radius factors of its outgoing
//     contributions (lhs.f:524-563, :626-653) -- and stores them in a
//     "skewed band" record: rows are grouped in bands of RB rows (one warp,
//     32 / RB lanes per row) and the record of step t of a band holds, for
//     every row r of the band, the cell at column t-r.  One wavefront step of
//     a warp is then one contiguous chunk (24 fields x RB cells).
//  2. k_lu_edges: point-Jacobi scaling of the halo residuals (lhs.f:567-598),
//     their contributions to the first/last interior row and column, and
//     (FP64) the reference's conservative->primitive->conservative round trip
//     of q (lhs.f:524-531, :805-811).
//  3. k_lu_sweep<FWD> (a cluster of 1..8 CTAs per slice, one warp per band):
//     the warps advance in a skewed lockstep; each warp streams its chunks
//     into a shared-memory ring with cp.async.bulk (TMA) completing on
//     mbarriers.  The lanes of a cell share its arithmetic (LuSplit), the
//     contribution to the next row passes through the warp's exchange buffer,
//     across bands through a shared-memory ring and across the CTAs of the cluster through the next
//     CTA's shared memory (st.async).  Every cell sees exactly the operands of
//     the reference's hyperplane order, so the sweep equals the sequential
//     one operation for operation.
#pragma once
#include <type_traits>
#include "dev_common.cuh"
#include "lu_shape.h"

namespace ot2d {

// record fields; each group of four is one 16-byte (f32) access
enum {
  LF_S = 0,    // 0..3: residual (forward input, then forward result)
  LF_SV = 4, LF_D = 5, LF_UU = 6, LF_VV = 7,
  LF_RI1 = 8, LF_RI2 = 9, LF_QX = 10, LF_UV2 = 11,     // xi metrics and contravariant velocity
  LF_RK1 = 12, LF_RK2 = 13, LF_QY = 14, LF_GE = 15,    // eta
  LF_FCX = 16, LF_FSX = 17, LF_FCY = 18, LF_FSY = 19,  // forward chk / spec (xi, eta)
  LF_BCX = 20, LF_BSX = 21, LF_BCY = 22, LF_BSY = 23,  // backward chk / spec
  // preconditioned records only: chk*qq (xi, eta) and gm1 (bSq-1)/c**2 of
  // the forward (24..27) and the backward (28..31) sweep
  LF_PF = 24, LF_PB = 28
};
// element offset of field f of row r within a chunk
template <class R, bool PRE = false>
__host__ __device__ __forceinline__ int lu_idx(int f, int r) {
  return r * LuLay<R, PRE>::LS + f;
}

// fields f..f+3 of row l of a chunk (f a multiple of 4) as 16-byte accesses
template <class R>
struct Lu4 { R x, y, z, w; };
template <bool PRE = false>
__device__ __forceinline__ void lu_st4(float* ch, int f, int l, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(ch + lu_idx<float, PRE>(f, l)) = make_float4(a, b, c, d);
}
template <bool PRE = false>
__device__ __forceinline__ void lu_st4(double* ch, int f, int l, double a, double b, double c, double d) {
  *reinterpret_cast<double2*>(ch + lu_idx<double, PRE>(f, l)) = make_double2(a, b);
  *reinterpret_cast<double2*>(ch + lu_idx<double, PRE>(f + 2, l)) = make_double2(c, d);
}

// Shared-memory accesses of the sweeps by 32-bit shared address (through
// generic pointers the address arithmetic was a third of a step's
// instructions): one, two or four consecutive values.
__device__ __forceinline__ void lu_lds(uint32_t a, float& x) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory");
}
__device__ __forceinline__ void lu_lds(uint32_t a, double& x) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
}
__device__ __forceinline__ void lu_lds2(uint32_t a, float& x, float& y) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void lu_lds2(uint32_t a, double& x, double& y) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ Lu4<float> lu_lds4(uint32_t a, float) {
  Lu4<float> v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ Lu4<double> lu_lds4(uint32_t a, double) {
  Lu4<double> v;
  lu_lds2(a, v.x, v.y);
  lu_lds2(a + 16, v.z, v.w);
  return v;
}
__device__ __forceinline__ void lu_sts(uint32_t a, double x) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}
__device__ __forceinline__ void lu_sts4(uint32_t a, const float* v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ void lu_sts4(uint32_t a, const double* v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]) : "memory");
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a + 16), "d"(v[2]), "d"(v[3]) : "memory");
}
// The same stores under a predicate, so that no lane branches, and global
// stores (to a 16-byte aligned address the four-value one).
__device__ __forceinline__ void lu_sts_if(bool p, uint32_t a, double x) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.shared.f64 [%0], %1;\n}" ::"r"(a), "d"(x), "r"((int)p) : "memory");
}
__device__ __forceinline__ void lu_sts4_if(bool p, uint32_t a, const float* v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %5, 0;\n @q st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"r"(a), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void lu_sts4_if(bool p, uint32_t a, const double* v) {
#pragma unroll
  for (int n = 0; n < 4; ++n) lu_sts_if(p, a + 8 * n, v[n]);
}
__device__ __forceinline__ void lu_stg_if(bool p, float* a, float x) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.global.f32 [%0], %1;\n}" ::"l"(a), "f"(x), "r"((int)p) : "memory");
}
__device__ __forceinline__ void lu_stg_if(bool p, double* a, double x) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.global.f64 [%0], %1;\n}" ::"l"(a), "d"(x), "r"((int)p) : "memory");
}
__device__ __forceinline__ void lu_stg4_if(bool p, float* a, const float* v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %5, 0;\n @q st.global.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"l"(a), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"((int)p)
               : "memory");
}
__device__ __forceinline__ void lu_stg4_if(bool p, double* a, const double* v) {
#pragma unroll
  for (int n = 0; n < 4; n += 2)
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q st.global.v2.f64 [%0], {%1, %2};\n}" ::"l"(a + n), "d"(v[n]),
                 "d"(v[n + 1]), "r"((int)p)
                 : "memory");
}

template <class R>
struct LuCell {
  R uu, vv, uv2, ge, ri1, ri2, rk1, rk2, qx, cx, qy, cy, vn, ugc, vgc, d;
  R bsq, term;   // preconditioned: bSq of the cell, gm1 (bSq-1)/c**2
};

// lhs.f:524-531 (conservative -> primitive) and :535-563 (diagonal); PRE:
// preilu2d's diagonal (lhs.f:60-101) from the preconditioned spectral radii
// 0.5 ((bSq+1)|qq| + sqrt(((1-bSq) qq)**2 + 4 bSq cc**2)) of both directions
template <class R, bool PRE = false>
__device__ __forceinline__ LuCell<R> lu_cell(const Slice<R>& S, const ot2d_params& p, int j, int k, R epsv) {
  const int64_t o = at(S.jd, j, k), qs = S.qs;
  LuCell<R> c;
  R q1 = S.q[o];
  R dj = (R)1.0 / by(q1);
  c.uu = S.q[qs + o] * dj;
  c.vv = S.q[2 * qs + o] * dj;
  R e = S.q[3 * qs + o] * dj;
  R rho = q1 * S.q[(p.nq - 1) * qs + o];
  c.uv2 = (R)0.5 * (c.uu * c.uu + c.vv * c.vv);
  R cjkl = root(S.k_ggm1 * (e - c.uv2));
  c.ri1 = S.xx[o]; c.ri2 = S.xy[o]; c.rk1 = S.yx[o]; c.rk2 = S.yy[o];
  c.ugc = S.ug ? S.ug[o] : (R)0; c.vgc = S.vg ? S.vg[o] : (R)0;
  R qq1 = c.ri1 * c.uu + c.ri2 * c.vv;
  R qqx = fabs(-c.ri1 * c.ugc - c.ri2 * c.vgc + qq1);
  R rr1 = root(sq(c.ri1) + sq(c.ri2));
  R qq2 = c.rk1 * c.uu + c.rk2 * c.vv;
  R qqy = fabs(-c.rk1 * c.ugc - c.rk2 * c.vgc + qq2);
  R rr2 = root(sq(c.rk1) + sq(c.rk2));
  R vnu = (R)2.0 * rr2 * rr2 * (S.k_rmue + S.turmu[o]) / by(S.k_rey * rho);
  R svt = S.tscale[o];
  c.qx = qq1; c.cx = cjkl * rr1; c.qy = qq2; c.cy = cjkl * rr2; c.vn = vnu;
  c.ge = S.k_gamma * e - S.k_gm1 * c.uv2;
  if constexpr (PRE) {
    const R btv = S.bt[o], mp2 = S.k_mp2;
    const R bSq = mp2 / by(btv - mp2 * (btv - (R)1));
    const R omb = (R)1. - bSq, opb = bSq + (R)1., fb = (R)4. * bSq;
    const R X = root((omb * qqx) * (omb * qqx) + (fb * c.cx) * c.cx);
    R term = (R)0.5 * (opb * qqx + X);
    const R Y = root((omb * qqy) * (omb * qqy) + (fb * c.cy) * c.cy);
    term = term + (R)0.5 * (opb * qqy + Y);
    c.d = (R)1.0 / by((R)1.0 + svt * (term * epsv + vnu));
    c.bsq = bSq;
    c.term = S.k_gm1 * (bSq - (R)1.) / by(cjkl * cjkl);
  } else {
    c.d = (R)1.0 / by((R)1.0 + svt * ((qqx + qqy + cjkl * (rr1 + rr2)) * epsv + vnu));
    c.bsq = (R)0; c.term = (R)0;
  }
  return c;
}

// chk / spec of one direction (lhs.f:636-640, :667-671, :735-739, :765-769)
template <class R, bool XI, bool FWD>
__device__ __forceinline__ void lu_chkspec(const LuCell<R>& c, R eps2, R& chk, R& spec) {
  R ri1 = XI ? c.ri1 : c.rk1, ri2 = XI ? c.ri2 : c.rk2, qq = XI ? c.qx : c.qy, cc = XI ? c.cx : c.cy;
  R qqn = -ri1 * c.ugc - ri2 * c.vgc + qq;
  R sp1 = fabs(qqn) + cc;
  R sm2 = eps2 * sp1;
  if (FWD) {
    chk = (R)0.5 + fsign((R)0.5, qqn + cc);
    spec = XI ? chk * (qqn + sp1) + sm2 : chk * (qqn + sp1) + c.vn + sm2;
  } else {
    chk = (R)0.5 - fsign((R)0.5, qqn - cc);
    spec = XI ? chk * (qqn - sp1) - sm2 : chk * (qqn - sp1) - c.vn - sm2;
  }
}

// contribution of a cell with correction s to its neighbour (lhs.f:643-653)
template <class R>
__device__ __forceinline__ void lu_apply(R chk, R spec, R ri1, R ri2, R qq, R uu, R vv, R uv2, R ge, R gm1,
                                         const R* s, R* a) {
  R s1 = s[0], s2 = s[1], s3 = s[2], s4 = s[3];
  R a4 = chk * (ri1 * s2 + ri2 * s3 - qq * s1);
  R a2 = chk * gm1 * (uv2 * s1 - (uu * s2 + vv * s3) + s4);
  a[0] = a4 + spec * s1;
  a[1] = ri1 * a2 + uu * a4 + spec * s2;
  a[2] = ri2 * a2 + vv * a4 + spec * s3;
  a[3] = qq * a2 + ge * a4 + spec * s4;
}

// preilu2d's chk / spec and chk*qq of one direction (lhs.f:160-179,
// :221-241, :321-340, :382-402): the convective split of the preconditioned
// eigenvalues (bSq+1) qq/2 +- X/2, X = sqrt(((1-bSq) qq)**2 + 4 bSq cc**2)
template <class R, bool XI, bool FWD>
__device__ __forceinline__ void lu_chkspec_pre(const LuCell<R>& c, R eps2, R& chk, R& cq, R& spec) {
  R ri1 = XI ? c.ri1 : c.rk1, ri2 = XI ? c.ri2 : c.rk2, qq = XI ? c.qx : c.qy, cc = XI ? c.cx : c.cy;
  R qqn = -ri1 * c.ugc - ri2 * c.vgc + qq;
  const R bSq = c.bsq, omb = (R)1. - bSq, opb = bSq + (R)1.;
  R X = root((omb * qqn) * (omb * qqn) + (((R)4. * bSq) * cc) * cc);
  if (FWD) chk = (R)0.5 + fsign((R)0.5, opb * qqn + X);
  else chk = (R)0.5 - fsign((R)0.5, opb * qqn - X);
  R sp1 = (R)0.5 * (opb * fabs(qqn) + X);
  R sm2 = eps2 * sp1;
  spec = XI ? chk * sp1 + sm2 : chk * sp1 + c.vn + sm2;
  cq = chk * qqn;
}

// preconditioned contribution of a cell with correction s to its neighbour
// (lhs.f:181-208): the split flux t, then t + term * [u,v,ge]^T
// [uv2, -u, -v, 1] t (the preconditioner), then +- spec * s
template <class R, bool FWD>
__device__ __forceinline__ void lu_apply_pre(R chk, R cq, R spec, R term, R ri1, R ri2, R qq, R uu, R vv, R uv2,
                                             R ge, R gm1, const R* s, R* a) {
  R s1 = s[0], s2 = s[1], s3 = s[2], s4 = s[3];
  R a4 = chk * (ri1 * s2 + ri2 * s3 - qq * s1);
  R a2 = chk * gm1 * (uv2 * s1 - (uu * s2 + vv * s3) + s4);
  const R t1 = a4 + cq * s1;
  const R t2 = ri1 * a2 + uu * a4 + cq * s2;
  const R t3 = ri2 * a2 + vv * a4 + cq * s3;
  const R t4 = qq * a2 + ge * a4 + cq * s4;
  const R r1 = uv2 * t1 - uu * t2 - vv * t3 + t4;
  const R p1 = r1 * term + t1, p2 = (uu * r1) * term + t2, p3 = (vv * r1) * term + t3, p4 = (ge * r1) * term + t4;
  if (FWD) {
    a[0] = p1 + spec * s1; a[1] = p2 + spec * s2; a[2] = p3 + spec * s3; a[3] = p4 + spec * s4;
  } else {
    a[0] = p1 - spec * s1; a[1] = p2 - spec * s2; a[2] = p3 - spec * s3; a[3] = p4 - spec * s4;
  }
}

template <class R, bool XI, bool FWD, bool PRE = false>
__device__ __forceinline__ void lu_contrib(const LuCell<R>& c, const R* s, R gm1, R eps2, R* a) {
  if constexpr (PRE) {
    R chk, cq, spec;
    lu_chkspec_pre<R, XI, FWD>(c, eps2, chk, cq, spec);
    lu_apply_pre<R, FWD>(chk, cq, spec, c.term, XI ? c.ri1 : c.rk1, XI ? c.ri2 : c.rk2, XI ? c.qx : c.qy, c.uu, c.vv,
                         c.uv2, c.ge, gm1, s, a);
  } else {
    R chk, spec;
    lu_chkspec<R, XI, FWD>(c, eps2, chk, spec);
    lu_apply(chk, spec, XI ? c.ri1 : c.rk1, XI ? c.ri2 : c.rk2, XI ? c.qx : c.qy, c.uu, c.vv, c.uv2, c.ge, gm1, s, a);
  }
}

// ---- kernel 1: records of the interior cells (one thread per (band, step, row))
// The record of row l of chunk (band, t) into ch, the chunk as k_lu_prep
// stages it in shared memory.
template <class R, bool PRE = false>
__device__ __forceinline__ void lu_prep_cell(const Slice<R>& S, const ot2d_params& p, int band, int t, int l, int scale,
                                             R* ch) {
  const int nrow = lu_nrow(S.kd), ncol = lu_ncol(S.jd);
  const int r = LuSplit<R, PRE>::RB * band + l, c = t - l;
  if (r >= nrow || c < 0 || c >= ncol) {
    const R z = (R)0;
#pragma unroll
    for (int f = 0; f < LuLay<R, PRE>::NF; f += 4) lu_st4<PRE>(ch, f, l, z, z, z, z);
    return;
  }
  const int j = p.jbeg + c, k = p.kbeg + r;
  const R eps2 = S.k_eps2, epsv = S.k_epsv;
  const int64_t o = at(S.jd, j, k);
  LuCell<R> cl = lu_cell<R, PRE>(S, p, j, k, epsv);
  const R ts = S.tscale[o];
  R sv[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    R v = S.s[n * S.qs + o];
    sv[n] = scale ? v * ts : v;
  }
  lu_st4<PRE>(ch, LF_S, l, sv[0], sv[1], sv[2], sv[3]);
  lu_st4<PRE>(ch, LF_SV, l, ts * (R)0.5, cl.d, cl.uu, cl.vv);
  lu_st4<PRE>(ch, LF_RI1, l, cl.ri1, cl.ri2, cl.qx, cl.uv2);
  lu_st4<PRE>(ch, LF_RK1, l, cl.rk1, cl.rk2, cl.qy, cl.ge);
  R a, b, a2, b2;
  if constexpr (PRE) {
    R q1, q2;
    lu_chkspec_pre<R, true, true>(cl, eps2, a, q1, b);
    lu_chkspec_pre<R, false, true>(cl, eps2, a2, q2, b2);
    lu_st4<PRE>(ch, LF_FCX, l, a, b, a2, b2);
    lu_st4<PRE>(ch, LF_PF, l, q1, q2, cl.term, (R)0);
    lu_chkspec_pre<R, true, false>(cl, eps2, a, q1, b);
    lu_chkspec_pre<R, false, false>(cl, eps2, a2, q2, b2);
    lu_st4<PRE>(ch, LF_BCX, l, a, b, a2, b2);
    lu_st4<PRE>(ch, LF_PB, l, q1, q2, cl.term, (R)0);
  } else {
    lu_chkspec<R, true, true>(cl, eps2, a, b);
    lu_chkspec<R, false, true>(cl, eps2, a2, b2);
    lu_st4(ch, LF_FCX, l, a, b, a2, b2);
    lu_chkspec<R, true, false>(cl, eps2, a, b);
    lu_chkspec<R, false, false>(cl, eps2, a2, b2);
    lu_st4(ch, LF_BCX, l, a, b, a2, b2);
  }
}

// halo-contribution arrays after the chunks: A forward [nrow][4], A backward,
// B forward [ncol][4], B backward (last column first: in sweep order)
template <class R, bool PRE = false>
__device__ __forceinline__ R* lu_halo(const Slice<R>& S, int which) {
  const int nrow = lu_nrow(S.kd), ncol = lu_ncol(S.jd);
  constexpr int RB = LuSplit<R, PRE>::RB;
  R* base = S.lurec + (int64_t)lu_nband(S.kd, RB) * lu_nstep(S.jd, RB) * LuLay<R, PRE>::CH;
  switch (which) {
    case 0: return base;
    case 1: return base + 4 * nrow;
    case 2: return base + 8 * nrow;
    default: return base + 8 * nrow + 4 * ncol;
  }
}

// ---- kernel 2: halo edges (one thread per cell of the slice)
template <class R, bool PRE = false>
__device__ __forceinline__ void lu_edge_cell(const Slice<R>& S, const ot2d_params& p, int j, int k, int scale) {
  const int js = p.jbeg, je = p.jend, ks = p.kbeg, ke = p.kend;
  const bool ij = j >= js && j <= je, ik = k >= ks && k <= ke;
  const int64_t o = at(S.jd, j, k);
  const R eps2 = S.k_eps2, epsv = S.k_epsv, gm1 = S.k_gm1;
  if (!(ij && ik)) {
    R sv[4];
    const R ts = S.tscale[o];
#pragma unroll
    for (int n = 0; n < 4; ++n) sv[n] = scale ? S.s[n * S.qs + o] * ts : S.s[n * S.qs + o];
    const bool edge = (ik && (j == js - 1 || j == je + 1)) || (ij && (k == ks - 1 || k == ke + 1));
    if (edge) {
      LuCell<R> c = lu_cell<R, PRE>(S, p, j, k, epsv);
#pragma unroll
      for (int n = 0; n < 4; ++n) sv[n] = sv[n] * c.d;
      R a[4];
      R* dst = nullptr;
      if (j == js - 1) { lu_contrib<R, true, true, PRE>(c, sv, gm1, eps2, a); dst = lu_halo<R, PRE>(S, 0) + 4 * (k - ks); }
      else if (j == je + 1) { lu_contrib<R, true, false, PRE>(c, sv, gm1, eps2, a); dst = lu_halo<R, PRE>(S, 1) + 4 * (k - ks); }
      else if (k == ks - 1) { lu_contrib<R, false, true, PRE>(c, sv, gm1, eps2, a); dst = lu_halo<R, PRE>(S, 2) + 4 * (j - js); }
      else { lu_contrib<R, false, false, PRE>(c, sv, gm1, eps2, a); dst = lu_halo<R, PRE>(S, 3) + 4 * (je - j); }
#pragma unroll
      for (int n = 0; n < 4; ++n) dst[n] = a[n];
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) S.s[n * S.qs + o] = sv[n];
  }
  // FP64 plain path: q leaves ilu2d round-tripped (lhs.f:524-531, :805-811)
  if constexpr (sizeof(R) == sizeof(double)) {
    const int64_t qs = S.qs;
    double q1 = S.q[o], J = S.q[(p.nq - 1) * qs + o];
    double dj = 1.0 / by(q1);
    double u = S.q[qs + o] * dj, v = S.q[2 * qs + o] * dj, e = S.q[3 * qs + o] * dj;
    double q1n = (q1 * J) / by(J);
    S.q[o] = q1n;
    S.q[qs + o] = u * q1n;
    S.q[2 * qs + o] = v * q1n;
    S.q[3 * qs + o] = e * q1n;
  }
}

// ---- kernel 3: the sweeps --------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Polls a sweep wait makes before it gives up (the status word of the slice
// records the timeout).  The solver can lower it (OT2D_OPT_POLL_LIMIT) to
// make the waits run out on purpose; the drain of copies still in flight
// after a give-up always uses this default bound.
constexpr uint32_t LU_POLL_DEFAULT = 1u << 22;

// Bounded wait on a ring slot; false after `lim` polls.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t lim = LU_POLL_DEFAULT) {
  for (uint32_t it = 0; it < lim; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// The same by a whole warp.  The vote makes the loop and its result uniform:
// the band leaves at the first wait that runs out, and a step costs what it
// costs without a check (one vote over the lanes' results ahead of a group's
// first read cost 85 cycles a group: both sweeps of a 1025x33 mesh 252 us with
// a vote at the end of the group, 263 ahead of it, 249 so).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, uint32_t lim) {
  for (uint32_t it = 0; it < lim; ++it)
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return false;
}

// address of a local shared-memory object in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t lu_mapa(uint32_t local, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// four values (one for FP64: lane v's own) into the next CTA's row, counted
// on its barrier
__device__ __forceinline__ void lu_send(uint32_t dst, uint32_t bar, const float* v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void lu_send1(uint32_t dst, uint32_t bar, double v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void lu_send(uint32_t dst, uint32_t bar, const double* v) {
#pragma unroll
  for (int n = 0; n < 4; ++n) lu_send1(dst + 8 * n, bar, v[n]);
}
// a whole warp's wait (as mbar_wait_warp) for a barrier of the link
__device__ __forceinline__ bool lu_link_wait(uint64_t* bar, uint32_t lim) {
  for (uint32_t it = 0; it < lim; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar))
        : "memory");
    if (__all_sync(0xffffffffu, (int)ok)) return true;
  }
  return false;
}
__device__ __forceinline__ void lu_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}

// The arithmetic of one wavefront step for the lanes of a warp.
//
// Two lanes per cell: lane 2r+d forms the whole correction of row r's cell
// and the contribution of direction d (0 xi, 1 eta) in out[], which it leaves
// in its slots of the exchange buffer for the cells that take it.
template <class R, bool FWD, bool PRE, int LP, int KS>
struct LuLanes;

template <class R, bool FWD, bool PRE, int KS>
struct LuLanes<R, FWD, PRE, 2, KS> {
  static constexpr uint32_t B = sizeof(R), SB = 4 * B, LN = (KS + 1) * SB;   // bytes: value, slot, lane
  // the lane's share of a cell's record
  struct Rec { Lu4<R> s, p, m, pp; R chk, spec, other; };
  R out[4], hx[4] = {0, 0, 0, 0};
  uint32_t wr, ra, rb, oD, oO, oC;
  int d;
  __device__ __forceinline__ LuLanes(int l, uint32_t ex) {
    d = l & 1;
    wr = ex + l * LN;
    ra = ex + (l & ~1) * LN;                                    // the row's xi lane
    rb = ex + ((FWD ? (l & ~1) - 1 : (l | 1) + 2) & 31) * LN;   // the previous row's eta lane
    oD = (d ? LF_RK1 : LF_RI1) * B;
    oO = (d ? LF_UV2 : LF_GE) * B;
    oC = ((FWD ? LF_FCX : LF_BCX) + 2 * d) * B;
  }
  __device__ __forceinline__ Rec load(uint32_t rec) const {
    Rec r;
    r.s = lu_lds4(rec + LF_S * B, R());
    r.p = lu_lds4(rec + LF_SV * B, R());
    r.m = lu_lds4(rec + oD, R());
    lu_lds2(rec + oC, r.chk, r.spec);
    lu_lds(rec + oO, r.other);
    if constexpr (PRE) r.pp = lu_lds4(rec + (FWD ? LF_PF : LF_PB) * B, R());   // chk*qq xi, eta, preconditioner factor
    return r;
  }
  __device__ __forceinline__ uint32_t eta_base() const { return rb; }
  __device__ __forceinline__ uint32_t eta_link(uint32_t slot) const { return slot; }
  // the halo's xi contribution to the row's first column
  __device__ __forceinline__ void halo_xi(const R* p) {
#pragma unroll
    for (int n = 0; n < 4; ++n) hx[n] = p[n];
  }
  // The cell of a step: eta the address of its incoming eta contribution, k
  // and kn the exchange slots of this and of the next step; recg this step's
  // global record, srow the row of s at the cell's column.  RAMP: some row may
  // be on its first column (first) or outside its columns (not valid: its
  // record is 0, so is its contribution, and nothing takes it).
  template <bool RAMP>
  __device__ __forceinline__ void cell(const Rec& r, uint32_t eta, int k, int kn, bool first, bool valid, R gm1, R* recg,
                                       R* srow, int64_t qs) {
    const Lu4<R> xb = lu_lds4(eta, R());
    Lu4<R> xa = lu_lds4(ra + k * SB, R());
    if (RAMP) {
      xa.x = first ? hx[0] : xa.x; xa.y = first ? hx[1] : xa.y;
      xa.z = first ? hx[2] : xa.z; xa.w = first ? hx[3] : xa.w;
    }
    const R uv2 = d ? r.other : r.m.w, ge = d ? r.m.w : r.other;
    const R st[4] = {r.s.x, r.s.y, r.s.z, r.s.w};
    const R in[4] = {xa.x + xb.x, xa.y + xb.y, xa.z + xb.z, xa.w + xb.w};
    const R sv = r.p.x, di = r.p.y;
    R sn[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) sn[n] = FWD ? (st[n] + sv * in[n]) * di : st[n] - sv * in[n] * di;
    if constexpr (PRE) {
      lu_apply_pre<R, FWD>(r.chk, d ? r.pp.y : r.pp.x, r.spec, r.pp.z, r.m.x, r.m.y, r.m.z, r.p.z, r.p.w, uv2, ge, gm1,
                           sn, out);
    } else {
      lu_apply(r.chk, r.spec, r.m.x, r.m.y, r.m.z, r.p.z, r.p.w, uv2, ge, gm1, sn, out);
    }
    lu_sts4(wr + kn * SB, out);
    if (FWD) {
      lu_stg4_if(d == 0, recg + LF_S, sn);         // into the record, for the backward sweep
    } else {
      // two variables per lane (srow: the lane's first)
      lu_stg_if(!RAMP || valid, srow, d ? sn[2] : sn[0]);
      lu_stg_if(!RAMP || valid, srow + qs, d ? sn[3] : sn[1]);
    }
  }
  __device__ __forceinline__ int first_var() const { return 2 * d; }
  __device__ __forceinline__ bool owns_eta() const { return d == 1; }
  __device__ __forceinline__ void put_if(bool c, uint32_t p) const { lu_sts4_if(c, p, out); }
  __device__ __forceinline__ void send(uint32_t dst, uint32_t bar) const { lu_send(dst, bar, out); }
  __device__ __forceinline__ void send_zero(uint32_t dst, uint32_t bar) const {
    const R z[4] = {0, 0, 0, 0};
    lu_send(dst, bar, z);
  }
};

// Four lanes per cell (FP64): lane 4r+v holds variable v.  Lanes 0..3 form
// a4 and a2 (lu_apply) of xi, then of eta -- one instruction stream over
// (A, B, C) = (ri1, ri2, qq) for a4 and (u, v, uv2) for a2 -- and each lane
// its variable's contribution to both directions.  The corrections, the four
// scalars and the eta contributions pass through parts of the exchange
// buffer, a warp barrier between a part's write and its reads.
template <bool FWD, int KS>
struct LuLanes<double, FWD, false, 4, KS> {
  static constexpr uint32_t B = 8, SB = 32, LN = (KS + 1) * SB;   // bytes: value, slot, row of slots
  struct Rec { double sv, d, a, b, st, cc, chk, pe, px, q, fsx, fsy; };
  double ox = 0, oe = 0, hx = 0;   // this variable's xi / eta contribution of the lane's last cell; the halo's xi
  uint32_t wr, rd, wre, rb, oA, oC, oK, oX, oE, oQ, vb;
  int v;
  bool odd;
  __device__ __forceinline__ LuLanes(int l, uint32_t exb) {
    v = l & 3;
    odd = v & 1;
    vb = v * B;
    wr = exb + l * B;
    rd = exb + (l & ~3) * B;
    wre = exb + 64 * B + (l >> 2) * LN + vb;
    rb = exb + 64 * B + ((FWD ? (l >> 2) - 1 : (l >> 2) + 1) & 7) * LN + vb;
    oA = (odd ? LF_UU : (v ? LF_RK1 : LF_RI1)) * B;
    oC = (odd ? LF_UV2 : (v ? LF_QY : LF_QX)) * B;
    oK = ((FWD ? LF_FCX : LF_BCX) + (v & 2)) * B;
    oX = (LF_RI1 - 1 + v) * B;                     // ri1, ri2, qx for v = 1, 2, 3
    oE = (LF_RK1 - 1 + v) * B;
    oQ = (v == 1 ? LF_UU : (v == 2 ? LF_VV : LF_GE)) * B;
  }
  __device__ __forceinline__ Rec load(uint32_t rec) const {
    Rec r;
    lu_lds(rec + LF_S * B + vb, r.st);
    lu_lds2(rec + LF_SV * B, r.sv, r.d);
    lu_lds2(rec + oA, r.a, r.b);
    lu_lds(rec + oC, r.cc);
    lu_lds(rec + oK, r.chk);
    lu_lds(rec + oE, r.pe);
    lu_lds(rec + oX, r.px);
    lu_lds(rec + oQ, r.q);
    lu_lds(rec + (FWD ? LF_FSX : LF_BSX) * B, r.fsx);
    lu_lds(rec + (FWD ? LF_FSY : LF_BSY) * B, r.fsy);
    return r;
  }
  __device__ __forceinline__ uint32_t eta_base() const { return rb; }
  __device__ __forceinline__ uint32_t eta_link(uint32_t slot) const { return slot + vb; }
  __device__ __forceinline__ void halo_xi(const double* p) { hx = p[v]; }
  template <bool RAMP>
  __device__ __forceinline__ void cell(const Rec& r, uint32_t eta, int, int kn, bool first, bool valid, double gm1,
                                       double* recg, double* srow, int64_t) {
    double xb;
    lu_lds(eta, xb);
    const double xa = RAMP && first ? hx : ox;
    const double sn = FWD ? (r.st + r.sv * (xa + xb)) * r.d : r.st - r.sv * (xa + xb) * r.d;
    lu_sts(wr, sn);
    __syncwarp();
    if (FWD) lu_stg_if(true, recg + LF_S + v, sn);
    else lu_stg_if(!RAMP || valid, srow, sn);
    const Lu4<double> s = lu_lds4(rd, 0.0);
    // a4 = chk*(ri1*s2 + ri2*s3 - qq*s1)
    // a2 = chk*gm1*(uv2*s1 - (u*s2 + v*s3) + s4); chk is 0 or 1
    const double x = r.a * s.y + r.b * s.z, y = r.cc * s.x;
    const double t = (odd ? y : x) - (odd ? x : y);
    const double w = (odd ? (__double2hiint(r.chk) ? gm1 : 0.0) : r.chk) * (odd ? t + s.w : t);
    lu_sts(wr + 32 * B, w);
    const double gx = r.fsx * sn, gy = r.fsy * sn;
    __syncwarp();
    const Lu4<double> a = lu_lds4(rd + 32 * B, 0.0);    // a4, a2 of xi; a4, a2 of eta
    const double my = r.pe * a.w + r.q * a.z;
    oe = (v ? my : a.z) + gy;
    lu_sts(wre + kn * SB, oe);
    const double mx = r.px * a.y + r.q * a.x;
    ox = (v ? mx : a.x) + gx;
  }
  __device__ __forceinline__ int first_var() const { return v; }
  __device__ __forceinline__ bool owns_eta() const { return true; }
  __device__ __forceinline__ void put_if(bool c, uint32_t p) const { lu_sts_if(c, p + vb, oe); }
  __device__ __forceinline__ void send(uint32_t dst, uint32_t bar) const { lu_send1(dst + vb, bar, oe); }
  __device__ __forceinline__ void send_zero(uint32_t dst, uint32_t bar) const { lu_send1(dst + vb, bar, 0.0); }
};

// bulk copy (TMA) into this CTA's shared memory, counted on bar; 16-byte
// aligned ends and size
__device__ __forceinline__ void lu_bulk(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// What a warp of a sweep works on (lu_sweep_slice), and where its first row's
// input comes from (IN) and its last row's contributions go (OUT).
enum { LU_HALO = 0, LU_NONE = 0, LU_RING = 1, LU_LINK = 2 };
template <class R>
struct LuBand {
  int band, nrow, ncol, nst, row0;           // row0: first row of the band
  uint32_t lim;
  int lag, D;
  R gm1;
  const R* rec;                              // the band's records
  R* rec_w;
  R* s;                                      // s at (first interior row of the band, first interior column), variable 1
  int64_t jd, qs;
  const R* halo;                             // xi contributions of the halo to the first column, 4 per row
  uint32_t stages, ex, xin, xout;            // shared addresses: record stages, exchange buffer, input row or ring, ring
  uint64_t *bars, *xb_in, *xb_out, *lbars;   // barriers: stages; the input ring's, the own ring's; the link's
  uint32_t ldst, lbar;                       // the next CTA's row and its barriers
};

// One band of one sweep.  Returns the group at which a bounded wait gave up,
// or -1.  A group whose waits did not all end is left alone: its records may
// not have landed, so nothing of it is read, stored, handed on or refilled.
template <class R, bool FWD, bool PRE, int PG, int IN, int OUT>
__device__ __forceinline__ int lu_band(const LuBand<R>& B, int l) {
  constexpr int CH = LuLay<R, PRE>::CH, LS = LuLay<R, PRE>::LS, LP = LuSplit<R, PRE>::LP, RB = LuSplit<R, PRE>::RB;
  constexpr int NS = LU_XB / PG, KS = lu_ks<PG>();
  constexpr uint32_t SB = 4 * sizeof(R), CHB = CH * sizeof(R);
  static_assert(KS % PG == 0 && LU_LG % PG == 0 && LU_XB % PG == 0 && RB % PG == 0, "groups do not straddle");
  const int ncol = B.ncol, nst = B.nst, D = B.D, ngrp = (nst + PG - 1) / PG;
  const uint32_t lim = B.lim;
  const int row = l / LP, r = B.row0 + row;
  const int lout = FWD ? RB - 1 : 0;                         // the row the next band takes
  // the row that takes from outside the band
  const int lin = FWD ? 0 : min(RB - 1, B.nrow - 1 - B.row0);
  const int prow = FWD ? row : RB - 1 - row;                 // steps this row trails the band's first
  constexpr int xmask = IN == LU_RING ? LU_XB - 1 : 0x7fffffff;
  LuLanes<R, FWD, PRE, LP, KS> L(l, B.ex);
  const int cols = r < B.nrow ? ncol : 0;                    // columns of this row (none beyond the mesh)
  if (cols) L.halo_xi(B.halo + 4 * r);
  const bool is_lin = row == lin, out_lane = row == lout && L.owns_eta();
  const int64_t qs = B.qs;
  const R gm1 = B.gm1;
  // this row's record of step 0 in global memory; its column of s at step 0,
  // the lane's first variable (backward); both step on with the sweep
  constexpr int SSTEP = FWD ? 1 : -1;
  R* rg = B.rec_w + (int64_t)row * LS;
  R* sr = B.s + (int64_t)L.first_var() * qs + (int64_t)row * B.jd + (FWD ? -prow : ncol - 1 + prow);
  const uint32_t eta0 = L.eta_base(), lin0 = L.eta_link(B.xin);
  // records of group g: chunks c0(g) .. c0(g)+size-1 of the band, ascending
  auto issue = [&](int g, int st) {
    const int n = min(PG, nst - g * PG), c0 = FWD ? g * PG : nst - g * PG - n;
    // (the stage's earlier reads are ordered by the warp barrier before; a
    // proxy fence here made each group wait for its global stores)
    mbar_expect_tx(&B.bars[st], (uint32_t)n * CHB);
    lu_bulk(B.stages + (uint32_t)st * PG * CHB, B.rec + (int64_t)c0 * CH, (uint32_t)n * CHB, &B.bars[st]);
  };
  if (l == 0)
    for (int g = 0; g < min(D, ngrp); ++g) issue(g, g);
  // Waits for group q of the previous band's, or the next band's, steps (each
  // phase of a ring slot's barrier is one group).
  const int qlast = ngrp - 1;
  auto wait_full = [&](int q) { return mbar_wait_warp(&B.xb_in[q % NS], (uint32_t)(q / NS) & 1, lim); };
  auto wait_empty = [&](int q) { return mbar_wait_warp(&B.xb_out[NS + q % NS], (uint32_t)(q / NS) & 1, lim); };
  bool ok = true;
  if (IN == LU_HALO) ok = mbar_wait_warp(&B.lbars[0], 0, lim);
  // Band lag: start `lag` steps after the neighbouring band's first
  // contribution is due (the operands of every cell are the same whatever
  // the lag; at most what the ring holds).
  if (IN == LU_RING && B.lag > 0)
    ok = wait_full(min(min(RB + B.lag, LU_XB) / PG - 1, qlast));
  // groups g0 .. g1-1 have every row active and none on its first column
  const bool full = B.row0 + RB <= B.nrow;
  const int g0 = full ? RB / PG : ngrp, g1 = full ? max(g0, ncol / PG) : ngrp;
  int stage = 0;
  uint32_t phase = 0;
  int g = 0;
  auto group = [&](auto ramp_) {
    constexpr bool RAMP = decltype(ramp_)::value;
    const int t0 = g * PG, ps = RAMP ? min(PG, nst - t0) : PG, p0 = t0 - prow;
    if (!(ok = mbar_wait_warp(&B.bars[stage], phase, lim))) return;
    // the first row's inputs of these steps (columns t0 .. t0+PG-1 in sweep
    // order, produced RB-1 steps later by the previous band), and room in the
    // ring for the last row's outputs
    if (IN == LU_RING && (!RAMP || t0 < ncol) && !(ok = wait_full(min(g + RB / PG, qlast)))) return;
    if (IN == LU_LINK && (!RAMP || t0 < ncol) && !(ok = lu_link_wait(&B.lbars[t0 / LU_LG], lim))) return;
    if (OUT == LU_RING && g + 1 >= (RB + LU_XB) / PG && !(ok = wait_empty(g + 1 - (RB + LU_XB) / PG))) return;
    const uint32_t st0 = B.stages + (uint32_t)stage * PG * CHB + (uint32_t)row * LS * sizeof(R);
    const uint32_t ch0 = FWD ? st0 : st0 + (uint32_t)(ps - 1) * CHB;
    const int k0 = PG == KS ? 0 : t0 & (KS - 1);
    const uint32_t eta = is_lin ? lin0 + (uint32_t)(t0 & xmask) * SB : eta0 + (uint32_t)k0 * SB;
    auto rec = L.load(ch0);
#pragma unroll
    for (int u = 0; u < PG; ++u) {
      if (RAMP && u >= ps) break;
      const auto cur = rec;
      if (u + 1 < PG && (!RAMP || u + 1 < ps)) rec = L.load(FWD ? ch0 + (u + 1) * CHB : ch0 - (u + 1) * CHB);
      const bool valid = !RAMP || (unsigned)(p0 + u) < (unsigned)cols;
      // (outside its columns the first row reads slot 0, in bounds)
      const uint32_t ea = RAMP && is_lin ? lin0 + (uint32_t)(valid ? (p0 + u) & xmask : 0) * SB : eta + u * SB;
      L.template cell<RAMP>(cur, ea, k0 + u, (k0 + u + 1) & (KS - 1), RAMP && p0 + u == 0, valid, gm1, rg + u * CH,
                            sr + u * SSTEP, qs);
      if (OUT == LU_RING) L.put_if(out_lane, B.xout + (uint32_t)((p0 + u) & (LU_XB - 1)) * SB);
      if (OUT == LU_LINK) {
        if (out_lane && valid) L.send(B.ldst + (uint32_t)(p0 + u) * SB, B.lbar + (uint32_t)((p0 + u) / LU_LG) * 8);
      }
      __syncwarp();
    }
    rg += PG * CH;
    sr += PG * SSTEP;
    if (l == 0) {
      // these steps' ring slots are read and written by the whole warp, and
      // its stage takes group g + D
      if (OUT == LU_RING) mbar_arrive(&B.xb_out[g % NS]);
      if (IN == LU_RING) mbar_arrive(&B.xb_in[NS + g % NS]);
      if (g + D < ngrp) issue(g + D, stage);
    }
    if (++stage == D) { stage = 0; phase ^= 1; }
    ++g;
  };
  while (g < ngrp && ok) {
    if (g == g0)
#pragma unroll 1
      while (g < g1 && ok) group(std::false_type());
    if (g < ngrp && ok) group(std::true_type());
  }
  if (ok) return -1;
  // The rest of the row that the next CTA takes, as zeros (its results are
  // discarded with the slice's): with it every barrier of the link completes,
  // so that CTA can wait for the last store before its shared memory goes.
  if (OUT == LU_LINK && out_lane)
    for (int q = max(0, g * PG - (RB - 1)); q < ncol; ++q)
      L.send_zero(B.ldst + (uint32_t)q * SB, B.lbar + (uint32_t)(q / LU_LG) * 8);
  // copies issued and not consumed, each in its own phase: wait (bounded)
  // before the CTA's shared memory goes away
  if (l == 0)
    for (int h = g; h < min(g + D, ngrp); ++h) mbar_wait_bounded(&B.bars[h % D], (uint32_t)(h / D) & 1);
  __syncwarp();
  return g;
}

// One sweep of one slice by the CTA `rank` of a cluster of cs.  The slice's
// bands are dealt to the CTAs in contiguous runs, one warp per band; a warp
// walks its nst local steps: at local step t row r of the band is on column
// t-r (forward) or ncol-1-(t-(RB-1-r)) (backward), so the rows of a band are
// on RB consecutive hyperplanes and the in-band dependency (the neighbouring
// row) arrives through the warp's exchange buffer from the previous step.
// The dependency across bands -- the last row of a band feeds the first row
// of the next, RB-1 steps later -- goes through the producer's cross-band
// ring guarded by mbarriers within a CTA (a counter published with a release
// store cost a memory fence behind every group's global stores), and into the
// next CTA's shared memory with st.async between CTAs (a whole row: nothing
// is overwritten, so nothing flows back), so the warps run without block-wide
// barriers.  Rows that have not reached their first column or are past their
// last one run along on records of 0, so that no step branches; the groups
// inside the columns of all rows of a full band also leave out their selects.
// PRE: the preilu2d records and contributions.
template <class R, bool FWD, bool PRE, int PG>
__device__ void lu_sweep_slice(const Slice<R>& S, int nwarp, int cs, int rank, int maxcol, int D, unsigned char* smem,
                               uint32_t lim, int lag) {
  constexpr int CH = LuLay<R, PRE>::CH, RB = LuSplit<R, PRE>::RB, NS = LU_XB / PG;
  const ot2d_params& p = *S.P;
  const int nrow = lu_nrow(S.kd), ncol = lu_ncol(S.jd), nb = lu_nband(S.kd, RB), nst = lu_nstep(S.jd, RB);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int per = (nb + cs - 1) / cs, base = rank * per, mine = max(0, min(per, nb - base));
  const int band = base + w;
  R* stages = (R*)smem;
  R* xrings = stages + (size_t)nwarp * D * PG * CH;
  R* exs = xrings + (size_t)lu_nring(nwarp) * LU_XB * 4;
  R* rowbuf = exs + (size_t)nwarp * lu_ex<R, PRE, PG>();
  uint64_t* bars = (uint64_t*)(rowbuf + (size_t)4 * maxcol);
  uint64_t* xbars = bars + (size_t)nwarp * D;               // per warp: full[NS], empty[NS] of its ring
  uint64_t* lbars = xbars + (size_t)lu_nring(nwarp) * 2 * NS;
  const bool wok = w < mine;
  // the CTA of the first band in sweep order takes the halo's contributions
  const bool first_cta = FWD ? rank == 0 : base + mine == nb;
  const bool linked = cs > 1 && mine > 0 && !first_cta;     // takes its row from the previous CTA
  for (int i = l; i < D; i += 32) mbar_init(&bars[(size_t)w * D + i], 1);
  if (nwarp > 1)
    for (int i = l; i < 2 * NS; i += 32) mbar_init(&xbars[(size_t)w * 2 * NS + i], 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int i = l; i < lu_ex<R, PRE, PG>(); i += 32) exs[(size_t)w * lu_ex<R, PRE, PG>() + i] = (R)0;
  if (linked) {
    for (int i = threadIdx.x; i < (ncol + LU_LG - 1) / LU_LG; i += blockDim.x) {
      mbar_init(&lbars[i], 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(&lbars[i], (uint32_t)min(LU_LG, ncol - i * LU_LG) * 4 * sizeof(R));
    }
  } else if (threadIdx.x == 0 && mine > 0) {
    // the halo's row, one bulk copy (a loop of loads through registers took
    // 10-20 us of a small mesh's sweep)
    mbar_init(&lbars[0], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(&lbars[0], (uint32_t)(4 * ncol * sizeof(R)));
    lu_bulk(smem_u32(rowbuf), lu_halo<R, PRE>(S, FWD ? 2 : 3), (uint32_t)(4 * ncol * sizeof(R)), &lbars[0]);
  }
  __syncthreads();
  if (cs > 1) lu_cluster_sync();
  int gfail = -1;
  if (wok) {
    // neighbouring bands in sweep order
    const bool has_next = FWD ? band + 1 < nb : band > 0;
    const bool prev_here = FWD ? w > 0 : w + 1 < mine;
    const bool next_here = has_next && (FWD ? w + 1 < mine : w > 0);
    const bool from_link = linked && !prev_here, to_link = has_next && !next_here;
    const int wprev = prev_here ? (FWD ? w - 1 : w + 1) : w;
    LuBand<R> B;
    B.band = band; B.nrow = nrow; B.ncol = ncol; B.nst = nst; B.row0 = RB * band;
    B.lim = lim; B.lag = lag; B.D = D;
    B.gm1 = S.k_gm1;
    B.rec_w = S.lurec + (int64_t)band * nst * CH;
    B.rec = B.rec_w;
    B.s = S.s + (int64_t)(p.kbeg + RB * band - 1) * S.jd + (p.jbeg - 1);
    B.jd = S.jd; B.qs = S.qs;
    B.halo = lu_halo<R, PRE>(S, FWD ? 0 : 1);
    B.stages = smem_u32(stages + (size_t)w * D * PG * CH);
    B.ex = smem_u32(exs + (size_t)w * lu_ex<R, PRE, PG>());
    B.xin = smem_u32(prev_here ? xrings + (size_t)wprev * LU_XB * 4 : rowbuf);
    B.xout = smem_u32(xrings + (size_t)w * LU_XB * 4);
    B.bars = bars + (size_t)w * D;
    B.xb_in = xbars + (size_t)wprev * 2 * NS;
    B.xb_out = xbars + (size_t)w * 2 * NS;
    B.lbars = lbars;
    const int nrank = FWD ? rank + 1 : rank - 1;
    B.ldst = B.lbar = 0;
    if (to_link) {
      B.ldst = lu_mapa(smem_u32(rowbuf), nrank);
      B.lbar = lu_mapa(smem_u32(lbars), nrank);
    }
    if (prev_here) {
      if (next_here) gfail = lu_band<R, FWD, PRE, PG, LU_RING, LU_RING>(B, l);
      else if (to_link) gfail = lu_band<R, FWD, PRE, PG, LU_RING, LU_LINK>(B, l);
      else gfail = lu_band<R, FWD, PRE, PG, LU_RING, LU_NONE>(B, l);
    } else if (from_link) {
      if (next_here) gfail = lu_band<R, FWD, PRE, PG, LU_LINK, LU_RING>(B, l);
      else if (to_link) gfail = lu_band<R, FWD, PRE, PG, LU_LINK, LU_LINK>(B, l);
      else gfail = lu_band<R, FWD, PRE, PG, LU_LINK, LU_NONE>(B, l);
    } else {
      if (next_here) gfail = lu_band<R, FWD, PRE, PG, LU_HALO, LU_RING>(B, l);
      else if (to_link) gfail = lu_band<R, FWD, PRE, PG, LU_HALO, LU_LINK>(B, l);
      else gfail = lu_band<R, FWD, PRE, PG, LU_HALO, LU_NONE>(B, l);
    }
    if (gfail >= 0 && l == 0 && S.ist) atomicOr(&S.ist[2], 4);
  }
  // a give-up before the halo's row has landed: wait (bounded) for it
  if (!linked && mine > 0 && threadIdx.x == 0) mbar_wait_bounded(&lbars[0], 0);
  // no CTA leaves while another may still write into it: past the cluster
  // barrier the previous CTA has issued its whole row, and what a band that
  // gave up has not waited for is waited for (bounded) here
  if (cs > 1) {
    lu_cluster_sync();
    if (linked && __syncthreads_or(gfail >= 0) && w == 0)
      for (int i = 0; i < (ncol + LU_LG - 1) / LU_LG; ++i) lu_link_wait(&lbars[i], LU_POLL_DEFAULT);
  }
}

}  // namespace ot2d
