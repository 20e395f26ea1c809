// lu_shape.h -- sizes of the LU-SGS sweeps (k_lusgs.cuh): how a mesh is cut
// into bands and records, the shared memory of a sweep CTA, and the launch
// that is chosen for a batch.  Plain C++, so that the host decides, and a
// test can check, what fits without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define LU_HD __host__ __device__ __forceinline__
#else
#define LU_HD inline
#endif

namespace ot2d {

// Lanes per cell and rows per band of the sweeps.  A sweep is a chain of
// ncol + nrow steps, so its time is the time of one step.  Two lanes per cell
// (both form the cell's correction, the even one its xi contribution, the odd
// one its eta contribution) leave an f32 step 70 instructions instead of 127
// and ~290 cycles; one lane per cell (bands of 32 rows) took 315.  FP64: the
// pipe takes a warp instruction every 64 cycles per SM sub-partition whatever
// the lanes do, so a step is the number of FP64 operations of a lane: 78 with
// one lane per cell (5900 cycles a step), 47 with two, 21 with four, one per
// variable (1930 cycles; the exchange between the lanes is the rest).  The
// preconditioned FP64 operator, whose preconditioner couples the four
// variables once more, stays at two.  Both sweeps and their records, 257x65
// FP64: 1710 -> 755 us; 385x97: 2658 -> 1150; FP32-mixed 769x193: 485 -> 301.
template <class R, bool PRE = false>
struct LuSplit {
  static constexpr int LP = (sizeof(R) == 8 && !PRE) ? 4 : 2;   // lanes per cell
  static constexpr int RB = 32 / LP;                            // rows per band
};

// A (band, step) chunk holds the records of the band's RB cells one after
// another (row-major): a cell's 24 fields are contiguous, so a lane reads
// several consecutive fields with 16-byte shared loads.  The record stride LS
// puts the rows of a load phase on disjoint banks: f32 24 elements (four rows
// and both directions' groups of a 16-byte phase cover the 32 banks), FP64 28
// (four rows x four 8-byte fields).  With Turkel preconditioning (PRE, the
// preilu2d operator of lhs.f:2-467) a record carries 8 more fields: the
// chk*qq products of both sweeps and the preconditioner factor.
template <class R, bool PRE = false>
struct LuLay {
  static constexpr int NF = PRE ? 32 : 24;                                   // fields per record
  static constexpr int LS = sizeof(R) == 4 ? (PRE ? 36 : 24) : (PRE ? 34 : 28);   // elements per cell record
  static constexpr int RB = LuSplit<R, PRE>::RB;
  static constexpr int CH = RB * LS;                                         // elements per chunk
};
LU_HD int lu_nrow(int kd) { return kd - 2; }
LU_HD int lu_ncol(int jd) { return jd - 2; }
// bands of rb rows and steps of a band
LU_HD int lu_nband(int kd, int rb) { return (kd - 2 + rb - 1) / rb; }
LU_HD int lu_nstep(int jd, int rb) { return jd - 2 + rb - 1; }
// elements of one slice's record (element size esize bytes): chunks + 4
// halo-contribution arrays, enough for the plain and the preconditioned
// layout so that a slice can use either (36 / 34 elements per cell in bands
// of 32 rows bound both)
LU_HD int64_t lu_rec_elems(int jd, int kd, int esize) {
  const int64_t ch = 32 * (esize == 4 ? 36 : 34);
  return (int64_t)lu_nband(kd, 32) * lu_nstep(jd, 32) * ch + 8 * (int64_t)(lu_nrow(kd) + lu_ncol(jd)) + 64;
}

// Cross-band ring: the last row of a band hands its outgoing (j,k-1)
// contribution at its p-th column (in sweep order) to the next band through
// slot p % LU_XB; the consumer's first row reads it at its own step p.
constexpr int LU_XB = 64;         // a power of two; a band may run this many columns ahead of the next
constexpr int LU_LG = 8;          // columns per barrier of a link between CTAs
constexpr int LU_MAX_WARPS = 16;  // bands per CTA of a sweep
constexpr int LU_MAX_CLUSTER = 8; // CTAs per slice

// PG, the steps per group: a group's records arrive with one bulk copy, and
// waits on the neighbouring bands are made and progress is published once per
// group, so a band trails the one before it by RB + PG steps.  A group's
// waits and bookkeeping cost about as much as two f32 steps: groups of 8 make
// a step 215 cycles, groups of 4 294 (f32 sweeps of a 513x33 mesh, 147 and
// 183 us), but hold twice the shared memory; in a batch whose sweeps share
// their SMs with the turbulence solve the smaller groups are faster (64
// 513x129 requests 1256 against 1402 us per iteration).  FP64 steps are an
// order longer: groups of 2, which trail least.
template <class R, bool WIDE>
LU_HD constexpr int lu_pg() { return sizeof(R) == 8 ? 2 : (WIDE ? 8 : 4); }
// Exchange buffer of a warp, through which the lanes of a step pass values on
// (a 16-byte store and load take the place of four shuffles).  A contribution
// made at step t goes to slot (t+1) % lu_ks() of its lane; the slots of a lane
// are 4 elements apart, as the columns of the cross-band ring are, so that a
// cell takes its eta input at the same step stride from either.
template <int PG>
LU_HD constexpr int lu_ks() { return PG < 4 ? 4 : PG; }
template <class R, bool PRE, int PG>
LU_HD constexpr int lu_ex() {
  return LuSplit<R, PRE>::LP == 2 ? 32 * 4 * (lu_ks<PG>() + 1) : 64 + 8 * 4 * (lu_ks<PG>() + 1);
}

// Shared memory of a sweep CTA of a cluster of cs: per warp D stages of a
// group's records with a barrier each, its cross-band ring with a full and an
// empty barrier per group of columns (a CTA of one warp has no ring), and its
// exchange buffer; then one row of contributions per column (at most maxcol):
// the halo's, with one barrier, for the CTA with the first band in sweep
// order, the previous CTA's last row, with one barrier per LU_LG columns, for
// the others.
LU_HD constexpr int lu_nring(int nwarp) { return nwarp > 1 ? nwarp : 0; }
LU_HD constexpr int lu_nlink(int cs, int maxcol) { return cs > 1 ? (maxcol + LU_LG - 1) / LU_LG : 1; }
template <class R, bool PRE, int PG>
LU_HD constexpr size_t lu_smem_bytes(int cs, int nwarp, int D, int maxcol) {
  return ((size_t)nwarp * (D * PG * LuLay<R, PRE>::CH + lu_ex<R, PRE, PG>()) + (size_t)lu_nring(nwarp) * LU_XB * 4 +
          (size_t)4 * maxcol) * sizeof(R) +
         ((size_t)nwarp * D + (size_t)lu_nring(nwarp) * 2 * (LU_XB / PG) + (size_t)lu_nlink(cs, maxcol)) * sizeof(uint64_t);
}

// Largest dynamic shared memory a CTA may opt in to on sm_103a (227 KB).
constexpr int SMEM_OPTIN_MAX = 227 * 1024;

// CTAs per slice of the sweeps (a cluster), for nb bands.  One warp per SM
// sub-partition (4 bands per CTA) makes a step fastest, but takes SMs from
// the residual and the turbulence solve of a large batch.  Measured per
// iteration (us), one CTA against ceil(nb / 4), RANS-SA in one launch.
// FP32-mixed, with the groups that go with each form (lu_pg): 513x129 alone 364,
// 275, 8 slices 454, 370, 16 slices 547, 474; 257x65 164, 151; 179, 164; 254,
// 199; 129x33 103, 97; 105, 101; 110, 106; 32 slices of 513x129 1276, 1328 and
// of 769x193 2715, 2786.  FP64: 513x129 alone 3675, 1771, 8 slices 4993, 3103,
// 16 slices 6431, 5068; 385x97 2180, 1320; 2949, 2100; 3791, 3121; 257x65 1167,
// 956; 1492, 1282; 1860, 1646; 129x33 the same (four bands: one CTA either way).
// Batches that run beside each other (halves, parts) share the SMs: in four
// parts, 64 slices of 513x129 (512 bands) 1228, 1269, of 385x97 (384) 747,
// 787, of 257x65 (256) 394, 383; 32 of 385x97 (192) 492, 483; FP64 257x65,
// 64 slices (512) 4697, 4759, 32 (256) 2680, 2641.
constexpr int LU_SPREAD_SLICES = 16, LU_SPREAD_BANDS = 256;
inline bool lu_spread(int nslice, int shared_bands) {
  return nslice <= LU_SPREAD_SLICES && shared_bands <= LU_SPREAD_BANDS;
}

// The launch of the sweeps: groups of pg steps, cs CTAs of nw warps per slice
// with D record stages per warp and smem bytes each; cs = 0: none fits.
struct LuLaunch { int pg = 0, cs = 0, nw = 0, D = 0; size_t smem = 0; };

// With groups of PG and at least mind stages.  More CTAs than the rule above
// only where the bands or their shared memory do not fit; group (0: as 8): in
// FP64 the stages where that is more than mind, within ~200 KB of shared
// memory.  (An f32 stage is four or eight steps: two are enough.)
template <class R, bool PRE, int PG>
inline LuLaunch lu_launch_pg(int nb, bool spread, int maxcol, int group, int mind) {
  const int want = spread ? std::min((nb + 3) / 4, LU_MAX_CLUSTER) : 1;
  for (int cs = want; cs <= LU_MAX_CLUSTER; ++cs) {
    const int nw = (nb + cs - 1) / cs;
    if (nw > LU_MAX_WARPS || lu_smem_bytes<R, PRE, PG>(cs, nw, mind, maxcol) > (size_t)SMEM_OPTIN_MAX) continue;
    int D = sizeof(R) == 8 && mind > 1 ? std::max(mind, group ? group : 8) : mind;
    while (D > mind && lu_smem_bytes<R, PRE, PG>(cs, nw, D, maxcol) > 200 * 1024) --D;
    return {PG, cs, nw, D, lu_smem_bytes<R, PRE, PG>(cs, nw, D, maxcol)};
  }
  return {};
}
// The choice for a batch whose largest mesh has kd_max rows and jd_max
// columns: where the wide groups do not fit eight CTAs (tall or long meshes,
// preconditioned ones first) the narrow ones, and where those do not (strips
// of thousands of columns) one stage per warp, whose copies then run between
// the groups and not beside them.
template <class R, bool PRE>
inline LuLaunch lu_launch(int kd_max, int jd_max, bool spread, int group) {
  constexpr int W = lu_pg<R, true>(), N = lu_pg<R, false>();
  const int nb = lu_nband(kd_max, LuSplit<R, PRE>::RB);   // jd_max: >= the columns of every slice
  LuLaunch l;
  if (spread) l = lu_launch_pg<R, PRE, W>(nb, spread, jd_max, group, 2);
  if (!l.cs) l = lu_launch_pg<R, PRE, N>(nb, spread, jd_max, group, 2);
  if (!l.cs) l = lu_launch_pg<R, PRE, N>(nb, spread, jd_max, group, 1);
  return l;
}

// The mesh limit of a batch (largest kd and jd of its slices; pre: it holds a
// preconditioned one): rows in bands of 32 with a two-chunk record ring (28
// f32 / 26 FP64 elements per cell, 36 / 34 preconditioned), a ring of 128
// columns and a counter per band, and one row of halo contributions within
// one CTA's shared memory, and the 3 doubles per wall cell that the force
// kernel stages.  The sweeps that set this limit are gone; it stays what it
// was, and lu_launch has a form for every mesh within it.
inline bool lu_mesh_fits(int es, bool pre, int kd_max, int jd_max) {
  if (kd_max < 3 || jd_max < 3 || kd_max - 2 > 1024) return false;
  const size_t ls = es == 4 ? (pre ? 36 : 28) : (pre ? 34 : 26), nb = (size_t)lu_nband(kd_max, 32);
  const size_t lu = nb * (2 * 32 * ls * es + 16 + 128 * 4 * es + 4) + 16 + 4 * (size_t)jd_max * es;
  return lu <= (size_t)SMEM_OPTIN_MAX && sizeof(double) * 3 * (size_t)jd_max <= (size_t)SMEM_OPTIN_MAX;
}

// ... and the launcher takes the batch, in whichever form its other slices
// and batches beside it call for (a preconditioned batch holds plain slices
// too)
template <class R>
inline bool lu_batch_fits(bool pre, int kd_max, int jd_max) {
  if (!lu_mesh_fits(sizeof(R), pre, kd_max, jd_max)) return false;
  for (bool spread : {false, true})
    if (!lu_launch<R, false>(kd_max, jd_max, spread, 0).cs || (pre && !lu_launch<R, true>(kd_max, jd_max, spread, 0).cs))
      return false;
  return true;
}

}  // namespace ot2d
