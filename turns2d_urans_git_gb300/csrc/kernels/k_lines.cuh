// k_lines.cuh -- recurrences along the j-lines of a mesh through staged tiles.
//
// A line along j is contiguous in memory, so one lane per line would read a
// different cache line with every lane.  A CTA of four warps takes 32 lines:
// tiles of 32 lines x 32 columns of every array pass through shared memory in
// three buffers.  Warp 0 works: lane l walks line l through the tile and
// reads and writes shared memory only.  Warps 1..3 move: while warp 0 works
// on tile t they store the results of tile t-1 and fetch tile t+2 (cp.async),
// each its share of the rows, so the recurrence neither waits on global
// memory nor spends its issue slots on copies.  (With a single moving warp
// the copies, about 1100 instructions per tile of four arrays, and not the
// recurrence set the time.)
#pragma once
#include "dev_common.cuh"

namespace ot2d {

constexpr int JL_TILE = 32 * 33;       // one array of a tile, rows padded to 33
constexpr int JL_NBUF = 3;
constexpr int JL_MOVERS = 3;           // moving warps
constexpr int JL_THREADS = 32 * (1 + JL_MOVERS);
// shared-memory elements for NA arrays
__host__ __device__ constexpr int jl_smem_elems(int na) { return JL_NBUF * na * JL_TILE; }

template <class R>
__device__ __forceinline__ void jl_cp_async(R* dst, const R* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "n"((int)sizeof(R))
               : "memory");
}
__device__ __forceinline__ void jl_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void jl_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
// the warps of the CTA meet (named barrier 1)
__device__ __forceinline__ void jl_meet() { asm volatile("bar.sync 1, %0;" ::"n"(JL_THREADS) : "memory"); }

// Forward pass over columns js..je, then backward pass, of the nrow lines
// k0 .. k0+nrow-1 (1-based rows of arrays with row length jd).  src[a]: the
// NA arrays read by the forward pass; dst[a]: where results of array a go and
// where the backward pass reads it.  FST / BLD / BST: bit a set if array a is
// stored by the forward pass / read by the backward pass / stored by it (BST
// within BLD).  fwd(t, j) and bwd(t, j) work on column j of the lane's line:
// array a's value at t[a * JL_TILE].
template <class R, int NA, unsigned FST, unsigned BLD, unsigned BST, class Fwd, class Bwd>
__device__ __forceinline__ void jl_solve(R* const (&src)[NA], R* const (&dst)[NA], int jd, int js, int je, int k0,
                                         int nrow, R* sm, Fwd fwd, Bwd bwd) {
  const int lane = threadIdx.x & 31, wid = (int)(threadIdx.x >> 5) - 1;
  const bool mover = wid >= 0;
  const int ntile = (je - js + 1 + 31) / 32;
  const bool mine = lane < nrow;
  auto buf = [&](int b) { return sm + b * NA * JL_TILE; };
  // movers: copies of tile t of the arrays in mask into buffer b, one
  // cp.async group; each lane copies column `lane` of the warp's rows, the
  // same elements it stores below
  auto fetch = [&](R* const (&arr)[NA], unsigned mask, int t, int b) {
    const int j = js + 32 * t + lane;
    if (j <= je) {
      int64_t o = at(jd, j, k0 + wid);
      R* d = buf(b) + wid * 33 + lane;
      for (int r = wid; r < nrow; r += JL_MOVERS) {
#pragma unroll
        for (int a = 0; a < NA; ++a)
          if (mask >> a & 1) jl_cp_async(d + a * JL_TILE, arr[a] + o);
        o += (int64_t)JL_MOVERS * jd;
        d += JL_MOVERS * 33;
      }
    }
    jl_commit();
  };
  auto store = [&](unsigned mask, int t, int b) {
    const int j = js + 32 * t + lane;
    if (j <= je) {
      int64_t o = at(jd, j, k0 + wid);
      const R* s = buf(b) + wid * 33 + lane;
      for (int r = wid; r < nrow; r += JL_MOVERS) {
#pragma unroll
        for (int a = 0; a < NA; ++a)
          if (mask >> a & 1) dst[a][o] = s[a * JL_TILE];
        o += (int64_t)JL_MOVERS * jd;
        s += JL_MOVERS * 33;
      }
    }
  };
  constexpr unsigned ALL = (1u << NA) - 1;
  // Forward.  Round t: tile t in buffer t % 3; the movers store tile t-1 and
  // then fetch tile t+2 into the buffer tile t-1 used (a lane's stores read
  // the elements its copies overwrite), and wait for tile t+1.
  if (mover) {
    fetch(src, ALL, 0, 0);
    if (ntile > 1) { fetch(src, ALL, 1, 1); jl_wait<1>(); }
    else jl_wait<0>();
  }
  jl_meet();
  for (int t = 0; t < ntile; ++t) {
    const int b = t % JL_NBUF;
    if (!mover) {
      if (mine) {
        R* p = buf(b) + lane * 33;
        const int j0 = js + 32 * t, n = min(32, je - j0 + 1);
        if (n == 32) {
#pragma unroll 8
          for (int jj = 0; jj < 32; ++jj) fwd(p + jj, j0 + jj);
        } else {
          for (int jj = 0; jj < n; ++jj) fwd(p + jj, j0 + jj);
        }
      }
    } else {
      const int bf = (t + 2) % JL_NBUF;   // = (t - 1) % 3
      if (t >= 1) store(FST, t - 1, bf);
      if (t + 2 < ntile) { fetch(src, ALL, t + 2, bf); jl_wait<1>(); }
      else jl_wait<0>();
    }
    jl_meet();
  }
  // Backward.  Round n: tile ntile-1-n in buffer n % 3.
  if (mover) {
    store(FST, ntile - 1, (ntile - 1) % JL_NBUF);
    // what was stored is read back below by the same lanes; order the stores
    // before the asynchronous copies
    __threadfence_block();
    fetch(dst, BLD, ntile - 1, 0);
    if (ntile > 1) { fetch(dst, BLD, ntile - 2, 1); jl_wait<1>(); }
    else jl_wait<0>();
  }
  jl_meet();
  for (int t = ntile - 1, n = 0; t >= 0; --t, ++n) {
    const int b = n % JL_NBUF;
    if (!mover) {
      if (mine) {
        R* p = buf(b) + lane * 33;
        const int j0 = js + 32 * t, m = min(32, je - j0 + 1);
        if (m == 32) {
#pragma unroll 8
          for (int jj = 31; jj >= 0; --jj) bwd(p + jj, j0 + jj);
        } else {
          for (int jj = m - 1; jj >= 0; --jj) bwd(p + jj, j0 + jj);
        }
      }
    } else {
      const int bf = (n + 2) % JL_NBUF;   // = (n - 1) % 3
      if (n >= 1) store(BST, t + 1, bf);
      if (t - 2 >= 0) { fetch(dst, BLD, t - 2, bf); jl_wait<1>(); }
      else jl_wait<0>();
    }
    jl_meet();
  }
  if (mover) store(BST, 0, (ntile - 1) % JL_NBUF);
}

// lsolvej (samodel2d.f:1306-1344, komegasst.f:1435-1475) of the tridiagonal
// systems a, b, c, s along the j-lines k0 .. k0+nrow-1: x * b replaces s, c is
// overwritten.  SAOUT: ((x + 0) - 0) * b, as vmu_sa forms it with s2 = 0
// (samodel2d.f:150-153).
template <class R, bool SAOUT>
__device__ void tri_solve_j(R* a, R* b, R* c, R* s, int jd, int js, int je, int k0, int nrow, R* sm) {
  R* const arr[4] = {a, b, c, s};
  R cp = (R)0, sp = (R)0, xn = (R)0;
  jl_solve<R, 4, 12u, 14u, 8u>(
      arr, arr, jd, js, je, k0, nrow, sm,
      [&](R* t, int j) {
        const R av = j == js ? (R)0 : t[0];
        const R bb = (R)1. / by(t[JL_TILE] - av * cp);
        sp = (t[3 * JL_TILE] - av * sp) * bb;
        cp = t[2 * JL_TILE] * bb;
        t[3 * JL_TILE] = sp;
        t[2 * JL_TILE] = cp;
      },
      [&](R* t, int j) {
        const R sv = t[3 * JL_TILE];
        xn = j == je ? sv : sv - t[2 * JL_TILE] * xn;
        if constexpr (SAOUT) t[3 * JL_TILE] = ((xn + (R)0.) - (R)0.) * t[JL_TILE];
        else t[3 * JL_TILE] = xn * t[JL_TILE];
      });
}

// lsolvek (samodel2d.f:1347-1385, komegasst.f:1478-1518) of the systems a, b,
// c, s along the line at column j, one thread per line: x replaces s.  The
// line is walked in chunks whose loads are issued one chunk ahead.  Lanes are
// neighbouring columns, so the loads coalesce; a warp per SM leaves nothing
// to hide them, which is why the chunks are long and what follows the solve
// (updates of the state) is a kernel over the cells.
template <class R>
__device__ void tri_solve_k(const R* a, const R* b, R* c, R* s, int jd, int ks, int ke, int j) {
  constexpr int U = sizeof(R) == 4 ? 16 : 8;
  R sp = (R)0, cp = (R)0;
  {
    R na[U], nb[U], nc[U], ns[U];
    auto load = [&](int k0) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u <= ke) { const int64_t o = at(jd, j, k0 + u); na[u] = a[o]; nb[u] = b[o]; nc[u] = c[o]; ns[u] = s[o]; }
    };
    load(ks);
    for (int k0 = ks; k0 <= ke; k0 += U) {
      R ra[U], rb[U], rc[U], rs[U];
#pragma unroll
      for (int u = 0; u < U; ++u) { ra[u] = na[u]; rb[u] = nb[u]; rc[u] = nc[u]; rs[u] = ns[u]; }
      if (k0 == ks) ra[0] = (R)0;
      if (k0 + U <= ke) load(k0 + U);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u <= ke) {
          const int64_t o = at(jd, j, k0 + u);
          const R bb = (R)1. / by(rb[u] - ra[u] * cp);
          sp = (rs[u] - ra[u] * sp) * bb;
          cp = rc[u] * bb;
          s[o] = sp;
          c[o] = cp;
        }
    }
  }
  R nc[U], ns[U], x = sp;
  auto load = [&](int k0) {   // rows k0, k0-1, ...
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k0 - u >= ks) { const int64_t o = at(jd, j, k0 - u); nc[u] = c[o]; ns[u] = s[o]; }
  };
  load(ke);
  for (int k0 = ke; k0 >= ks; k0 -= U) {
    R rc[U], rs[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { rc[u] = nc[u]; rs[u] = ns[u]; }
    if (k0 - U >= ks) load(k0 - U);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k0 - u >= ks) {
        if (k0 - u < ke) x = rs[u] - rc[u] * x;
        s[at(jd, j, k0 - u)] = x;
      }
  }
}

}  // namespace ot2d
