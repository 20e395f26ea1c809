// kernels_fp64.cu -- the plain FP64 path.  Compiled with -fmad=false so that
// a*b+c rounds twice, as the reference Fortran and the oracle evaluate it.
#include "launchers.cuh"
namespace ot2d {
OT2D_INSTANTIATE(double)

namespace {
__global__ void k_stqol(const double* __restrict__ q, double* __restrict__ qtn, double* __restrict__ qtnm1,
                        double* __restrict__ qnewt, int64_t qs, int nv, int ntac, int istep) {
  const int64_t n = qs * nv;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    mv_stqol_elem(q, qtn, qtnm1, qnewt, i, ntac, istep);
}

// The geometry of a routine call (GeomArgs), one thread per cell: the host's
// expressions (geom.cpp) in their order.  Formed on the host between copies
// it was most of a call on device arrays: rhsup 257x65 267 -> 116 us.
// Bound by launch latency at such sizes (two 8-byte reads per vertex and four
// writes per cell).
__global__ void k_geometry(const ot2d_params* __restrict__ P, GeomArgs g) {
  const ot2d_params& p = *P;
  const int jd = p.jd, jm = p.jmax, nh = p.nhalo;
  const int cid = blockIdx.x * blockDim.x + threadIdx.x;
  if (cid >= jd * p.kd) return;
  const int j = cid % jd + 1, k = cid / jd + 1;
  auto V = [&](const double* v, int a, int b) { return v[mv_at(jm, a, b)]; };
  const int a = j - nh + 1, b = k - nh + 1;
  const bool inside = a >= 1 && a <= jm && b >= 1 && b <= p.kmax;
  // the area swept by a face with the other vertex (a1, b1), over dt
  auto swept = [&](int a1, int b1, double sgn) {
    auto area = [&](const double* xn, const double* yn, const double* xo, const double* yo) {
      const double dx1 = V(xn, a, b) - V(xo, a1, b1), dy1 = V(yn, a, b) - V(yo, a1, b1);
      const double dx2 = V(xo, a, b) - V(xn, a1, b1), dy2 = V(yo, a, b) - V(yn, a1, b1);
      return sgn * (0.5 * (dx1 * dy2 - dx2 * dy1) / by(p.dt));
    };
    double t = area(g.xv, g.yv, g.xold, g.yold);
    if (p.ntac == 2 && p.istep > 1) t = 1.5 * t - 0.5 * area(g.xold, g.yold, g.xole, g.yole);
    return t;
  };
  if (g.faces) {
    double fx = 0, fy = 0, ft = 0, gx = 0, gy = 0, gt = 0;
    if (inside && b > 1 && k >= p.kbeg && k <= p.kend && j >= p.jbeg - 1 && j <= p.jend) {
      fx = (V(g.yv, a, b) - V(g.yv, a, b - 1));
      fy = -(V(g.xv, a, b) - V(g.xv, a, b - 1));
      if (g.speeds)
        ft = g.xold ? swept(a, b - 1, -1.)
                    : -0.5 * (V(g.ugv, a, b) + V(g.ugv, a, b - 1)) * fx - 0.5 * (V(g.vgv, a, b) + V(g.vgv, a, b - 1)) * fy;
    }
    if (inside && a > 1 && j >= p.jbeg && j <= p.jend && k >= p.kbeg - 1 && k <= p.kend) {
      gx = -(V(g.yv, a, b) - V(g.yv, a - 1, b));
      gy = (V(g.xv, a, b) - V(g.xv, a - 1, b));
      if (g.speeds)
        gt = g.xold ? swept(a - 1, b, 1.)
                    : -0.5 * (V(g.ugv, a, b) + V(g.ugv, a - 1, b)) * gx - 0.5 * (V(g.vgv, a, b) + V(g.vgv, a - 1, b)) * gy;
    }
    double* o = g.faces + cid;
    o[0] = fx; o[g.ws] = fy; o[2 * g.ws] = gx; o[3 * g.ws] = gy;
    if (g.speeds) { g.speeds[cid] = ft; g.speeds[g.ws + cid] = gt; }
  }
  if (g.sn) {
    double d = 0.0;
    if (j < p.jtail1 || j > p.jtail2 || k > 1) {
      double fx, fy;   // the wall face of the column, or the trailing edge
      if (j >= p.jtail1 && j <= p.jtail2) {
        fx = 0.5 * (V(g.xv, j - nh, 1) + V(g.xv, j - nh + 1, 1));
        fy = 0.5 * (V(g.yv, j - nh, 1) + V(g.yv, j - nh + 1, 1));
      } else {
        fx = V(g.xv, p.jtail1 - nh, 1);
        fy = V(g.yv, p.jtail1 - nh, 1);
      }
      const double dx = g.x[cid] - fx, dy = g.y[cid] - fy;
      d = root(dx * dx + dy * dy);
    }
    g.sn[cid] = d;
  }
}
}  // namespace

cudaError_t launch_geometry(const ot2d_params* d_p, int cells, const GeomArgs& g, cudaStream_t st) {
  k_geometry<<<(cells + 127) / 128, 128, 0, st>>>(d_p, g);
  return cudaGetLastError();
}

cudaError_t launch_stqol(const double* q, double* qtn, double* qtnm1, double* qnewt, int64_t qs, int nv, int ntac,
                         int istep, cudaStream_t st) {
  const int64_t n = qs * nv;
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  k_stqol<<<(int)blocks, 256, 0, st>>>(q, qtn, qtnm1, qnewt, qs, nv, ntac, istep);
  return cudaGetLastError();
}

cudaError_t branch_of_device(Branch*& out) {
  static thread_local Branch br[16];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  Branch& b = br[dev];
  if (!b.st) {
    if ((e = cudaStreamCreateWithFlags(&b.st, cudaStreamNonBlocking)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&b.join, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&b.join_end, cudaEventDisableTiming)) != cudaSuccess) return e;
    for (cudaEvent_t* ev : {&b.resid, &b.rbc, &b.edges})
      if ((e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming)) != cudaSuccess) return e;
  }
  out = &b;
  return cudaSuccess;
}
}
