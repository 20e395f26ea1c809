"""FP64 division and square root on the integer pipe against the IEEE ones.

The host build of the functions takes the relative error of the
single-precision estimates as a parameter: 2**-22 either way is twice what
rcp.approx and rsqrt.approx are documented to be off.  Results are compared
bit for bit (NaNs as NaNs).
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
KERNELS = os.path.join(HERE, "..", "turns2d_urans_git_gb300", "csrc", "kernels")

HOST = r"""
#include "soft64.h"
extern "C" void run(const double* a, const double* b, double* q, double* r, long n, float err) {
  ot2d::soft64::seed_error() = err;
  for (long i = 0; i < n; ++i) { q[i] = ot2d::soft64::div(a[i], b[i]); r[i] = ot2d::soft64::sqrt_rn(a[i]); }
}
"""
DEVICE = r"""
#include "soft64.h"
__global__ void k(const double* a, const double* b, double* q, double* r, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { q[i] = ot2d::soft64::div(a[i], b[i]); r[i] = ot2d::soft64::sqrt_rn(a[i]); }
}
extern "C" int run(const double* a, const double* b, double* q, double* r, long n) {
  k<<<(unsigned)((n + 255) / 256), 256>>>(a, b, q, r, n);
  return (int)cudaDeviceSynchronize();
}
"""


def operands(n, seed):
    """Pairs with significands at random, near 1 and near 2, exponents near 1
    and over the whole range, exact quotients and squares, and the specials."""
    g = np.random.default_rng(seed)

    def values(m):
        frac = g.integers(0, 1 << 52, m, dtype=np.uint64)
        low = g.integers(0, 256, m, dtype=np.uint64) << g.integers(0, 45, m, dtype=np.uint64)
        kind = g.integers(0, 4, m)
        frac = np.where(kind == 1, low, np.where(kind == 2, (1 << 52) - 1 - low, frac)).astype(np.uint64)
        ex = np.where(kind == 3, g.integers(0, 2048, m), g.integers(963, 1083, m)).astype(np.uint64)
        sign = g.integers(0, 2, m, dtype=np.uint64)
        return ((sign << np.uint64(63)) | (ex << np.uint64(52)) | frac).view(np.float64)

    a, b = values(n), values(n)
    with np.errstate(all="ignore"):
        a[::7] = a[::7] * b[::7]                     # at or beside an exact quotient
        a[1::7] = (np.abs(a[1::7]).astype(np.float32).astype(np.float64)) ** 2    # exact roots
        a[2::7] = np.abs(a[2::7])
    tiny, big = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    sp = np.array([0.0, -0.0, 1.0, -1.0, 3.0, np.inf, -np.inf, np.nan, tiny, -tiny, tiny / 2, 5e-324, big, -big,
                   1.0 + 2**-52, 2.0 - 2**-52, 1.0 - 2**-53, 2**-1021.0, 2**1023.0])
    x, y = np.meshgrid(sp, sp)
    return np.concatenate([a, x.ravel()]), np.concatenate([b, y.ravel()])


def same(x, ref):
    return (x.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(x) & np.isnan(ref))


def reference(a, b):
    with np.errstate(all="ignore"):
        return a / b, np.sqrt(a)


@pytest.mark.parametrize("err", [0.0, 2.0**-22, -(2.0**-22)])
def test_host(tmp_path, err):
    src, lib = tmp_path / "h.cpp", tmp_path / "h.so"
    src.write_text(HOST)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", KERNELS, str(src), "-o",
                    str(lib)], check=True)
    run = ctypes.CDLL(str(lib)).run
    P = ctypes.c_void_p
    run.argtypes = [P, P, P, P, ctypes.c_long, ctypes.c_float]
    a, b = operands(1 << 20, 1)
    q, r = np.empty_like(a), np.empty_like(a)
    run(a.ctypes.data, b.ctypes.data, q.ctypes.data, r.ctypes.data, len(a), err)
    rq, rr = reference(a, b)
    assert same(q, rq).all() and same(r, rr).all()


@pytest.mark.gpu
def test_device(tmp_path):
    import torch

    src, lib = tmp_path / "d.cu", tmp_path / "d.so"
    src.write_text(DEVICE)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-fmad=false", "-gencode", "arch=compute_103a,code=sm_103a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", KERNELS, str(src), "-o", str(lib)], check=True)
    run = ctypes.CDLL(str(lib)).run
    P = ctypes.c_void_p
    run.argtypes = [P, P, P, P, ctypes.c_long]
    a, b = operands(1 << 24, 2)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dq, dr = torch.empty_like(da), torch.empty_like(da)
    torch.cuda.synchronize()
    assert run(da.data_ptr(), db.data_ptr(), dq.data_ptr(), dr.data_ptr(), len(a)) == 0
    rq, rr = reference(a, b)
    assert same(dq.cpu().numpy(), rq).all() and same(dr.cpu().numpy(), rr).all()
