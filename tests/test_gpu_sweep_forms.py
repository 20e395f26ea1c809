"""The forms of the LU-SGS sweeps against each other, bit for bit: a request
alone (a cluster of CTAs per slice, wide groups in f32), a few requests of
different heights (clusters in which some CTAs have no band), and more
requests than the rule spreads (one CTA per slice, narrow groups in f32).  The
numbers come from the rule itself (csrc/kernels/lu_shape.h), and the forms are
checked to differ; plain and preconditioned, FP64 and f32."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from turns2d_urans_git_gb300 import api
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED, OT2D_FP64, OT2D_OPT_PIPELINE

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
KERNELS = os.path.join(HERE, "..", "turns2d_urans_git_gb300", "csrc", "kernels")
STEPS = 8

SHAPE = r"""
#include "lu_shape.h"
using namespace ot2d;
extern "C" int spread_slices() { return LU_SPREAD_SLICES; }
extern "C" void form(int es, int pre, int kd, int jd, int nslice, int* out) {
  const bool s = lu_spread(nslice, 0);
  const LuLaunch l = es == 4 ? (pre ? lu_launch<float, true>(kd, jd, s, 0) : lu_launch<float, false>(kd, jd, s, 0))
                             : (pre ? lu_launch<double, true>(kd, jd, s, 0) : lu_launch<double, false>(kd, jd, s, 0));
  out[0] = l.pg; out[1] = l.cs;
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    src, lib = d / "s.cpp", d / "s.so"
    src.write_text(SHAPE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", KERNELS, str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


def _run(precision, cases):
    sv = api.Solver(precision, check_every=STEPS, keep_q=True)
    sv.set_option(OT2D_OPT_PIPELINE, 0)          # one graph: every slice in one launch
    ids = [sv.add(c[1], c[2], c[3], orders=0.0, max_iters=STEPS) for c in cases]
    sv.iterate(STEPS)
    sv.sync()
    assert all(sv.result(i).status == 0 for i in ids)
    out = [sv.get_q(i, c[1]) for i, c in zip(ids, cases)]
    sv.close()
    return out


@pytest.mark.parametrize("precision", [OT2D_FP64, OT2D_FP32_MIXED])
@pytest.mark.parametrize("pre", [False, True])
@pytest.mark.parametrize("tall", [(65, 146), (97, 200)])
def test_forms_agree(shape, precision, pre, tall):
    cases = []
    for j, k in (tall, (49, 17), (81, 90)):
        c = api.config_c2(jmax=j, kmax=k, fsmach=0.3, alfa=1.0, rey=2e6, ds_wall=1e-3)
        if pre:
            c[1].iprecon, c[1].Mp = 1, 0.3
        cases.append(c)
    many = shape.spread_slices() + 1
    es, f1, fn = 4 if precision == OT2D_FP32_MIXED else 8, (C.c_int * 2)(), (C.c_int * 2)()
    shape.form(es, int(pre), tall[1] + 1, 98, len(cases), f1)
    shape.form(es, int(pre), tall[1] + 1, 98, many, fn)
    assert f1[1] > fn[1] >= 1                    # fewer CTAs per slice ...
    assert es == 8 or f1[0] > fn[0]              # ... and smaller groups
    alone = [_run(precision, [c])[0] for c in cases]
    few = _run(precision, cases)
    lots = _run(precision, [cases[i % 3] for i in range(many)])
    for i, q in enumerate(alone):
        assert np.all(np.isfinite(q))
        assert np.array_equal(q, few[i])
        for m in range(i, many, 3):
            assert np.array_equal(q, lots[m])
