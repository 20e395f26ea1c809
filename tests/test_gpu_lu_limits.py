"""LU-SGS sweeps on meshes near the limit of what a solver admits, where a
sweep takes a smaller form of itself (lu_shape.h): narrow instead of wide
groups in f32, one CTA per band without a ring, one record stage per band.

Tolerance of the FP64 drop-ins: 1e-12 relative, the bound of the FP64 path.
The f32 form is compared bit for bit with another launch of the same mesh (the
FP64 path's limit is lower)."""
import ctypes as C

import numpy as np
import pytest

from tests import oracle_binding as ob
from tests.helpers import Case, relerr
from turns2d_urans_git_gb300 import api, routines as rt
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED, OT2D_OPT_PIPELINE

pytestmark = pytest.mark.gpu


# array sizes jd, kd = vertices + 1.  Plain: the longest strips (jd 6718; kd
# 34: four CTAs of a warp, kd 10: one band); preconditioned: jd 6590, one
# stage (kd 34: two CTAs of a warp, kd 12: one band)
@pytest.mark.parametrize("size,pre", [((6717, 33), False), ((6717, 9), False), ((6589, 33), True), ((6589, 11), True)])
def test_longest_strips(size, pre):
    c = Case(jmax=size[0], kmax=size[1], viscous=True, seed=8, ds_wall=1e-3)
    p, L, pp = c.p, ob.lib(), C.byref(c.p)
    p.Mp = 0.5 if pre else 1.0
    L.oro_time_step(pp, *[ob.ptr(a) for a in (c.q, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg, c.tscale, c.bt, c.iblank)])
    so = np.random.default_rng(4).uniform(-1, 1, c.n2 * p.nv) * 1e-4
    s, qo, q = so.copy(), c.q.copy(), c.q.copy()
    args = (c.xx, c.xy, c.yx, c.yy, c.ug, c.vg, c.turmu, c.tscale) + ((c.bt,) if pre else ())
    (L.oro_preilu2d if pre else L.oro_ilu2d)(pp, ob.ptr(qo), ob.ptr(so), *[ob.ptr(a) for a in args])
    rt.set_params(p)
    (rt.preilu2d if pre else rt.ilu2d)(q, s, c.jd, c.kd, p.jbeg, p.jend, p.kbeg, p.kend, *args)
    assert relerr(s, so) <= 1e-12
    assert relerr(q, qo) <= 1e-12


# f32, at most 16 slices: wide groups of records do not fit eight CTAs here, so
# a request alone runs the narrow groups on a cluster; among 17 (and with the
# wide form never considered) on as few CTAs as hold its bands
@pytest.mark.parametrize("size,pre", [((1201, 520), True), ((6601, 390), False)])
def test_tall_f32_meshes_take_the_narrow_groups(size, pre):
    case = api.cmesh_case(size[0], size[1], ds_wall=2e-3, irhsy=-3, ilim=1, ilhs=1, iconstant_cfl=1, dt=2.0, fsmach=0.3,
                          alfa=1.0, invisc=1, lamin=1)
    prm = case[1]
    if pre:
        prm.iprecon, prm.Mp = 1, 0.3

    def run(n):
        sv = api.Solver(OT2D_FP32_MIXED, check_every=3, keep_q=True)
        sv.set_option(OT2D_OPT_PIPELINE, 0)
        ids = [sv.add(prm, case[2], case[3], orders=0.0, max_iters=100) for _ in range(n)]
        sv.iterate(3)
        sv.sync()
        assert all(sv.result(i).status == 0 and sv.result(i).iterations == 3 for i in ids)
        q = [sv.get_q(i, prm) for i in (ids[0], ids[-1])]
        sv.close()
        return q

    alone = run(1)[0]
    assert np.all(np.isfinite(alone))
    for q in run(17):
        assert np.array_equal(q, alone)
