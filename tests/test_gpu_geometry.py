"""The geometry that the drop-in routines form from the caller's grid (face
normals, face speeds, wall distance), through rhsup and vmu_sa against the
oracle: host arrays and device arrays, each twice (a first call allocates its
staging space, the next ones use what is kept).  Tolerance 1e-12 relative,
the bound of the FP64 path; the second call's results equal the first's bit
for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests import oracle_binding as ob
from tests.helpers import Case, relerr
from turns2d_urans_git_gb300 import routines as rt

pytestmark = pytest.mark.gpu
TOL = 1e-12
SIZES = [(21, 12), (33, 31), (67, 66), (257, 129)]


def _place(a, device):
    return torch.from_numpy(np.array(a)).cuda() if device else np.array(a)


def _host(a):
    return a.cpu().numpy() if hasattr(a, "cpu") else a


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("ts", [False, True])
def test_rhsup_geometry(size, device, ts):
    c = Case(jmax=size[0], kmax=size[1], seed=3, ds_wall=1e-3)
    c.p.timespectral = 1 if ts else 0
    g = np.random.default_rng(4)
    c.ugv[:], c.vgv[:] = g.uniform(-0.1, 0.1, c.ugv.size), g.uniform(-0.1, 0.1, c.vgv.size)
    s0 = g.uniform(-1, 1, c.n2 * c.p.nv) * 1e-3
    so = s0.copy()
    ob.lib().oro_rhsup(C.byref(c.p), *[ob.ptr(a) for a in (c.q, so, c.xv, c.yv, c.iblank, c.ugv, c.vgv)])
    rt.set_params(c.p)
    a = [_place(v, device) for v in (c.q, c.xx, c.xy, c.yx, c.yy, c.x, c.y, c.xv, c.yv, c.iblank, c.ugv, c.vgv, c.bt)]
    q, xx, xy, yx, yy, x, y, xv, yv, ib, ugv, vgv, bt = a
    out = []
    for _ in range(2):
        s = _place(s0, device)
        torch.cuda.synchronize()
        rt.rhsup(q, s, xx, xy, yx, yy, x, y, xv, yv, xv, yv, xv, yv, ib, ugv, vgv, c.jd, c.kd, 1, 1, bt)
        out.append(_host(s))
    assert relerr(out[0], so) <= TOL
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("device", [False, True])
def test_vmu_sa_wall_distance(size, device):
    c = Case(jmax=size[0], kmax=size[1], viscous=True, seed=11, ds_wall=1e-3)
    L = ob.lib()
    L.oro_time_step(C.byref(c.p), *[ob.ptr(a) for a in (c.q, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg, c.tscale, c.bt, c.iblank)])
    s0 = np.random.default_rng(5).uniform(-1, 1, c.n2 * c.p.nv) * 1e-6
    geo = (c.x, c.y, c.xv, c.yv, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg)
    qo, so, to = c.q.copy(), s0.copy(), c.turmu.copy()
    L.oro_vmu_sa(C.byref(c.p), ob.ptr(qo), ob.ptr(so), ob.ptr(to), *[ob.ptr(a) for a in geo], ob.ptr(c.tscale),
                 ob.ptr(c.iblank))
    rt.set_params(c.p)
    dgeo = [_place(a, device) for a in geo]
    ts, ib = _place(c.tscale, device), _place(c.iblank, device)
    out = []
    for _ in range(2):
        q, s, t = (_place(a, device) for a in (c.q, s0, c.turmu))
        torch.cuda.synchronize()
        rt.vmu_sa(q, s, t, *dgeo, c.jd, c.kd, ts, ib, 1, 1)
        out.append((_host(q), _host(t)))
    assert relerr(out[0][0], qo) <= TOL and relerr(out[0][1], to) <= TOL
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
