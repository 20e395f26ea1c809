"""The LU-SGS sweeps at the edges of their band layout: bands with a single
row, meshes whose bands fill one or several CTAs of a cluster, short and long
rows, plain and preconditioned (ilu2d, lhs.f:470-814; preilu2d, lhs.f:2-467).

Tolerance of the FP64 drop-ins: 1e-12 relative, the bound of the FP64 path
(the sweeps keep the reference's operations, so they agree bit for bit)."""
import ctypes as C

import numpy as np
import pytest

from tests import oracle_binding as ob
from tests.helpers import Case, relerr
from turns2d_urans_git_gb300 import api, routines as rt
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED, OT2D_FP64

pytestmark = pytest.mark.gpu


# interior rows = kmax - 1: 8, 9, 16, 17 (one row past a band of 8 / 16), 33
# (five FP64 bands: two CTAs), 72 (nine: three), 130 (17: five), 257 (33 FP64
# bands: eight CTAs of five warps)
@pytest.mark.parametrize("size", [(33, 9), (41, 10), (65, 17), (35, 18), (41, 34), (97, 73), (49, 131), (65, 258)])
@pytest.mark.parametrize("pre", [False, True])
def test_lusgs_band_layouts(size, pre):
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


@pytest.mark.parametrize("precision", [OT2D_FP64, OT2D_FP32_MIXED])
@pytest.mark.parametrize("size", [(65, 74), (49, 131)])
def test_cluster_and_single_cta_sweeps_agree(precision, size):
    """A request alone (its sweeps on a cluster of CTAs) and among 13 (one
    CTA per request) gives the same state bit for bit."""
    case = api.config_c2(jmax=size[0], kmax=size[1], fsmach=0.3, alfa=1.0, rey=2e6, ds_wall=1e-3)

    def run(n):
        sv = api.Solver(precision, check_every=10, keep_q=True)
        sv.set_option(10, 0)
        ids = [sv.add(case[1], case[2], case[3], orders=0.0, max_iters=10) for _ in range(n)]
        sv.iterate(10)
        sv.sync()
        assert all(sv.result(i).status == 0 for i in ids)
        out = [sv.get_q(i, case[1]) for i in ids]
        sv.close()
        return out

    alone, = run(1)
    many = run(13)
    assert np.all(np.isfinite(alone))
    assert np.array_equal(alone, many[0]) and np.array_equal(alone, many[12])
