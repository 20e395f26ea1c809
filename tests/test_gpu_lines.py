"""The line solves at the edges of their tiles and chunks: arc2d's
pentadiagonal and tridiagonal inversions (lhs.f:817-1057), the SA solve
(samodel2d.f:2-197) and the k-omega SST solve (komegasst.f:2-187), FP64
drop-ins against the oracle.

Lines along j are solved in tiles of 32 columns by CTAs of 32 lines, lines
along k in chunks of 4 (FP64) or 8 rows: the sizes leave one tile or chunk
exactly full, one column or row over, and partial ones.  Tolerance 1e-12
relative, the bound of the FP64 path."""
import ctypes as C

import numpy as np
import pytest

from tests import oracle_binding as ob
from tests.helpers import Case, relerr
from turns2d_urans_git_gb300 import routines as rt

pytestmark = pytest.mark.gpu
TOL = 1e-12
# interior columns jmax - 1, rows kmax - 1 (arc2d: kmax + 1 lines along j)
SIZES = [(21, 12), (33, 31), (35, 32), (65, 33), (67, 66)]


def _case(size, iturb=1):
    c = Case(jmax=size[0], kmax=size[1], viscous=True, seed=11, iturb=iturb, ds_wall=1e-3)
    ob.lib().oro_time_step(C.byref(c.p), *[ob.ptr(a) for a in (c.q, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg, c.tscale, c.bt,
                                                               c.iblank)])
    rt.set_params(c.p)
    return c


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("ilhs", [2, 3])
def test_arc2d_line_edges(size, ilhs):
    c = _case(size)
    p = c.p
    p.ilhs = ilhs
    rt.set_params(p)
    so = np.random.default_rng(23).uniform(-1, 1, c.n2 * p.nv) * 1e-4
    s, qo, q = so.copy(), c.q.copy(), c.q.copy()
    args = (c.xx, c.xy, c.yx, c.yy, c.ug, c.vg, c.turmu, c.iblank, c.tscale, c.bt)
    ob.lib().oro_arc2d(C.byref(p), ob.ptr(qo), ob.ptr(so), *[ob.ptr(a) for a in args])
    rt.arc2d(q, s, c.jd, c.kd, p.jbeg, p.jend, p.kbeg, p.kend, *args)
    assert relerr(s[:4 * c.n2], so[:4 * c.n2]) <= TOL
    assert relerr(q, qo) <= TOL


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("iturb", [1, 2])
def test_turbulence_line_edges(size, iturb):
    c = _case(size, iturb)
    so = np.random.default_rng(5).uniform(-1, 1, c.n2 * c.p.nv) * 1e-6
    s, qo, q, to, t = so.copy(), c.q.copy(), c.q.copy(), c.turmu.copy(), c.turmu.copy()
    geo = (c.x, c.y, c.xv, c.yv, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg)
    f = ob.lib().oro_vmu_sa if iturb == 1 else ob.lib().oro_komegasst
    f(C.byref(c.p), ob.ptr(qo), ob.ptr(so), ob.ptr(to), *[ob.ptr(a) for a in geo], ob.ptr(c.tscale), ob.ptr(c.iblank),
      *(() if iturb == 1 else (None,)))
    if iturb == 1:
        rt.vmu_sa(q, s, t, *geo, c.jd, c.kd, c.tscale, c.iblank, 1, 1)
    else:
        rt.komegasst(q, s, t, *geo, c.jd, c.kd, c.tscale, c.iblank, 1)
    turb = slice(4 * c.n2, (4 + iturb) * c.n2)
    assert not np.array_equal(qo[turb], c.q[turb])
    assert relerr(q[turb], qo[turb]) <= TOL
    assert relerr(t, to) <= TOL
