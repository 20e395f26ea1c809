"""A drop-in call follows the work that its caller has queued on the default
stream for the arrays it reads, without a synchronisation in between: vmu_sa
on a q that a copy behind a 20 ms delay is still to fill, with the mesh in
host memory and in device memory."""
import numpy as np
import pytest
import torch

from tests.helpers import Case
from turns2d_urans_git_gb300 import routines as rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_mesh", [False, True])
def test_vmu_sa_follows_pending_work(device_mesh):
    c = Case(jmax=65, kmax=25, viscous=True, seed=11, ds_wall=1e-3)
    c.tscale[:] = 0.1
    place = (lambda a: torch.from_numpy(np.array(a)).cuda()) if device_mesh else np.array
    geo = [place(a) for a in (c.x, c.y, c.xv, c.yv, c.xx, c.xy, c.yx, c.yy, c.ug, c.vg)]
    ts, ib = place(c.tscale), place(c.iblank)
    state = torch.from_numpy(np.array(c.q)).cuda()
    other = torch.from_numpy(Case(jmax=65, kmax=25, viscous=True, seed=12, ds_wall=1e-3).q).cuda()
    s, turmu0 = torch.zeros(c.n2 * c.p.nv, dtype=torch.float64, device="cuda"), torch.from_numpy(np.array(c.turmu)).cuda()
    rt.set_params(c.p)

    def call(pending):
        q, turmu = other.clone(), turmu0.clone()
        torch.cuda.synchronize()
        if pending:
            torch.cuda._sleep(40_000_000)
        q.copy_(state)
        if not pending:
            torch.cuda.synchronize()
        rt.vmu_sa(q, s, turmu, *geo, c.jd, c.kd, ts, ib, 1, 1)
        torch.cuda.synchronize()
        return q.cpu().numpy(), turmu.cpu().numpy()

    for _ in range(2):                       # a first call allocates, which synchronises by itself
        ref = call(False)
    got = call(True)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
