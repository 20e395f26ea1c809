"""The host-buffer path in parts (ot2d_solver_iterate_host) while the batch
changes under it: unlisted requests retire at several checks of one call, and
some parts hold no listed request, so that nothing but the order of the
streams keeps their iterations behind the rebuilt batch's time step."""
import ctypes as C

import numpy as np
import pytest

from turns2d_urans_git_gb300 import api
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED, OT2D_FP64

pytestmark = pytest.mark.gpu


def _cases(n, size=(129, 33)):
    return [api.config_c2(jmax=size[0], kmax=size[1], fsmach=0.2 + 0.01 * i, alfa=0.25 * i, rey=2e6, ds_wall=1e-4)
            for i in range(n)]


def _host_iterate(sv, ids, q, steps):
    L = api.lib()
    P = C.POINTER(C.c_double)
    L.ot2d_solver_iterate_host.argtypes = [C.c_void_p, C.c_int32, C.POINTER(C.c_int32), C.POINTER(P), C.c_int32]
    return L.ot2d_solver_iterate_host(sv._h, len(ids), (C.c_int32 * len(ids))(*ids),
                                      (P * len(q))(*[a.ctypes.data_as(P) for a in q]), steps)


@pytest.mark.parametrize("precision", [OT2D_FP64, OT2D_FP32_MIXED])
@pytest.mark.parametrize("listed", [[0], [1, 9, 17]])
def test_unlisted_requests_retire_during_the_call(precision, listed):
    cases, steps = _cases(24), 10
    caps = [1000 if k in listed or k >= 20 else 2 + k % 5 for k in range(24)]   # 16 or more retire at 2 .. 6
    caps = [1000 if k % 3 == 2 else c for k, c in enumerate(caps)]              # a third stay: the parts go on
    out = {}
    for path in ("device", "host"):
        sv = api.Solver(precision, check_every=1, keep_q=True)
        ids = [sv.add(c[1], c[2], c[3], orders=0.0, max_iters=m) for c, m in zip(cases, caps)]
        if path == "device":
            sv.iterate(steps)
        else:
            q = [np.ascontiguousarray(sv.get_q(ids[k], cases[k][1])) for k in listed]
            assert _host_iterate(sv, [ids[k] for k in listed], q, steps) == 0
        sv.sync()
        out[path] = [sv.get_q(i, c[1]) for i, c in zip(ids, cases)]
        for i, m in zip(ids, caps):
            assert sv.result(i).status == 0 and sv.result(i).iterations == min(m, steps)
        if path == "host":
            for k, a in zip(listed, q):
                assert np.array_equal(a, out["host"][k])
        sv.close()
    for a, b in zip(out["device"], out["host"]):
        assert np.array_equal(a, b)
