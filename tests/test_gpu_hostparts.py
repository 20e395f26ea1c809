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


def test_resident_iterations_stay_as_they_were():
    """A call of the host-buffer path leaves the device-resident iteration's
    launches alone: its parts are its own.  The two paths in turn give the
    bits of the device path alone.  A refused call changes nothing either."""
    cases = _cases(20)
    L = api.lib()
    L.ot2d_solver_graph_kernels.argtypes = [C.c_void_p]

    def run(host):
        sv = api.Solver(OT2D_FP32_MIXED, check_every=100, keep_q=True)
        ids = [sv.add(c[1], c[2], c[3], orders=0.0, max_iters=1000) for c in cases]
        sv.iterate(3)
        kernels = L.ot2d_solver_graph_kernels(sv._h)
        if host:
            q = [np.ascontiguousarray(sv.get_q(i, c[1])) for i, c in zip(ids, cases)]
            assert _host_iterate(sv, [ids[0], 12345], q[:2], 1) != 0    # no such request
            assert L.ot2d_solver_graph_kernels(sv._h) == kernels
            assert _host_iterate(sv, ids, q, 2) == 0
        else:
            sv.iterate(2)
        assert L.ot2d_solver_graph_kernels(sv._h) == kernels
        sv.iterate(3)
        sv.sync()
        out = [sv.get_q(i, c[1]) for i, c in zip(ids, cases)]
        sv.close()
        return kernels, out

    (ka, a), (kb, b) = run(False), run(True)
    assert ka == kb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
