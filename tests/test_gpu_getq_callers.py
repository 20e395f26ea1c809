"""ot2d_solver_get_q for callers other than one thread with the solver's
device current: a thread whose current context is another one, and several
threads that read states of one solver at once.  Fresh buffers, whose copies
go through the solver's pinned chunks."""
import ctypes as C
import mmap
import threading

import numpy as np
import pytest

from turns2d_urans_git_gb300 import api
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED

pytestmark = pytest.mark.gpu


def _solver(n):
    cases = [api.cmesh_case(257, 129, ds_wall=2e-3, irhsy=-3, ilim=1, ilhs=1, iconstant_cfl=1, dt=2.0, fsmach=0.3,
                            alfa=0.5 * i, invisc=1, lamin=1) for i in range(n)]
    sv = api.Solver(OT2D_FP32_MIXED)
    ids = [sv.add(c[1], c[2], c[3], orders=0.0, max_iters=1000) for c in cases]
    sv.iterate(2)
    return sv, ids, [c[1] for c in cases]


def _fresh(p):
    return np.frombuffer(mmap.mmap(-1, 8 * p.jd * p.kd * p.nspec * p.nq))


def _get(sv, i, q):
    return api.lib().ot2d_solver_get_q(sv._h, i, q.ctypes.data_as(C.POINTER(C.c_double)))


def test_another_context_is_current():
    """The thread's current context is a second one on the same GPU, as after
    work on another device: the solver's own device is used for the copy."""
    cu = C.CDLL("libcuda.so.1")
    sv, ids, prm = _solver(1)
    ref = _fresh(prm[0])
    assert _get(sv, ids[0], ref) == 0
    other, (sv2, ids2, prm2) = C.c_void_p(), _solver(1)     # sv2: nothing of its copies set up yet
    assert cu.cuCtxCreate_v2(C.byref(other), 0, 0) == 0
    try:
        q = _fresh(prm2[0])
        assert _get(sv2, ids2[0], q) == 0
        assert np.array_equal(q, ref)
    finally:
        cu.cuCtxDestroy_v2(other)
    sv.close()
    sv2.close()


def test_threads_read_at_once():
    sv, ids, prm = _solver(8)
    ref = [_fresh(p) for p in prm]
    assert all(_get(sv, i, q) == 0 for i, q in zip(ids, ref))
    assert not np.array_equal(ref[0], ref[1])
    for _ in range(5):
        out = [_fresh(p) for p in prm]
        rc = [None] * len(ids)
        start = threading.Barrier(len(ids))

        def read(k):
            start.wait()
            rc[k] = _get(sv, ids[k], out[k])

        ts = [threading.Thread(target=read, args=(k,)) for k in range(len(ids))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert rc == [0] * len(ids)
        for a, b in zip(out, ref):
            assert np.array_equal(a, b)
    sv.close()
