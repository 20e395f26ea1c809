"""Threads that call drop-in routines and end give back the device memory
their calls kept (scratch, staging space, slice tables): the free memory after
eight of them, one after another and at once, is what it was before.  16 MB of
slack is less than one thread's scratch (over 20 MB at this size).  (A thread's
destructors run after Python's join has returned, so the memory is read until
it is back, for ten seconds at most; the CUDA driver takes 28 MB of its own,
once, when a process's second thread calls.)"""
import threading
import time

import numpy as np
import pytest
import torch

from tests.helpers import Case
from turns2d_urans_git_gb300 import routines as rt

pytestmark = pytest.mark.gpu
SLACK = 16 << 20


def test_a_thread_returns_what_it_kept():
    c = Case(jmax=385, kmax=97, seed=3, ds_wall=1e-3)
    out = []

    def call():
        s = np.zeros(c.n2 * c.p.nv)
        rt.set_params(c.p)
        for _ in range(2):
            rt.rhsup(c.q, s, c.xx, c.xy, c.yx, c.yy, c.x, c.y, c.xv, c.yv, c.xv, c.yv, c.xv, c.yv, c.iblank, c.ugv, c.vgv,
                     c.jd, c.kd, 1, 1, c.bt)
        out.append(s)

    def threads(n):
        ts = [threading.Thread(target=call) for _ in range(n)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()

    threads(1)
    threads(1)
    time.sleep(2)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(4):
        threads(1)
    threads(4)
    end = time.time() + 10
    while torch.cuda.mem_get_info()[0] < free - SLACK and time.time() < end:
        time.sleep(0.1)
    assert torch.cuda.mem_get_info()[0] >= free - SLACK
    assert len(out) == 10 and np.abs(out[0]).max() > 0
    assert all(np.array_equal(s, out[0]) for s in out)
