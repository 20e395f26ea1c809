"""ot2d_solver_get_q writes the same state into pages that are not there yet
(through pinned chunks of 1 MB: the sizes are less than one chunk, one and a
part, several) and into pages that are, from the first byte of a page or
not."""
import ctypes as C
import mmap

import numpy as np
import pytest

from turns2d_urans_git_gb300 import api
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(33, 13), (257, 129), (385, 257)])
def test_fresh_and_used_buffers(size):
    c = api.config_c1(jmax=size[0], kmax=size[1])
    sv = api.Solver(OT2D_FP32_MIXED)
    i = sv.add(c[1], c[2], c[3], orders=0.0, max_iters=100)
    sv.iterate(2)
    n = c[1].jd * c[1].kd * c[1].nspec * c[1].nq
    used, fresh, odd = np.ones(n), mmap.mmap(-1, 8 * n), mmap.mmap(-1, 8 * n + 8)
    got = [used, np.frombuffer(fresh), np.frombuffer(odd)[1:]]
    for q in got:
        assert api.lib().ot2d_solver_get_q(sv._h, i, q.ctypes.data_as(C.POINTER(C.c_double))) == 0
    sv.close()
    assert np.abs(got[0]).max() > 0 and not np.array_equal(got[0], np.ones(n))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
