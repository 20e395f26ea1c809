"""A LU-SGS sweep whose bounded waits run out, over the layouts of its bands:
one CTA, clusters of two to eight with the row between CTAs handed over by
remote stores, clusters with CTAs that hold no band (a small mesh beside a
tall one), plain and preconditioned.  Wherever a wait gives up, the kernel
returns, the request retires with OT2D_ERR_TIMEOUT and a finite state, and
the same solver then runs the same requests to the bits of an undisturbed
run: nothing of the group whose wait failed was used or refilled, and every
copy and remote store had landed before its shared memory was given back.

No fault is involved: the wait limit is lowered, every wait is bounded."""
import numpy as np
import pytest

from turns2d_urans_git_gb300 import api
from turns2d_urans_git_gb300.abi import OT2D_ERR_TIMEOUT, OT2D_FP32_MIXED, OT2D_FP64, OT2D_OPT_POLL_LIMIT

pytestmark = pytest.mark.gpu
STEPS = 6


def _cases(size, pre):
    out = [api.config_c2(jmax=j, kmax=k, fsmach=0.2, alfa=1.0, rey=2e6, ds_wall=1e-3) for j, k in (size, (33, 13))]
    for c in out:
        if pre:
            c[1].iprecon, c[1].Mp = 1, 0.3
    return out


def _run(sv, cases):
    ids = [sv.add(c[1], c[2], c[3], orders=0.0, max_iters=STEPS) for c in cases]
    sv.iterate(STEPS)
    sv.sync()
    return [(sv.get_q(i, c[1]), sv.result(i)) for i, c in zip(ids, cases)]


# interior rows 68 (FP64: 9 bands of 8, three CTAs; f32: five of 16, two),
# 256 (32 and 16 bands: eight and four CTAs), 193 (25 and 13 bands: seven and
# four CTAs, the last one short)
@pytest.mark.parametrize("precision", [OT2D_FP64, OT2D_FP32_MIXED])
@pytest.mark.parametrize("size", [(97, 69), (65, 257), (129, 194)])
@pytest.mark.parametrize("pre", [False, True])
def test_give_up_leaves_the_solver_usable(precision, size, pre):
    cases = _cases(size, pre)
    sv = api.Solver(precision, check_every=1, keep_q=True)
    good = _run(sv, cases)
    assert all(r.status == 0 and r.iterations == STEPS for _, r in good)
    # one poll ends the first waits, more polls later ones: the give-up comes
    # at different groups of the sweep
    for limit in (1, 2, 5, 20, 100):
        sv.set_option(OT2D_OPT_POLL_LIMIT, limit)
        for (q, r), (q0, _) in zip(_run(sv, cases), good):
            assert r.status in (0, OT2D_ERR_TIMEOUT), (limit, r.status)
            assert np.all(np.isfinite(q))
            assert r.status or np.array_equal(q, q0), limit
            assert limit > 1 or q.shape != good[0][0].shape or r.status == OT2D_ERR_TIMEOUT
    sv.set_option(OT2D_OPT_POLL_LIMIT, 1 << 22)
    for (q, r), (q0, r0) in zip(_run(sv, cases), good):
        assert r.status == 0 and np.array_equal(q, q0) and r.cl == r0.cl
    sv.close()
