"""A server that stops with results nobody fetched gives their pinned memory back."""
import ctypes
import time

import pytest

pytestmark = pytest.mark.gpu


def _held(gi, r):
    v = gi._abi.ResultArrays()
    gi.lib().gi_result_view(r._owner.handle, ctypes.byref(v))
    return v.held_bytes


def test_unfetched_results_are_released(gi):
    from gpuintersector import meshgen as mg

    v, t = mg.icosphere(3)
    with gi.Context(0) as c:
        A, B = c.upload(v, t), c.upload(v * 0.9 + [0.3, 0.0, 0.0], t)
        r = c.intersect(A, B)
        alone = _held(gi, r)
        assert alone > 0
        del r
        srv = gi.Server(c, 4, True, gi.GI_PREC_FP32_CASCADE)
        tickets = [srv.submit(A, None, B, None) for _ in range(6)]
        fetched = srv.wait(tickets[-1])  # the rounds before it are done too
        assert fetched.stats["pairs"] > 0
        time.sleep(0.05)
        srv.stop()
        del fetched
        r = c.intersect(A, B)
        assert _held(gi, r) == alone
        del r
        for m in (A, B):
            m.release()
