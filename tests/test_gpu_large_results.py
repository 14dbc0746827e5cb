"""Ordered results past the one-launch finish and the small-count ordering: all on
one face of A (the finish refuses), counts around the gather's tiles of 1,024,
with one segment each or with none, one and three; a result that outgrows the
call's guess (copied from device memory), the same again (written to the host by
the gather), a smaller one after a larger, alone, in a batch and unordered;
against the exact oracle."""
import numpy as np
import pytest

from conftest import canonical
from test_gpu_finish import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,odd", [(25600, False), (25601, False), (40000, True)])
def test_gather_to_host(gi, oc, k, odd):
    vA, tA, vB, tB = _scene(k, odd)
    ref = oc.intersect_meshes(vA[:3], tA[:1], oc.pose_identity(), vB, tB, oc.pose_identity(), want_segments=True)
    ep, es = canonical(ref["segs"], ref["seg_pair"])
    few = 24600  # a shorter B with the same first triangles

    def same(r, n):
        assert np.array_equal(r.pairs, ref["pairs"][:n])
        m = int((ep < n).sum())
        gp, gs = canonical(r.segments, r.seg_pair)
        assert np.array_equal(gp, ep[:m]) and np.array_equal(gs, es[:m])

    n_all, n_few = len(ref["pairs"]), int((ref["pairs"][:, 1] < few).sum())
    with gi.Context(0) as c:
        A, B, C = c.upload(vA, tA), c.upload(vB, tB), c.upload(vB, tB[:few])
        for mesh, n in ((B, n_all), (B, n_all), (C, n_few), (B, n_all)):
            same(c.intersect(A, mesh), n)
        assert np.array_equal(c.intersect(A, B, want_segments=False).pairs, ref["pairs"])
        for _ in range(2):
            for r, n in zip(c.intersect_batch([(A, None, B, None), (A, None, C, None)]), (n_all, n_few)):
                same(r, n)
        r = c.intersect(A, B, sort_output=False)
        order = np.argsort(r.pairs[:, 1])
        assert np.array_equal(r.pairs[order], ref["pairs"])
        gp, gs = canonical(r.segments, np.argsort(order).astype(np.int32)[r.seg_pair])
        assert np.array_equal(gp, ep) and np.array_equal(gs, es)
        for m in (A, B, C):
            m.release()
