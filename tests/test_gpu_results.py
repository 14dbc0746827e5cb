"""How results reach Python: whole-batch arrays from a fresh context (results
outgrow the block's guess) and a warm one, of one job and of several, sorted and
not; large results as views while the context's results hold little pinned
memory, as copies beyond that."""
import numpy as np
import pytest

from conftest import gi_pose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("njobs", [1, 2, 5])
@pytest.mark.parametrize("sort_output", [True, False])
def test_batch_flat_fresh_and_warm(gi, njobs, sort_output):
    from gpuintersector import meshgen as mg

    cfgs = [mg.config1(seed=50 + k) for k in range(njobs)]
    with gi.Context(0) as c:
        jobs = [(c.upload(d["vA"], d["tA"]), None, c.upload(d["vB"], d["tB"]), gi_pose(gi, d["poseB"])) for d in cfgs]
        alone = [c.intersect(*j[:1], j[2], j[1], j[3]) for j in jobs]
        want = [r.pairs.copy() for r in alone]
        segs = [np.sort(r.segments.ravel()) for r in alone]
        del alone
        with gi.Context(0) as f:
            fresh = [(f.upload(d["vA"], d["tA"]), None, f.upload(d["vB"], d["tB"]), gi_pose(gi, d["poseB"])) for d in cfgs]
            for ctx, js in ((f, fresh), (f, fresh), (c, jobs)):
                b = ctx.intersect_batch_flat(js, sort_output=sort_output)
                assert b.job.dtype == np.uint32 and b.seg_pair.dtype == np.int64 and b.offsets.dtype == np.int64
                assert np.array_equal(np.diff(b.offsets), [len(w) for w in want])
                assert np.array_equal(np.bincount(b.job, minlength=njobs), [len(w) for w in want])
                for k, w in enumerate(want):
                    got = b.pairs[b.job == k]
                    if not sort_output:
                        got = got[np.lexsort((got[:, 1], got[:, 0]))]
                    assert np.array_equal(got, w)
                    assert np.array_equal(np.sort(b.segments[b.job[b.seg_pair] == k].ravel()), segs[k])
                assert b.stats["pairs"] == len(want[0])
            for A, _, B, _ in fresh:
                A.release()
                B.release()
        for A, _, B, _ in jobs:
            A.release()
            B.release()


def test_large_results_views_and_copies(gi, monkeypatch):
    from gpuintersector import meshgen as mg

    cfg = mg.config3(n=200, seed=8)
    with gi.Context(0) as c:
        A, B = c.upload(cfg["vA"], cfg["tA"]), c.upload(cfg["vB"], cfg["tB"])
        r = c.intersect(A, B)
        pairs, segments = r.pairs, r.segments
        assert pairs.nbytes + segments.nbytes > gi.Result.ZERO_COPY_BYTES and not pairs.flags.owndata
        monkeypatch.setattr(gi.Result, "ZERO_COPY_HELD", 0)
        s = c.intersect(A, B)
        assert s.pairs.flags.owndata and s.stats["pairs"] == len(s.pairs)
        assert np.array_equal(s.pairs, pairs) and np.array_equal(s.segments, segments)
        small = mg.uv_sphere(32, 20, 1.0)
        M = c.upload(*small)
        t = c.intersect(M, M)
        assert not t.pairs.flags.owndata  # small results stay views
        for m in (A, B, M):
            m.release()
    assert np.array_equal(s.pairs, pairs)  # views outlive the context
