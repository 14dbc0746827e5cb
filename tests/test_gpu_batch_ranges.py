"""The jobs of a batch on the GPU, by the ranges that the results give for them:
offsets of the whole-batch arrays and the per-job results, sorted or not, on the
one-launch finish and on the general path (more than 262,144 results)."""
import numpy as np
import pytest

from conftest import gi_pose

pytestmark = pytest.mark.gpu


def _configs(kind):
    from gpuintersector import meshgen as mg

    if kind == "grids":  # 0.2 M results each
        return [dict(mg.config3(n=n, seed=n), poseB=None) for n in (200, 190)]
    return [mg.config1(seed=80 + k) for k in range(6)]


def _canonical(pairs, segments, seg_pair):
    order = np.lexsort((pairs[:, 1], pairs[:, 0]))
    rows = np.column_stack([pairs[seg_pair], segments])
    return pairs[order], rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("kind", ["spheres", "grids"])
@pytest.mark.parametrize("sort_output", [True, False])
def test_jobs_by_their_ranges(gi, kind, sort_output):
    with gi.Context(0) as c:
        jobs = [(c.upload(d["vA"], d["tA"]), None, c.upload(d["vB"], d["tB"]), gi_pose(gi, d["poseB"]))
                for d in _configs(kind)]
        want, nsegs = [], []
        for A, pa, B, pb in jobs:
            r = c.intersect(A, B, pa, pb)
            want.append(_canonical(r.pairs, r.segments, r.seg_pair))
            nsegs.append(len(r.segments))
            del r
        assert (sum(len(w[0]) for w in want) > 1 << 18) == (kind == "grids")
        for _ in range(2):
            b = c.intersect_batch_flat(jobs, sort_output=sort_output)
            assert b.stats["pairs"] == len(want[0][0]) and b.stats["segments"] == nsegs[0]
            for k, (pairs, rows) in enumerate(want):
                lo, hi = b.offsets[k], b.offsets[k + 1]
                assert np.all(b.job[lo:hi] == k)
                mine = (b.seg_pair >= lo) & (b.seg_pair < hi)
                got = _canonical(b.pairs[lo:hi], b.segments[mine], b.seg_pair[mine] - lo)
                assert np.array_equal(got[0], pairs) and np.array_equal(got[1], rows)
            for r, (pairs, rows) in zip(c.intersect_batch(jobs, sort_output=sort_output), want):
                got = _canonical(r.pairs, r.segments, r.seg_pair)
                assert np.array_equal(got[0], pairs) and np.array_equal(got[1], rows)
        for A, _, B, _ in jobs:
            A.release()
            B.release()
