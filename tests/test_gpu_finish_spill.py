"""A first call whose keys spill past the finish's small buckets and its overflow list
(few faces of A hold all results): refused once; the next call has large buckets
and ends with the one-launch finish.  Keys that crowd into partitions over its limit
keep the following calls off it.  Known pairs: stacked planes and needles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(planes, needles, far):
    """A: `planes` large triangles at z = 0, 1, .. and `far` ones out of reach;
    B: `needles` thin upright triangles that cross every plane."""
    size = 4.0 * needles
    z = np.arange(planes)[:, None, None] * [[[0.0, 0.0, 1.0]]]
    big = [[[-size, -size, 0.0], [4 * size, -size, 0.0], [-size, 4 * size, 0.0]]] + z
    off = np.arange(far)[:, None, None] * [[[3.0, 0.0, 0.0]]] + [[[0.0, 0.0, 9e4], [1.0, 0.0, 9e4], [0.0, 1.0, 9e4]]]
    vA = np.concatenate([big.reshape(-1, 3), off.reshape(-1, 3)])
    x = np.arange(needles)[:, None, None] * [[[1.0, 0.0, 0.0]]]
    vB = ([[[0.25, 0.5, -10.0], [0.5, 0.75, planes + 10.0], [0.75, 0.25, planes + 10.0]]] + x).reshape(-1, 3)
    return tuple(a for v in (vA, vB) for a in (v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)))


@pytest.mark.parametrize("planes,needles,far,again", [(128, 1000, 3968, True), (64, 3000, 4032, False)])
def test_spilled_and_crowded_first_calls(gi, planes, needles, far, again):
    vA, tA, vB, tB = _scene(planes, needles, far)
    want = np.stack(np.meshgrid(np.arange(planes), np.arange(needles), indexing="ij"), -1).reshape(-1, 2)
    with gi.Context(0) as c:
        A, B = c.upload(vA, tA), c.upload(vB, tB)
        phases = []
        for _ in range(3):
            r = c.intersect(A, B)
            phases.append(r.stats["finish_phases"])
            assert np.array_equal(r.pairs, want)
            assert np.array_equal(r.seg_pair, np.arange(len(want))) and len(r.segments) == len(want)
            assert np.array_equal(r.segments[:, 2], want[:, 0]) and np.array_equal(r.segments[:, 5], want[:, 0])
        assert phases == ([0, 4, 4] if again else [0, 0, 0])
        for m in (A, B):
            m.release()
