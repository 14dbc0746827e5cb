"""The one-launch finish on the GPU at the edges of its partitions and runs:
results that all share one face of A, so that their keys fall into two
partitions, counted around the bucket size (256), the shortest run (16) and the
partition limit (2,048), with one segment each or with none, one and three; the
first call of a context (results kept in device memory and copied) and the next
(written into the result block); alone and in a batch; against the exact oracle."""
import numpy as np
import pytest

from conftest import canonical

pytestmark = pytest.mark.gpu


def _scene(k, odd):
    """A: one large triangle in z = 0 and 2,047 far ones; B: k small triangles on
    it, crossing it, or (odd) in turn crossing, inside it in its plane (three
    segments), touching it with a corner, and far above it (no result)."""
    side = 4.0 * (int(np.ceil(np.sqrt(max(k, 1)))) + 2)
    big = [[-side, -side, 0.0], [4 * side, -side, 0.0], [-side, 4 * side, 0.0]]
    far = np.arange(2047)[:, None, None] * [[[3.0, 0.0, 0.0]]] + [[[5e4, 0, 9e3], [5e4 + 1, 0, 9e3], [5e4, 1, 9e3]]]
    vA = np.concatenate([np.array(big), far.reshape(-1, 3)])
    n = int(np.ceil(np.sqrt(max(k, 1))))
    at = np.stack([4.0 * (np.arange(k) % n), 4.0 * (np.arange(k) // n), np.zeros(k)], 1)[:, None]
    cross = np.array([[0.1, 0.2, -1.0], [1.3, 0.4, 1.0], [0.7, 1.6, 1.0]])
    flat = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]])
    touch = np.array([[0.5, 0.25, 0.0], [1.0, 0.0, 1.0], [0.0, 1.0, 1.0]])
    kinds = [cross, flat, touch, cross + [0.0, 0.0, 9.0]] if odd else [cross]
    vB = (at + np.stack([kinds[j % len(kinds)] for j in range(k)] or [cross])[:k]).reshape(-1, 3)
    if k == 0:
        vB = np.array([[0.0, 0.0, 50.0], [1.0, 0.0, 50.0], [0.0, 1.0, 50.0]])
    return vA, np.arange(len(vA), dtype=np.uint32).reshape(-1, 3), vB, np.arange(len(vB), dtype=np.uint32).reshape(-1, 3)


def _same(r, ref):
    assert np.array_equal(r.pairs, ref["pairs"])
    gp, gs = canonical(r.segments, r.seg_pair)
    ep, es = canonical(ref["segs"], ref["seg_pair"])
    assert np.array_equal(gp, ep) and np.array_equal(gs, es)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("k", [0, 1, 15, 16, 17, 257, 511, 512, 513, 1500, 2049, 4096])
def test_finish_partition_edges(gi, oc, k, odd):
    vA, tA, vB, tB = _scene(k, odd)
    ref = oc.intersect_meshes(vA, tA, oc.pose_identity(), vB, tB, oc.pose_identity(), want_segments=True)
    with gi.Context(0) as c:
        A, B = c.upload(vA, tA), c.upload(vB, tB)
        for _ in range(3):
            r = c.intersect(A, B)
            assert r.stats["launches"] == 2
            _same(r, ref)
        assert np.array_equal(c.intersect(A, B, want_segments=False).pairs, ref["pairs"])
        for _ in range(2):
            for r in c.intersect_batch([(A, None, B, None), (A, None, B, None)]):
                _same(r, ref)
        A.release()
        B.release()


def test_finish_large_and_uneven_batch(gi, oc):
    """Over 65,536 results (the larger buckets, from the second call on), with
    none to three segments each, alone and in a batch with a small job between
    two large ones."""
    from gpuintersector import meshgen as mg

    grid, small = mg.config3(n=128, seed=9), mg.config1(seed=4)
    refs = [oc.intersect_meshes(d["vA"], d["tA"], oc.pose_identity(), d["vB"], d["tB"], oc.pose_identity(),
                                want_segments=True) for d in (grid, small)]
    assert 65536 < len(refs[0]["pairs"]) < 120000
    with gi.Context(0) as c:
        G = (c.upload(grid["vA"], grid["tA"]), c.upload(grid["vB"], grid["tB"]))
        S = (c.upload(small["vA"], small["tA"]), c.upload(small["vB"], small["tB"]))
        for _ in range(3):
            r = c.intersect(*G)
            _same(r, refs[0])
        assert r.stats["launches"] == 2
        for _ in range(2):
            rs = c.intersect_batch([(G[0], None, G[1], None), (S[0], None, S[1], None), (G[0], None, G[1], None)])
            for r, ref in zip(rs, (refs[0], refs[1], refs[0])):
                _same(r, ref)
        for m in G + S:
            m.release()
