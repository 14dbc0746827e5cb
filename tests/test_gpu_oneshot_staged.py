"""One-shot calls whose vertex arrays are copied through the staging buffers although
the meshes have few triangles (vertices that no triangle uses): the results of
resident meshes, and each mesh's own error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big", ["a", "b", "ab"])
def test_many_vertices_few_triangles(gi, big):
    from gpuintersector import meshgen as mg

    u, t = mg.icosphere(4)
    extra = np.full((400_000, 3), 7.0)  # 9.6 MB
    vA = np.concatenate([u, extra]) if "a" in big else u
    vB = np.concatenate([u * 0.9 + [0.3, 0.1, 0.0], extra]) if "b" in big else u * 0.9 + [0.3, 0.1, 0.0]
    with gi.Context(0) as c:
        A, B = c.upload(vA, t), c.upload(vB, t)
        want = c.intersect(A, B)
        pairs, segments = want.pairs.copy(), want.segments.copy()
        for m in (A, B):
            m.release()
        assert len(pairs) > 0
        for _ in range(3):
            r = c.intersect_oneshot(vA, t, vB, t)
            assert np.array_equal(r.pairs, pairs) and np.array_equal(r.segments, segments)
        bad, far = t.copy(), vA.copy()
        bad[5, 1] = len(vA) + len(vB)
        far[3] = 1e200
        for args, status in (((vA, bad, vB, t), gi._abi.GI_ERR_INVALID_ARG), ((vA, t, vB, bad), gi._abi.GI_ERR_INVALID_ARG),
                             ((far, t, vB, t), gi._abi.GI_ERR_RANGE), ((far, t, vB, bad), gi._abi.GI_ERR_RANGE)):
            with pytest.raises(gi.GIError) as e:
                c.intersect_oneshot(*args)
            assert e.value.status == status
        assert np.array_equal(c.intersect_oneshot(vA, t, vB, t).pairs, pairs)
