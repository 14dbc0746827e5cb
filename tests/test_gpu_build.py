"""Mesh builds on the GPU at the sizes where their kernels change: the smallest
trees, the edges of the box pyramid (32 and 256 leaves) and of the radix tiles
(1,024 and 3,072 keys), 20 and 21 small tiles, and both sides of the
limit for small tiles and the bounded node array (2^19 triangles); each mesh is
intersected in FP32, FP64 and FP32 form again (the two trees number their nodes
apart) and compared with the exact oracle.  Invalid input at both sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _strip(n, rng):
    """n triangles of a jittered height field, in random order."""
    w = max(2, int(np.ceil(np.sqrt(n / 2.0))))
    i, j = np.meshgrid(np.arange(w + 1), np.arange(w + 1), indexing="ij")
    v = np.stack([i, j, 0.3 * rng.standard_normal(i.shape)], -1).reshape(-1, 3).astype(np.float64) / w
    a, b = np.meshgrid(np.arange(w), np.arange(w), indexing="ij")
    q = (a * (w + 1) + b).ravel()
    t = np.concatenate([np.stack([q, q + w + 1, q + w + 2], 1), np.stack([q, q + w + 2, q + 1], 1)])
    return v, t[rng.permutation(len(t))[:n]].astype(np.uint32)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 31, 32, 33, 255, 256, 257, 511, 513, 1023, 1024, 1025, 3072, 3073, 20000, 20480, 20481, 524288, 524289])
def test_build_sizes(ctx, gi, oc, n):
    rng = np.random.default_rng(n)
    vA, tA = _strip(n, rng)
    assert len(tA) == n
    vB = rng.uniform(-0.1, 1.1, size=(240, 3))
    vB[:, 2] = rng.uniform(-0.2, 0.2, size=240)
    vB[:, :2] = vB[:, :2] * (0.3 if n < 100 else 1.0)
    tB = np.arange(240, dtype=np.uint32).reshape(-1, 3)
    ref = oc.intersect_meshes(vB, tB, oc.pose_identity(), vA, tA, oc.pose_identity(), want_segments=True)
    A, B = ctx.upload(vA, tA), ctx.upload(vB, tB)
    assert A.info()["nodes"] <= max(1, 2 * n // 3 + 1)
    for precision in (0, 1, 0):
        r = ctx.intersect(B, A, precision=precision)
        assert np.array_equal(r.pairs, ref["pairs"])
        assert np.array_equal(np.sort(r.segments.ravel()), np.sort(ref["segs"].ravel()))
    A.release()
    B.release()


@pytest.mark.parametrize("n", [1000, 524289])
def test_invalid_input(ctx, gi, n):
    v, t = _strip(n, np.random.default_rng(5))
    used = ctx.upload(v, t)
    used.release()
    bad = t.copy()
    bad[n // 2, 1] = len(v)
    with pytest.raises(gi.GIError) as e:
        ctx.upload(v, bad)
    assert e.value.status == gi._abi.GI_ERR_INVALID_ARG
    for x in (2.0 ** 101, 2.0 ** -101, np.nan, np.inf):
        far = np.concatenate([v, [[0.0, x, 0.0]]])  # a vertex that no triangle uses
        with pytest.raises(gi.GIError) as e:
            ctx.upload(far, t)
        assert e.value.status == gi._abi.GI_ERR_RANGE
    with pytest.raises(gi.GIError) as e:
        ctx.intersect_oneshot(v, t, v, bad)
    assert e.value.status == gi._abi.GI_ERR_INVALID_ARG
    only = ctx.upload(v, np.zeros((0, 3), np.uint32))  # vertices alone are a mesh without triangles
    assert only.info()["nodes"] == 0
    only.release()
