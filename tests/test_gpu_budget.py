"""HBM budget on the GPU: a context counts what its resident meshes were admitted
with, no more after failed uploads and no less after releases."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(level=5):
    from gpuintersector import meshgen as mg

    return mg.icosphere(level)


def _bytes(gi, v, t):
    with gi.Context(0, hbm_budget_bytes=1 << 33) as c:
        m = c.upload(v, t)
        n = m.info()["bytes"]
        m.release()
    return n


def _refused(gi, c, v, t):
    with pytest.raises(gi.GIError) as e:
        c.upload(v, t)
    return e.value.status == gi._abi.GI_ERR_OOM


def test_failed_uploads_free_no_budget(gi):
    v, t = _mesh()
    bad = t.copy()
    bad[-1, 2] = len(v)
    with gi.Context(0, hbm_budget_bytes=int(1.9 * _bytes(gi, v, t))) as c:
        A = c.upload(v, t)
        for _ in range(3):
            with pytest.raises(gi.GIError) as e:
                c.upload(v[: len(v) // 2], np.minimum(bad, len(v) // 2))
            assert e.value.status == gi._abi.GI_ERR_INVALID_ARG
        assert _refused(gi, c, v, t)
        A.release()
        c.upload(v, t).release()


@pytest.mark.parametrize("fp64", [False, True])
def test_released_meshes_free_what_they_took(gi, fp64):
    v, t = _mesh()
    with gi.Context(0, hbm_budget_bytes=int(2.5 * _bytes(gi, v, t))) as c:
        A, B = c.upload(v, t), c.upload(v, t)
        if fp64:  # builds the FP64 copies of both
            c.intersect(A, B, precision=1, want_segments=False).pairs
        assert _refused(gi, c, v, t)
        A.release()
        C = c.upload(v, t)
        assert _refused(gi, c, v, t)
        B.release()
        C.release()
        A, B = c.upload(v, t), c.upload(v, t)
        A.release()
        B.release()
