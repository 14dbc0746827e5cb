"""The traversal's hand-over pool when it is too small: contexts that start with one
slot.  Every call gives the oracle's pairs; a pool that ran short is larger for the
next call, until the blocks share their node pairs again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.random((n, 1, 3)) + 0.04 * rng.standard_normal((n, 3, 3))
    return v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["nested", "soup"])
@pytest.mark.parametrize("jobs", [1, 2])
def test_pool_grows_after_a_call_that_ran_short(gi, kind, jobs):
    from gpuintersector import meshgen as mg

    if kind == "nested":
        v, t = mg.icosphere(6)
        scene = (v, t, v * 1.0005 + 1e-3, t)
    else:
        scene = _soup(12000, 1) + _soup(12000, 2)
    with gi.Context(0) as c:
        A, B = c.upload(*scene[:2]), c.upload(*scene[2:])
        r = c.intersect(A, B, want_segments=False)
        want, usual = r.pairs.copy(), r.stats["pool_slots"]
        assert len(want) > 0 and usual > 100
        del r
        for m in (A, B):
            m.release()
    slots = []
    with gi.Context(0, flags=gi._abi.GI_FLAG_TINY_BUFFERS) as c:
        A, B = c.upload(*scene[:2]), c.upload(*scene[2:])
        for _ in range(12):
            b = c.intersect_batch_flat([(A, None, B, None)] * jobs, want_segments=False)
            slots.append(b.stats["pool_slots"])
            for j in range(jobs):
                assert np.array_equal(b.pairs[b.offsets[j]:b.offsets[j + 1]], want)
            if slots[-1] > usual // 4:
                break
        for m in (A, B):
            m.release()
    assert slots[-1] > usual // 4, slots
