"""The exact stage's results outgrow their buffer inside the one-launch finish: the
first calls of contexts whose buffers start at 64 entries, on coplanar grids (every
result comes from the exact stage) and on touching ones; no wait may run out, and
the rerun gives the oracle's pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(8, 0), (24, 0), (64, 0), (64, 1)])
def test_exact_results_outgrow_their_buffer(gi, oc, n, precision):
    from gpuintersector import meshgen as mg

    d = mg.config3(n=n, seed=n)
    ref = oc.intersect_meshes(d["vA"], d["tA"], oc.pose_identity(), d["vB"], d["tB"], oc.pose_identity())["pairs"]
    assert len(ref) > 64
    for _ in range(4):
        with gi.Context(0, flags=gi._abi.GI_FLAG_TINY_BUFFERS) as c:
            A, B = c.upload(d["vA"], d["tA"]), c.upload(d["vB"], d["tB"])
            r = c.intersect(A, B, precision=precision)
            assert r.stats["retries"] > 0 and r.stats["escalated"] > 64
            assert np.array_equal(r.pairs, ref[np.lexsort((ref[:, 1], ref[:, 0]))])
            for m in (A, B):
                m.release()
