"""Construction codes on the GPU: every kind of point a result's segments can be
made of (vertices, edge-plane crossings, coplanar edge-edge crossings, each edge
in either direction and from either triangle), against the exact CPU oracle."""
import numpy as np
import pytest

from conftest import canonical

pytestmark = pytest.mark.gpu


def _cells(rng, n, hi, flat, collinear):
    """n cells along x, one triangle of integer corners in [0, hi]^3 per cell
    (flat: z = 0; collinear: the third corner on the line of the first two)."""
    t = rng.integers(0, hi + 1, size=(n, 3, 3)).astype(np.float64)
    if flat:
        t[:, :, 2] = 0.0
    if collinear:
        t[:, 2] = t[:, 0] + (t[:, 1] - t[:, 0]) * rng.integers(-1, 3, size=(n, 1))
    t[:, :, 0] += 64.0 * np.arange(n)[:, None]
    return t.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("degenerate", ["none", "a", "b", "both"])
def test_degenerate_pairs_segments(ctx, gi, oc, flat, degenerate):
    rng = np.random.default_rng([7, flat, len(degenerate)])
    vA, tA = _cells(rng, 4000, 4, flat, degenerate in ("a", "both"))
    vB, tB = _cells(rng, 4000, 4, flat, degenerate in ("b", "both"))
    ref = oc.intersect_meshes(vA, tA, oc.pose_identity(), vB, tB, oc.pose_identity(), want_segments=True)
    assert 50 < len(ref["pairs"]) < 4000
    A, B = ctx.upload(vA, tA), ctx.upload(vB, tB)
    for precision in (0, 1):
        r = ctx.intersect(A, B, None, None, precision=precision)
        assert np.array_equal(r.pairs, ref["pairs"])
        gp, gs = canonical(r.segments, r.seg_pair)
        ep, es = canonical(ref["segs"], ref["seg_pair"])
        assert np.array_equal(gp, ep) and np.array_equal(gs, es)
    A.release()
    B.release()
