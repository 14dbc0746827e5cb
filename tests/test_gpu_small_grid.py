"""Touching and coplanar pairs on binary grids around the limits of the exact
stage's 32-bit form (differences below 2^14 grid units; coordinates below 2^50):
spans on both sides, grids of fractions and of large units, far from the origin,
with negative zeros; against the exact oracle.  Corners are drawn from few values
per axis, so most pairs share planes, lines or corners."""
import numpy as np
import pytest

from conftest import canonical

pytestmark = pytest.mark.gpu


def _pairs(rng, n, values, flat, unit, offset):
    t = rng.choice(values, size=(2, n, 3, 3)).astype(np.float64)
    if flat:
        t[..., 2] = values[0]
    else:
        t[:, ::3, :, 2] = values[0]  # a third of the cells lies in one plane
    t = t * unit + offset
    t[t == 0.0] *= -1.0
    return t


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("span", [3, (1 << 13) - 1, 1 << 13, (1 << 14) - 1, 1 << 14, (1 << 14) + 1, 1 << 20])
@pytest.mark.parametrize("unit,offset", [(1.0, 0.0), (2.0 ** -40, 0.0), (2.0 ** 30, 0.0), (1.0, 2.0 ** 36), (1.0, 2.0 ** 50),
                                         (0.1, 0.0)])
def test_small_grid_pairs(ctx, gi, oc, flat, span, unit, offset):
    rng = np.random.default_rng([span, flat, int(abs(np.log2(unit))), int(offset > 0)])
    n = 600
    values = np.array([0, span, span // 2, 1])
    tri = _pairs(rng, n, values, flat, unit, offset)
    t = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    # one list of n pairs: the k-th triangles of both (far too many others overlap)
    vA, vB = tri[0].reshape(-1, 3), tri[1].reshape(-1, 3)
    step = 4.0 * (span + 1) * unit  # cells apart along y
    shift = (np.repeat(np.arange(n), 3) * step)[:, None] * [[0.0, 1.0, 0.0]]
    vA, vB = vA + shift, vB + shift
    ref = oc.intersect_meshes(vA, t, oc.pose_identity(), vB, t, oc.pose_identity(), want_segments=True)
    A, B = ctx.upload(vA, t), ctx.upload(vB, t)
    r = ctx.intersect(A, B)
    assert np.array_equal(r.pairs, ref["pairs"])
    gp, gs = canonical(r.segments, r.seg_pair)
    ep, es = canonical(ref["segs"], ref["seg_pair"])
    assert np.array_equal(gp, ep) and np.array_equal(gs, es)
    A.release()
    B.release()
