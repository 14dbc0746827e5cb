"""Escalated pairs whose coordinates differ in size by more than FP64's exponents
can scale away: large integers beside the tiny heights that a pose matrix makes.
The 32-bit integer form must not take a height for 0 because scaling it underflows;
answers against exact fractions of the posed vertices."""
import numpy as np
import pytest

from fraction_ref import NONE, tri_tri

pytestmark = pytest.mark.gpu

TRI = np.array([[0.0, 0.0, 0.0], [4.0, 0.0, 0.0], [0.0, 4.0, 0.0]])
T = np.array([[0, 1, 2]], dtype=np.uint32)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("size", [2.0**97, 1.0])
@pytest.mark.parametrize("height", [0.0, 1e-300, 2.0**-1021])
def test_tiny_heights_are_not_zero(gi, size, height, precision):
    import torch

    vA, vB = TRI * size, (TRI + [1.0, 1.0, 1.0]) * [size, size, 1.0]
    pose = gi.pose_raw([1, 0, 0, 0, 1, 0, 0, 0, height], [0, 0, 0], [0, 0, 0])
    posed = gi.pose_apply(pose, vB)
    assert np.array_equal(posed, vB * [1.0, 1.0, height])
    want = tri_tri(vA, posed)[0] != NONE
    assert want == (height == 0.0)
    with gi.Context(0) as c:
        A, B = c.upload(vA, T), c.upload(vB, T)
        assert len(c.intersect(A, B, None, pose, precision=precision).pairs) == int(want)
        pairs = torch.zeros((1, 2), dtype=torch.int32, device="cuda")
        out = torch.full((1,), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        c.classify_pairs(A, B, None, pose, pairs.data_ptr(), 1, out.data_ptr(), precision)
        assert out.item() == int(want)
        A.release()
        B.release()
