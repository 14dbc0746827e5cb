"""Pair lists whose pairs the FP32 filter cannot decide but FP64 can, mixed with
plain, exactly touching and coplanar ones, against the exact oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1000, 40000])
@pytest.mark.parametrize("gap", [1e-9, 1e-6, 0.0])
def test_near_touching_pairs(ctx, gi, oc, n, gap):
    import torch

    rng = np.random.default_rng([n, int(gap * 1e12)])
    tri = rng.uniform(0.0, 1.0, size=(n, 3, 3))
    tri[:, :, 2] = 0.0
    other = rng.uniform(0.0, 1.0, size=(n, 3, 3))
    other[:, 0, 2] = gap * rng.uniform(-1.0, 1.0, size=n)  # one corner within the gap of A's plane
    tri[:, :, 0] += 2.0 * np.arange(n)[:, None]
    other[:, :, 0] += 2.0 * np.arange(n)[:, None]
    t = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    vA, vB = tri.reshape(-1, 3), other.reshape(-1, 3)
    pairs = np.stack([np.arange(n), (np.arange(n) + (np.arange(n) % 5 == 4)) % n], 1).astype(np.int32)
    want = oc.classify_pairs(vA, t, oc.pose_identity(), vB, t, oc.pose_identity(), pairs)
    A, B = ctx.upload(vA, t), ctx.upload(vB, t)
    d_pairs = torch.from_numpy(pairs).cuda()
    for precision in (0, 1):
        for call in (ctx.classify_pairs, ctx.classify_pairs_noalloc):
            d_out = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            call(A, B, None, None, d_pairs.data_ptr(), n, d_out.data_ptr(), precision=precision)
            assert np.array_equal(d_out.cpu().numpy(), want)
    A.release()
    B.release()
