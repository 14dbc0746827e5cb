"""gi_mesh_info's bytes on the GPU: vertices, indices, leaves and the tree's nodes,
the same with and without a budget; under a budget, which admits by them, the
device memory that many meshes take is no more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(nt):
    rng = np.random.default_rng(nt)
    v = (rng.random((nt, 1, 3)) + 0.01 * rng.random((nt, 3, 3))).reshape(-1, 3)
    return v, np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("nt", [1, 2, 3, 1000, 20481, 1 << 19, (1 << 19) + 1])
def test_bytes_with_and_without_a_budget(gi, nt):
    v, t = _mesh(nt)
    got = []
    for budget in (0, 1 << 34):
        with gi.Context(0, hbm_budget_bytes=budget) as c:
            m = c.upload(v, t)
            got.append(m.info())
            m.release()
    assert got[0]["nodes"] == got[1]["nodes"] <= 2 * (nt // 3) + 2
    for g in got:
        assert g["bytes"] == 24 * len(v) + 16 + 12 * nt + (24 + 16) * nt + 128 * g["nodes"]


def test_budgeted_meshes_take_what_they_count(gi):
    import torch

    v, t = _mesh(1 << 19)
    count = 24
    with gi.Context(0, hbm_budget_bytes=1 << 34) as c:
        c.upload(v, t).release()  # the build's scratch stays in the context's pool
        before = torch.cuda.mem_get_info()[0]
        ms = [c.upload(v, t) for _ in range(count)]
        taken = before - torch.cuda.mem_get_info()[0]
        counted = sum(m.info()["bytes"] for m in ms)
        slack = count * 128 * (2 * ((1 << 19) // 3) + 2 - ms[0].info()["nodes"])  # of the bound's node arrays
        for m in ms:
            m.release()
    # the first mesh reuses the released one's memory; the pool grows in whole chunks
    assert slack > 200 << 20 and taken < counted + (slack >> 1), (taken, counted, slack)
