"""The workloads that the intersector's speed is judged by, through its public entry points.

listed() names them, draw(rng) gives another one of the same ranges, prepare(case, seed) makes what a
program holds before the call (resident meshes, poses, host or device arrays), run(state) is one pass,
work(case) the bytes and operations that a pass cannot do without, and exact(case, seed) the segments'
endpoints in plain FP64 arithmetic on the intersecting pairs of a brute-force grid search.

Meshes are the ones of the package's generators: UV spheres, displaced geodesic spheres, coplanar integer
grids.  A case's kind:

  pose      both meshes resident, a new rigid pose, one intersect: the step of a pose-update loop
  batch     many resident pairs in one call: a serving round or an assembly check
  oneshot   host arrays in, pairs and segments out: upload, both builds, intersect, release
  rebuild   device arrays in (a simulation's deformed meshes): both builds and an intersect, every step
  classify  the exact test over an explicit candidate list that lives on the device
"""
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-cubql-intersector-standalone_b200"))
import gpuintersector as gi  # noqa: E402
from gpuintersector import meshgen as mg  # noqa: E402

FP32, FP64 = gi.GI_PREC_FP32_CASCADE, gi.GI_PREC_FP64


def listed():
    return [
        # the smallest call in earnest: two hand-sized UV spheres, one pose (launches and latency only)
        dict(name="pose-uv1k", kind="pose", mesh="uv", p=32, q=20, posed="b", segments=True, precision=FP32),
        # a tool against a part at interactive rates: two UV spheres of 20,224 triangles
        dict(name="pose-uv20k", kind="pose", mesh="uv", p=128, q=80, posed="b", segments=True, precision=FP32),
        # collision check of two scanned parts, both moving, pairs only (what the controller's pipeline returns)
        dict(name="pose-200k-pairs", kind="pose", mesh="sphere", p=100, q=100, posed="ab", segments=False,
             precision=FP32),
        # the headline: pose updates of two meshes of 1.3 M triangles with intersection segments
        dict(name="pose-1m3", kind="pose", mesh="sphere", p=256, q=256, posed="b", segments=True, precision=FP32),
        # the same without the FP32 filter (the plain FP64 form that the cascade is compared with)
        dict(name="pose-1m3-fp64", kind="pose", mesh="sphere", p=256, q=256, posed="b", segments=True,
             precision=FP64),
        # coplanar degeneracies at scale (CAD faces on a common plane): the exact stage decides over a million pairs
        dict(name="pose-grid512", kind="pose", mesh="grid", p=512, q=512, posed="", segments=True, precision=FP32),
        # a serving round: 48 resident pairs of 10 k to 100 k triangles, one pose update each
        dict(name="batch-48", kind="batch", jobs=48, tmin=10000, tmax=100000, segments=True),
        # an assembly check: 256 uneven pairs of 1 k to 200 k triangles in one call
        dict(name="batch-256", kind="batch", jobs=256, tmin=1000, tmax=200000, segments=True),
        # one-shot from ordinary host arrays, interactive size
        dict(name="oneshot-uv20k", kind="oneshot", mesh="uv", p=128, q=80, pinned=False),
        # one-shot from pinned host arrays at the headline size
        dict(name="oneshot-1m3", kind="oneshot", mesh="sphere", p=256, q=256, pinned=True),
        # deforming meshes that live on the device, uneven sizes: build both and intersect every step
        dict(name="rebuild-300k", kind="rebuild", mesh="sphere", p=123, q=91),
        # a broad phase of the caller's own: about a million candidate pairs tested exactly
        dict(name="classify-1m", kind="classify", mesh="sphere", p=256, q=256, spread=96, precision=FP32),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["pose", "pose", "pose", "pose", "batch", "oneshot", "rebuild", "classify"])
    if kind == "batch":
        tmin = _log(rng, 1000, 20000)
        return dict(kind=kind, jobs=_log(rng, 2, 200), tmin=tmin, tmax=_log(rng, 2 * tmin, 200000),
                    segments=rng.random() < 0.7)
    mesh = rng.choice(["uv", "sphere", "sphere"])
    if kind == "pose" and rng.random() < 0.2:
        n = _log(rng, 31, 500)
        return dict(kind=kind, mesh="grid", p=n, q=n, posed="", segments=rng.random() < 0.7,
                    precision=rng.choice([FP32, FP64]))
    if mesh == "uv":
        p, q = _log(rng, 17, 150), _log(rng, 11, 100)
    else:
        p, q = _log(rng, 8, 250), _log(rng, 8, 250)
    if kind == "oneshot":
        return dict(kind=kind, mesh=mesh, p=p, q=q, pinned=rng.random() < 0.5)
    if kind == "rebuild":
        return dict(kind=kind, mesh=mesh, p=p, q=q)
    if kind == "classify":
        return dict(kind=kind, mesh=mesh, p=p, q=q, spread=rng.randrange(3, 96), precision=rng.choice([FP32, FP64]))
    return dict(kind=kind, mesh=mesh, p=p, q=q, posed=rng.choice(["b", "ab"]), segments=rng.random() < 0.7,
                precision=rng.choice([FP32, FP32, FP32, FP64]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=64)
def _sphere(n):
    return mg.geodesic_cached(n)


def _displaced(n, rng):
    u, t = _sphere(n)
    return mg.displace(u, mg.displacement_params(rng)), t


def _place(rng, reach):
    """Where B lies in A's frame, (R, T): a uniform rotation and an offset of the given length in a random direction."""
    d = rng.standard_normal(3)
    return mg.random_rotation(rng), reach * d / np.linalg.norm(d)


def _renumbered(v, t, rng):
    """The same mesh with its vertices and triangles numbered from other ones."""
    k = int(rng.integers(v.shape[0]))
    t = np.where(t + np.uint32(k) >= v.shape[0], t + np.uint32(k) - np.uint32(v.shape[0]), t + np.uint32(k))
    return np.roll(v, k, axis=0), np.roll(t.astype(np.uint32), int(rng.integers(t.shape[0])), axis=0)


# The shapes and how they lie to each other follow from the case's sizes; the seed moves the whole scene rigidly and
# renumbers vertices and triangles.  So inputs and outputs of two seeds differ in every number, not in their counts.
def _scene(base, vA, tA, vB, tB, posed, reach, seed):
    """vA, tA, pose of A (or None), vB, tB, pose of B: B at `reach` from A, the scene moved by the seed."""
    R, T = _place(base, reach)
    rng = np.random.default_rng(seed)
    Q, s = mg.random_rotation(rng), rng.uniform(-1.0, 1.0, 3)
    vA, tA = _renumbered(vA, tA, rng)
    vB, tB = _renumbered(vB, tB, rng)
    zero = np.zeros(3)
    if "a" in posed:
        pA = (Q, zero, s)
    else:
        vA, pA = vA @ Q.T + s, None
    return vA, tA, pA, vB, tB, (Q @ R, zero, Q @ T + s)


def _meshes(case, seed):
    """vA, tA, pose of A (or None), vB, tB, pose of B (or None)."""
    p, q = case["p"], case["q"]
    if case["mesh"] == "grid":
        c = mg.config3(seed=[p, q], n=p)
        rng = np.random.default_rng([seed, 3])
        s = rng.integers(-(1 << 18), 1 << 18, 3).astype(np.float64)
        vA, tA = _renumbered(c["vA"] + s, c["tA"], rng)
        vB, tB = _renumbered(c["vB"] + s, c["tB"], rng)
        return vA, tA, None, vB, tB, None
    base = np.random.default_rng([p, q])
    if case["mesh"] == "uv":
        vA, tA = mg.uv_sphere(p, q, 1.0)
        vB, tB = vA, tA
    else:
        vA, tA = _displaced(p, base)
        vB, tB = _displaced(q, base)
    return _scene(base, vA, tA, vB, tB, case.get("posed", "b"), base.uniform(0.25, 0.6), [seed, 11])


def _batch_freqs(case):
    """Geodesic frequencies of the two meshes of every job, T log-uniform in [tmin, tmax]."""
    rng = np.random.default_rng([case["jobs"], case["tmin"], case["tmax"]])
    t = np.exp(rng.uniform(np.log(case["tmin"]), np.log(case["tmax"]), (case["jobs"], 2)))
    grid = mg._freq_grid(case["tmin"], case["tmax"])
    return grid[np.abs(np.log(20.0 * grid.astype(float) ** 2)[None, None] - np.log(t)[..., None]).argmin(-1)]


def _batch_jobs(case, seed):
    for j, (nA, nB) in enumerate(_batch_freqs(case)):
        base = np.random.default_rng([case["tmin"], j])
        vA, tA = _displaced(int(nA), base)
        vB, tB = _displaced(int(nB), base)
        yield _scene(base, vA, tA, vB, tB, "b", base.uniform(0.2, 1.5), [seed, 4, j])


def _gi_pose(p):
    return None if p is None else gi.pose_raw(*p)


_context = []


def _ctx():
    """The program's one context."""
    if not _context:
        _context.append(gi.Context(0))
    return _context[0]


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    if kind == "batch":
        jobs = []
        for vA, tA, pA, vB, tB, pB in _batch_jobs(case, seed):
            jobs.append((ctx.upload(vA, tA), _gi_pose(pA), ctx.upload(vB, tB), _gi_pose(pB)))
        return dict(ctx=ctx, kind=kind, jobs=jobs, segments=case["segments"])
    vA, tA, pA, vB, tB, pB = _meshes(case, seed)
    s = dict(ctx=ctx, kind=kind, pA=_gi_pose(pA), pB=_gi_pose(pB))
    if kind == "oneshot":
        arrays = [np.ascontiguousarray(x) for x in (vA, tA, vB, tB)]
        if case["pinned"]:
            arrays = [torch.from_numpy(x).pin_memory().numpy() for x in arrays]
        return dict(s, arrays=arrays)
    if kind == "rebuild":
        return dict(s, arrays=[torch.from_numpy(x).cuda() for x in (vA, tA.view(np.int32), vB, tB.view(np.int32))])
    s.update(A=ctx.upload(vA, tA), B=ctx.upload(vB, tB), precision=case["precision"])
    if kind == "classify":
        # every intersecting pair with `spread` neighbours of its B triangle in index order
        hits = ctx.intersect(s["A"], s["B"], s["pA"], s["pB"], want_segments=False).pairs
        d = np.arange(case["spread"]) - case["spread"] // 2
        b = (hits[:, 1][:, None] + d[None]) % tB.shape[0]
        pairs = np.stack([np.repeat(hits[:, 0], d.size), b.ravel()], 1).astype(np.int32)
        pairs = np.random.default_rng([seed, 5]).permutation(pairs.reshape(-1, d.size, 2)).reshape(-1, 2)
        s.update(pairs=torch.from_numpy(np.ascontiguousarray(pairs)).cuda(),
                 out=torch.empty(pairs.shape[0], dtype=torch.uint8, device="cuda"))
        return s
    return dict(s, segments=case["segments"])


# ------------------------------------------------------------------ one pass
def _arrays(r, segments=True):
    if not segments:
        return {"pairs": r.pairs}
    return {"pairs": r.pairs, "segments": r.segments, "seg_pair": r.seg_pair}


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "pose":
        r = ctx.intersect(s["A"], s["B"], s["pA"], s["pB"], want_segments=s["segments"], precision=s["precision"])
        return _arrays(r, s["segments"])
    if kind == "batch":
        r = ctx.intersect_batch_flat(s["jobs"], want_segments=s["segments"])
        return dict(_arrays(r, s["segments"]), job=r.job, offsets=r.offsets)
    if kind == "oneshot":
        return _arrays(ctx.intersect_oneshot(*s["arrays"], s["pA"], s["pB"]))
    if kind == "rebuild":
        vA, tA, vB, tB = s["arrays"]
        ctx.wait_stream(torch.cuda.current_stream().cuda_stream)
        A = ctx.upload_device(vA.data_ptr(), vA.shape[0], tA.data_ptr(), tA.shape[0])
        B = ctx.upload_device(vB.data_ptr(), vB.shape[0], tB.data_ptr(), tB.shape[0])
        r = ctx.intersect(A, B, s["pA"], s["pB"])
        A.release()
        B.release()
        return _arrays(r)
    ctx.classify_pairs(s["A"], s["B"], s["pA"], s["pB"], s["pairs"].data_ptr(), s["pairs"].shape[0],
                       s["out"].data_ptr(), precision=s["precision"])
    return s["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def _tris(mesh, p, q):
    """Triangles of the two meshes."""
    if mesh == "sphere":
        return 20 * p * p, 20 * q * q
    t = 2 * p * (q - 1) if mesh == "uv" else 2 * p * q
    return t, t


def _crossings(ta, tb):
    """Intersecting pairs of two sphere-like meshes: a new one wherever the curve enters a triangle of either."""
    return 5.0 * (ta ** 0.5 + tb ** 0.5)


def _pair_work(pairs, segments):
    """Both triangles' indices and FP64 vertices in, the pair (and a segment with its pair index) out; two planes,
    twelve sides and four line-order determinants a pair, two crossing points a segment."""
    return dict(bytes=pairs * (2 * 84 + 8 + (52 if segments else 0)), flops=pairs * (260 + (160 if segments else 0)))


def _mesh_bytes(t):
    return 12 * t + 24 * (t // 2 + 2)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_pair_work(_crossings(20 * a * a, 20 * b * b), case["segments"]) for a, b in _batch_freqs(case).tolist()]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    ta, tb = _tris(case["mesh"], case["p"], case["q"])
    if case["mesh"] == "grid":
        pairs = 2.55 * ta
        out = pairs * (8 + (52 if case["segments"] else 0))
        return dict(bytes=_mesh_bytes(ta) + _mesh_bytes(tb) + out, flops=pairs * 260)
    pairs = _crossings(ta, tb)
    if kind == "classify":
        n = pairs * case["spread"]
        return dict(bytes=n * 9 + 84 * (min(n, ta) + min(n, tb)), flops=n * 120)
    w = _pair_work(pairs, case.get("segments", True))
    if kind in ("oneshot", "rebuild"):
        w["bytes"] += _mesh_bytes(ta) + _mesh_bytes(tb)
    return w


# ------------------------------------------------------------------ the same in plain FP64 arithmetic
def _posed(v, t, p):
    """Triangle corners (T, 3, 3) in the world frame: ((R (v - C)) + C) + T, every operation rounded by itself."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    if p is not None:
        R, C, T = (torch.from_numpy(np.asarray(x, dtype=np.float64)).to(dev) for x in p)
        x = v - C
        rows = [(R[i, 0] * x[:, 0] + R[i, 1] * x[:, 1]) + R[i, 2] * x[:, 2] for i in range(3)]
        v = (torch.stack(rows, 1) + C) + T
    return v[torch.from_numpy(t.astype(np.int64)).to(dev)]


def _box_pairs(P, Q):
    """Pairs (i, j) whose axis-aligned boxes meet: Q's boxes sorted by the cell of their low corner, P's boxes
    looked up in the cells that such a corner can lie in (cells as wide as the widest box)."""
    plo, phi, qlo, qhi = P.amin(1), P.amax(1), Q.amin(1), Q.amax(1)
    h = float(torch.maximum((phi - plo).max(), (qhi - qlo).max())) * 1.0001
    org = torch.minimum(plo.amin(0), qlo.amin(0)) - 2 * h
    cell = lambda x: ((x - org) / h).floor().long()
    key = lambda c: (c[:, 0] << 40) + (c[:, 1] << 20) + c[:, 2]
    qkey, order = key(cell(qlo)).sort()
    first, last = cell(plo - h), cell(phi)
    found = []
    for dx in range(4):
        for dy in range(4):
            for dz in range(4):
                c = first + torch.tensor([dx, dy, dz], device=P.device)
                use = (c <= last).all(1).nonzero()[:, 0]
                if not len(use):
                    continue
                k = key(c[use])
                lo, hi = torch.searchsorted(qkey, k), torch.searchsorted(qkey, k, right=True)
                n = hi - lo
                i = torch.repeat_interleave(use, n)
                at = torch.arange(len(i), device=P.device) - torch.repeat_interleave(n.cumsum(0) - n, n)
                j = order[torch.repeat_interleave(lo, n) + at]
                hit = ((plo[i] <= qhi[j]) & (qlo[j] <= phi[i])).all(1)
                found.append(torch.stack([i[hit], j[hit]], 1))
    return torch.cat(found)


def _exact_segments(vA, tA, pA, vB, tB, pB):
    """Segments (m, 6) of the intersecting pairs in order of (a, b): for triangles in general position, the crossings
    of A's edges through B's plane that lie inside B's interval, then B's edges' inside A's."""
    P, Q = _posed(vA, tA, pA), _posed(vB, tB, pB)
    ij = _box_pairs(P, Q)
    P, Q = P[ij[:, 0]], Q[ij[:, 1]]
    normal = lambda X: torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0])
    nP, nQ = normal(P), normal(Q)
    sP = ((P - Q[:, :1]) * nQ[:, None]).sum(-1)
    sQ = ((Q - P[:, :1]) * nP[:, None]).sum(-1)
    split = lambda s: (s.amin(1) < 0) & (s.amax(1) > 0)
    keep = split(sP) & split(sQ)
    ij, P, Q, nP, nQ, sP, sQ = (x[keep] for x in (ij, P, Q, nP, nQ, sP, sQ))

    def crossings(X, s):
        neg = s < 0
        lone = torch.where(neg[:, 1] == neg[:, 2], 0, torch.where(neg[:, 0] == neg[:, 2], 1, 2))
        ends = torch.tensor([[1, 2], [0, 2], [0, 1]], device=X.device)[lone]
        r = torch.arange(len(X), device=X.device)
        L, sl = X[r, lone][:, None], s[r, lone][:, None]
        E, se = X[r[:, None], ends], s[r[:, None], ends]
        return L + (sl / (sl - se))[..., None] * (E - L)

    X, Y = crossings(P, sP), crossings(Q, sQ)
    line = torch.linalg.cross(nP, nQ)
    tx, ty = (X * line[:, None]).sum(-1), (Y * line[:, None]).sum(-1)
    inside = lambda t, u: (t > u.amin(1, keepdim=True)) & (t < u.amax(1, keepdim=True))
    pts = torch.cat([X, Y], 1)
    mark = torch.cat([inside(tx, ty), inside(ty, tx)], 1)
    hit = mark.sum(1) == 2
    ij, pts, mark = ij[hit], pts[hit], mark[hit]
    order = (ij[:, 0] * tB.shape[0] + ij[:, 1]).argsort()
    return pts[mark].reshape(-1, 6)[order].cpu().numpy()


def exact(case, seed):
    # pairs, indices and flags are whole numbers; coplanar overlaps have no general-position form
    if case["kind"] == "classify" or case.get("mesh") == "grid" or not case.get("segments", True):
        return None
    if case["kind"] == "batch":
        seg = np.concatenate([_exact_segments(*j) for j in _batch_jobs(case, seed)])
        return {"pairs": None, "segments": seg, "seg_pair": None, "job": None, "offsets": None}
    return {"pairs": None, "segments": _exact_segments(*_meshes(case, seed)), "seg_pair": None}
