"""Pull segments built on the device: their number against the greedy rule in
plain Python, the steps they drive against the oracle, and the tiled kernel's
plan against the flat kernel, on masks that break rows everywhere, nowhere
(one segment over many groups of 32 nodes) and far apart."""
import numpy as np
import pytest

from helpers import classify

pytestmark = pytest.mark.gpu


def _mask(kind):
    rng = np.random.default_rng(11)
    if kind == "voxel":
        m = np.zeros((3, 3, 3), np.uint8)
        m[1, 1, 1] = 1
        return m
    if kind == "box":
        return np.ones((9, 17, 33), np.uint8)
    if kind == "row":
        return np.ones((1, 1, 517), np.uint8)
    if kind == "column":
        m = np.zeros((701, 3, 3), np.uint8)
        m[:, 1, 1] = 1
        return m
    if kind == "comb":
        m = np.ones((7, 12, 41), np.uint8)
        m[:, ::3] = 0
        m[::2, :, 20] = 0
        return m
    if kind == "plates":  # sources that come and go in long stretches
        m = np.ones((24, 30, 40), np.uint8)
        m[5] = 0
        m[6:12, 7, ::2] = 0
        m[13:, 9:11] = 0
        m[18, :, 3:37] = 0
        return m
    p = {"noise": 0.5, "dense": 0.97, "sparse": 0.08}[kind]
    return (rng.random((14, 19, 37)) < p).astype(np.uint8)


def _greedy(mask, c):
    nz, ny, nx = mask.shape
    idx = np.full(mask.shape, -1, np.int64)
    pts = np.argwhere(mask)
    idx[tuple(pts.T)] = np.arange(len(pts))
    pad = np.pad(idx, 1, constant_values=-1)
    src = np.stack([pad[pts[:, 0] + 1 - e[2], pts[:, 1] + 1 - e[1], pts[:, 2] + 1 - e[0]] for e in c], 1)
    d = np.where(src >= 0, src - np.arange(len(pts))[:, None], 0)
    segs, cur, has = 0, None, None
    for a in range(len(pts)):
        v = src[a] >= 0
        if cur is None or np.any(v & has & (cur != d[a])):
            segs += 1
            cur, has = np.zeros(len(c), np.int64), np.zeros(len(c), bool)
        new = v & ~has
        cur[new] = d[a][new]
        has |= v
    return segs


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("kind", ["voxel", "box", "row", "column", "comb", "plates", "noise", "dense", "sparse"])
def test_gpu_segments(gpu_lib, oracle_lib, kind, Q):
    mask = _mask(kind)
    c, w, _ = oracle_lib.lattice(Q)
    s = gpu_lib.Solver(Q, "f64", gpu_lib.LBM_PHYSICS, 0.7)
    s.set_geometry(mask)
    assert s.counts()["segments"] == _greedy(mask, np.asarray(c, int))
    n = int(mask.sum())
    f = np.asarray(w, float)[None] * (1.0 + 1e-3 * np.random.default_rng(5).normal(size=(n, Q)))
    o = oracle_lib.Sim(Q, oracle_lib.PHYSICS, classify(mask, [], Q), (0.0, 0.0, 0.0), 1.0, 0.7, [])
    s.set_distributions(f)
    o.set_f(f)
    s.step(3)
    o.step(3)
    assert np.max(np.abs(s.distributions() - o.f()[0])) <= 1e-14
    # the tiled kernel reads its windows, segments and entries from the plan
    t = [gpu_lib.Solver(Q, "f32", gpu_lib.LBM_PHYSICS, 0.7) for _ in range(2)]
    for k, h in enumerate(t):
        h.set_geometry(mask)
        h.set_variant(5 if k else 0)
        h.set_distributions(f)
        h.step(5)
    assert np.array_equal(t[0].distributions(), t[1].distributions())
