"""Jump flooding, the prior's axis sums and the smoothing filter at grid sizes
around their blocks, against the same steps in NumPy (values equal)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DIMS = [(1, 1, 1), (2, 3, 5), (5, 9, 31), (4, 17, 33), (9, 5, 64), (3, 7, 65), (7, 6, 129), (33, 12, 20), (300, 5, 6)]


def _p(t):
    return C.c_void_p(t.data_ptr())


def _mask(dims):
    m = (np.random.default_rng(sum(dims)).random(dims) < 0.8).astype(np.uint8)
    m[:, dims[1] // 3:, : dims[2] // 2] = 1
    return m


def _flood(mask, planar):
    """Nearest seed by jump flooding: offsets N/2 .. 1 and 1 again, neighbours
    in z, y, x order, the strictly nearer one replacing."""
    D, H, W = mask.shape
    p = np.pad(mask, 1)
    near = [p[1:-1, 1:-1, 2:], p[1:-1, 1:-1, :-2], p[1:-1, 2:, 1:-1], p[1:-1, :-2, 1:-1]]
    if not planar:
        near += [p[2:, 1:-1, 1:-1], p[:-2, 1:-1, 1:-1]]
    seed = (mask > 0) & ~np.logical_and.reduce([n > 0 for n in near])
    at = np.stack(np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij"), -1)
    best = np.where(seed[..., None], at, -1)
    big = max(H, W) if planar else max(D, H, W)
    k = 1
    while k * 2 < big:
        k *= 2
    steps = []
    while k >= 1:
        steps.append(k)
        k //= 2
    far = np.iinfo(np.int64).max
    for k in steps + [1]:
        src = best.copy()
        bd = np.where(src[..., 0] >= 0, ((src - at) ** 2).sum(-1), far)
        for dz in ((0,) if planar else (-1, 0, 1)):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    q = at + np.array([dz, dy, dx]) * k
                    ok = ((q >= 0) & (q < np.array(mask.shape))).all(-1)
                    qc = np.where(ok[..., None], q, 0)
                    s = src[qc[..., 0], qc[..., 1], qc[..., 2]]
                    d = np.where(ok & (s[..., 0] >= 0), ((s - at) ** 2).sum(-1), far)
                    upd = d < bd
                    bd = np.where(upd, d, bd)
                    best = np.where(upd[..., None], s, best)
    dist = np.where(bd < far, np.sqrt(np.where(bd < far, bd, 0).astype(np.float32)), np.float32(0))
    inside = dist + np.float32(0.5)
    return np.where(mask > 0, inside, np.float32(0) if planar else -inside)


@pytest.mark.parametrize("dims", DIMS)
def test_gpu_flooding_and_prior(gpu_lib, dims):
    L = gpu_lib.load()
    mask = _mask(dims)
    n = mask.size
    m = torch.from_numpy(mask.reshape(-1)).cuda()
    d3 = (C.c_int * 3)(*dims)
    f = [torch.empty(n, device="cuda") for _ in range(4)]
    scratch = torch.empty(2 * n + 3 * dims[0], dtype=torch.int32, device="cuda")
    gpu_lib._check(L.lbm_sdf_from_mask(_p(m), d3, _p(f[0]), _p(scratch), None))
    gpu_lib._check(L.lbm_ws_prior(_p(m), d3, 0.03, 0.02, _p(f[1]), _p(f[2]), _p(f[3]), _p(scratch), None))
    sdf, dist, drho, uz = (t.cpu().numpy().reshape(dims) for t in f)
    assert np.array_equal(sdf, _flood(mask, False))
    assert np.array_equal(dist, _flood(mask, True))
    R = dist.reshape(dims[0], -1).max(1).astype(np.float64)
    on = np.flatnonzero(R > 0)
    Q = np.pi * R[on[0]] ** 2 * 0.03 / 2.0 if len(on) else 0.0
    Rs = np.maximum(R, 1.0)
    drop = np.where(R > 0, 24.0 * 0.02 * Q / (np.pi * Rs ** 4), 0.0)
    tail = np.concatenate([np.cumsum(drop[::-1])[::-1][1:], [0.0]])
    # FP64 sums rounded to FP32 once: within one FP32 rounding
    np.testing.assert_allclose(drho[mask > 0], np.broadcast_to(tail[:, None, None], dims)[mask > 0], rtol=2e-7, atol=0)
    e = Rs[:, None, None] - dist
    ref = (2.0 * Q / (np.pi * Rs * Rs))[:, None, None] * np.clip(1.0 - e * e / (Rs * Rs)[:, None, None], 0.0, 1.0)
    # FP32: the profile 1 - e^2 / R^2 is within a few roundings of 1
    np.testing.assert_allclose(uz, np.where(mask > 0, ref, 0.0), rtol=1e-6, atol=1e-6 * max(ref.max(), 1e-30))


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("rounds", [0, 1, 2])
def test_gpu_smoothing(gpu_lib, dims, rounds):
    L = gpu_lib.load()
    mask = _mask(dims)
    v = np.random.default_rng(2).normal(size=dims).astype(np.float32)
    m = torch.from_numpy(mask.reshape(-1)).cuda()
    t = torch.from_numpy(v.reshape(-1).copy()).cuda()
    tmp = torch.empty_like(t)
    gpu_lib._check(L.lbm_ws_smooth(_p(m), (C.c_int * 3)(*dims), _p(t), _p(tmp), rounds, None))
    ref = v
    for _ in range(rounds):
        for axis in (0, 1, 2):
            num, den = np.float32(2) * ref, np.full(dims, 2, np.float32)
            for sh in (-1, 1):  # the upper neighbour first
                src = np.roll(ref, sh, axis)
                ok = np.roll(mask, sh, axis) > 0
                edge = [slice(None)] * 3
                edge[axis] = -1 if sh < 0 else 0
                ok[tuple(edge)] = False
                num = np.where(ok, num + src, num)
                den = den + ok
            ref = np.where(mask > 0, (num / den).astype(np.float32), np.float32(0))
    assert np.array_equal(t.cpu().numpy().reshape(dims), ref)
