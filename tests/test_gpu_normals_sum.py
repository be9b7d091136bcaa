"""Wall normals -- the sum over all triangles of normal area / distance^2 --
against an extended-precision sum of the same terms: triangle counts around
the groups of four and the split over blocks, lattice spacings at which the
product of four squared distances is inside and outside the range of the
shared reciprocal, and a centroid close to a node."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangles(n, size, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.2, 1.2, (n, 1, 3)) * np.array(size)
    return np.ascontiguousarray(np.concatenate([(c + rng.normal(0.0, 1.0, (n, 3, 3))).reshape(n, 9), np.zeros((n, 3))], 1))


def _weights(tri):
    """Normal times area, and centroid, as FP64 rounds them in the kernel's order."""
    a, b, c = tri[:, 0:3], tri[:, 3:6], tri[:, 6:9]
    p, q = b - a, c - a
    n = np.stack([p[:, 1] * q[:, 2] - p[:, 2] * q[:, 1], p[:, 2] * q[:, 0] - p[:, 0] * q[:, 2],
                  p[:, 0] * q[:, 1] - p[:, 1] * q[:, 0]], 1)
    norm = np.sqrt(n[:, 0] * n[:, 0] + n[:, 1] * n[:, 1] + n[:, 2] * n[:, 2])
    return n / norm[:, None] * (0.5 * norm)[:, None], (a + b + c) / 3.0


@pytest.mark.parametrize("ntri", [1, 2, 3, 4, 5, 255, 257, 1030])
@pytest.mark.parametrize("spacing", [1e-60, 1e-26, 1.0, 1e26, 1e60])
@pytest.mark.parametrize("near", [0.0, 1e-7])
def test_gpu_normals_sum(gpu_lib, ntri, spacing, near):
    """A term carries about 16 roundings (4 in d^2, 6 in the products, the
    reciprocal's two, the weight's 4) and the sum up to ntri: eps (16 + ntri) of
    the terms' magnitudes, twice for the division by the length and twice again
    for the weights, which NumPy rounds in the same order."""
    mask = np.zeros((7, 8, 9), np.uint8)
    mask[1:6, 1:7, 1:8] = 1
    tri = _triangles(ntri, (9.0, 8.0, 7.0), ntri)
    if near:
        # the first triangle's centroid beside the node (3, 3, 2), which lies next to the wall
        tri[0, :9] += np.tile(np.array([3.0, 3.0, 2.0]) + near - (tri[0, 0:3] + tri[0, 3:6] + tri[0, 6:9]) / 3.0, 3)
    tri[:, :9] *= spacing
    s = gpu_lib.Solver(19, "f64", gpu_lib.LBM_PHYSICS, 0.8, spacing)
    s.set_geometry(mask)
    s.set_normals(tri)
    w = s.wss()
    s.close()
    pt = w["pt"]
    x = np.stack([pt % 9, pt // 9 % 8, pt // 72], 1).astype(np.float64) * spacing
    nw, cen = _weights(tri)
    d = x[:, None, :].astype(np.longdouble) - cen[None].astype(np.longdouble)
    terms = nw[None].astype(np.longdouble) / (d * d).sum(-1)[..., None]
    total, mag = terms.sum(1), np.abs(terms).sum(1)
    length = np.sqrt((total * total).sum(-1))
    ref = (total / length[:, None]).astype(np.float64)
    bound = 4 * 2.0 ** -53 * (16 + ntri) * (mag.max(-1) / length).astype(np.float64) + 1e-15
    assert len(pt) > 20 and np.isfinite(ref).all()
    assert (np.abs(w["normal"] - ref).max(-1) <= bound).all()
