"""GPU voxelizer's per-column decisions against the brute-force oracle where
a ray meets edges and vertices, at the word edges of the bit field, and with
more undecided pairs than the first pair list holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(lo, hi):
    """A closed box as 12 triangles (tri12 rows)."""
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    rows = []
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        for side, at in ((-1.0, lo[a]), (1.0, hi[a])):
            p = np.zeros((4, 3))
            p[:, a] = at
            p[:, b] = [lo[b], hi[b], hi[b], lo[b]]
            p[:, c] = [lo[c], lo[c], hi[c], hi[c]]
            n = np.zeros(3)
            n[a] = side
            for t in ((0, 1, 2), (0, 2, 3)):
                rows.append(np.concatenate([p[list(t)].reshape(-1), n]))
    return np.array(rows)


def _octahedron(c, r):
    """Eight triangles whose vertices lie on the lattice (rays through vertices and edges)."""
    c = np.asarray(c, float)
    ax = [np.array(v, float) * r for v in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    rows = []
    for x in (0, 1):
        for y in (2, 3):
            for z in (4, 5):
                # z apex first: the reference's bounding box skips third vertices in y and z
                v = np.stack([c + ax[z], c + ax[y], c + ax[x]])
                n = np.cross(v[1] - v[0], v[2] - v[0])
                rows.append(np.concatenate([v.reshape(-1), n / np.linalg.norm(n)]))
    return np.array(rows)


def _same(gpu_lib, oracle_lib, tri, spacing=1.0, **kw):
    ref, _, _ = oracle_lib.voxelize(tri, spacing, culled=False, **kw)
    got, desc = gpu_lib.voxelize(tri, spacing, **kw)
    assert np.array_equal(got, ref)
    assert desc.fluid_count == int(ref.sum())


@pytest.mark.parametrize("nz", [1, 31, 32, 33, 63, 64, 65, 97])
@pytest.mark.parametrize("shift", [0.0, 0.25, 0.5])
def test_gpu_columns_word_edges(gpu_lib, oracle_lib, nz, shift):
    """Boxes wider than one thread's columns; facets on (shift 1/2) and off the ray starts."""
    tri = np.concatenate([_box((0, 0, shift), (11, 9, nz + shift)), _box((2, 3, 0.4 * nz), (9, 7, 0.7 * nz))])
    _same(gpu_lib, oracle_lib, tri)


@pytest.mark.parametrize("spacing", [1.0, 0.5, 0.3])
def test_gpu_columns_through_vertices(gpu_lib, oracle_lib, spacing):
    tri = np.concatenate([_octahedron((8, 8, 8), 8), _octahedron((8, 8, 8), 3)])
    _same(gpu_lib, oracle_lib, tri, spacing)
    # a lattice beyond the bounding box, ray ends on it
    _same(gpu_lib, oracle_lib, tri, spacing, bbox=[0, 16, 0, 16, 0, 16], origin=(-1.0, -2.0, -4.5), dims=(20, 22, 61))


def test_gpu_columns_more_undecided_pairs_than_the_list(gpu_lib, oracle_lib):
    """Facets tilted out of the vertical by rounding alone: every column they may meet is left undecided."""
    rng = np.random.default_rng(3)
    th = rng.uniform(0, 2 * np.pi, 200)
    d = np.stack([np.cos(th), np.sin(th)], 1)
    p = rng.uniform(6, 12, (200, 2))
    v = np.zeros((200, 3, 3))
    v[:, 0, :2], v[:, 1, :2], v[:, 2, :2] = p - 3 * d, p + 3 * d, p + 2 * d
    v[:, 0, 2], v[:, 1, 2], v[:, 2, 2] = 0.1, 1.3, 6.7
    n = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    n[:, 2] = rng.uniform(-0.2, 0.2, 200)  # file normals that reach the point-in-triangle test
    tri = np.concatenate([np.concatenate([v.reshape(200, 9), n], 1), _box((0, 0, 0), (18, 18, 7))])
    _same(gpu_lib, oracle_lib, tri, 0.75)
