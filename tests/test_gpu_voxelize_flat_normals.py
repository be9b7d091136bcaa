"""GPU voxelizer on facets whose file normal's z lies around the reference's
threshold (it rejects a plane crossing whose denominator, ray length times that
z, is below 1e-16), against the brute-force oracle: zero, just below, at, just
above, and far above it, on facets that the rays do pass through."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [1.0, 0.5])
@pytest.mark.parametrize("origin_z", [0.0, -3.25])
def test_gpu_voxelize_normals_around_the_threshold(gpu_lib, oracle_lib, spacing, origin_z):
    rng = np.random.default_rng(5)
    n = 240
    c = rng.uniform(2.0, 14.0, (n, 1, 3))
    v = c + rng.normal(0.0, 3.0, (n, 3, 3))
    nrm = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    length = 16.0 + 0.1 - 0.5 * spacing  # of a ray whose ends are not moved
    f = np.array([0.0, -0.0, 1e-3, 0.9, 0.99, 0.999, 1.0, 1.001, 1.01, 1.1, 2.0, 1e3, 1e12, 1e15, 0.98, 1.02])
    nrm[:, 2] = f[np.arange(n) % len(f)] * 1e-16 / length * rng.choice([-1.0, 1.0], n)
    tri = np.concatenate([v.reshape(n, 9), nrm], 1)
    dims = [int(16 / spacing)] * 3
    kw = dict(bbox=[0.0, 16.0, 0.0, 16.0, 0.0, 16.0], origin=(0.17, 0.23, origin_z), dims=dims)
    ref, _, _ = oracle_lib.voxelize(tri, spacing, culled=False, **kw)
    got, desc = gpu_lib.voxelize(tri, spacing, **kw)
    assert ref.any() and not ref.all()
    assert np.array_equal(got, ref) and desc.fluid_count == int(ref.sum())
