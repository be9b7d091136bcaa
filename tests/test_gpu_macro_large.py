"""rho and u of nodes whose offsets' sums near the end of FP32's range take the
full FP64 populations, beside ordinary nodes, against FP64 sums of the
distributions that the same state reads out."""
import numpy as np
import pytest

from test_gpu_macro import _moments, _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("prec", ["f32", "bf16"])
def test_gpu_macro_beyond_the_error_free_sums(gpu_lib, Q, prec):
    """19 or 27 FP64 additions on the reference's side and on the full f's (1e-13
    relative to the largest); populations up to 1e36, so that f / w stays inside
    BF16's range at the smallest weight 1 / 216."""
    s = _solver(gpu_lib, Q, prec, gpu_lib.LBM_PHYSICS)
    f = s.distributions()
    rng = np.random.default_rng(Q)
    f[::7] = np.exp(rng.uniform(np.log(1e28), np.log(1e36), f[::7].shape))
    f[1::7] = np.exp(rng.uniform(np.log(1e-9), np.log(1e9), f[1::7].shape))
    s.set_distributions(f)
    rho, u = s.macro()
    back = s.distributions()
    s.close()
    assert np.isfinite(back).all() and np.isfinite(rho).all() and np.isfinite(u).all()
    r, v = _moments(back, Q)
    assert (r > 1e31).sum() > len(r) // 10  # the sums' bound is 1e30
    np.testing.assert_allclose(rho, r, rtol=1e-13)
    # u's terms are of the size of rho: relative to 1
    np.testing.assert_allclose(u, v, rtol=0, atol=1e-13)
