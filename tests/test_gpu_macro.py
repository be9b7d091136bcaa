"""rho and u of every node (the FP32-arithmetic formats: error-free FP32 sums of
the offsets) against FP64 sums of the distributions that the same state reads
out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(capi, Q, prec, mode):
    mask = np.zeros((9, 8, 13), np.uint8)
    mask[1:8, 1:7, 1:12] = 1
    mask[4, 3, 5] = mask[1, 1, 1] = 0
    s = capi.Solver(Q, prec, mode, 0.6)
    s.set_geometry(mask, [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", 1, 0.05), capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", 7, 1.003)])
    return s


def _directions(Q):
    """The engine's order, from its momentum lists."""
    c = np.zeros((Q, 3))
    if Q == 19:
        plus = [(0, 6, 7, 8, 9), (2, 6, 10, 14, 15), (4, 8, 12, 14, 16)]
        minus = [(1, 10, 11, 12, 13), (3, 7, 11, 16, 17), (5, 9, 13, 15, 17)]
    else:
        plus = [(1, 7, 8, 11, 13, 19, 21, 23, 25), (3, 7, 9, 15, 16, 19, 21, 24, 26), (5, 11, 12, 15, 17, 19, 22, 23, 26)]
        minus = [(2, 9, 10, 12, 14, 20, 22, 24, 26), (4, 8, 10, 17, 18, 20, 22, 23, 25), (6, 13, 14, 16, 18, 20, 21, 24, 25)]
    for k in range(3):
        c[list(plus[k]), k], c[list(minus[k]), k] = 1, -1
    return c


def _moments(f, Q):
    rho = f.sum(1)
    return rho, (f @ _directions(Q)) / rho[:, None]


@pytest.mark.parametrize("Q,prec,mode", [(Q, p, "physics") for Q in (19, 27) for p in ("f64", "f32", "f16", "bf16")] +
                         [(19, "f64", "parity"), (19, "f32", "parity"), (19, "f16", "parity")])
@pytest.mark.parametrize("steps", [0, 1, 30])
def test_gpu_macro_matches_distributions(gpu_lib, Q, prec, mode, steps):
    """Nineteen or 27 FP64 additions of values below 1 on the reference's side
    (3e-15), 2^-48 of the offsets' sums on the other: 1e-14."""
    s = _solver(gpu_lib, Q, prec, gpu_lib.LBM_PARITY if mode == "parity" else gpu_lib.LBM_PHYSICS)
    s.step(steps)
    rho, u = s.macro()
    r, v = _moments(s.distributions(), Q)
    s.close()
    assert np.abs(rho - r).max() <= 1e-14 and np.abs(u - v).max() <= 1e-14


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("prec", ["f32", "bf16"])
def test_gpu_macro_far_out_values(gpu_lib, Q, prec):
    """Populations near the end of FP32's range, in a state that is read out
    as it was set: relative to the largest."""
    s = _solver(gpu_lib, Q, prec, gpu_lib.LBM_PHYSICS)
    f = s.distributions()
    rng = np.random.default_rng(Q)
    f[::7] = np.exp(rng.uniform(np.log(1e24), np.log(3e36), f[::7].shape))
    f[1::7] = np.exp(rng.uniform(np.log(1e-9), np.log(1e9), f[1::7].shape))
    try:
        s.set_distributions(f)
        rho, u = s.macro()
        back = s.distributions()
    except gpu_lib.LbmError:
        pytest.skip("the state was refused")
    r, v = _moments(back, Q)
    s.close()
    np.testing.assert_allclose(rho, r, rtol=1e-13)
    # u's terms are of the size of rho: relative to 1
    np.testing.assert_allclose(u, v, rtol=0, atol=1e-13)
