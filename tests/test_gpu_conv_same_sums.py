"""Layers whose order of summation is the mma.sync kernel's, whichever engine runs
them: the stride-2 input gradient and the grids of a network's lowest levels.  A
network's values depend on that order through BF16 rounding."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


def _data(ci, co, dims, ks, stride):
    g = torch.Generator(device="cuda").manual_seed(ci + 3 * co + sum(dims) + ks + stride)

    def bf(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)

    od = [(d - 1) // stride + 1 for d in dims]
    return bf(*dims, ci), bf(co, ks ** 3, ci, scale=0.2), torch.randn(co, generator=g, device="cuda") * 0.1, bf(*od, co), od


def _run(L, gpu_lib, x, w, b, dy, dims, ci, co, ks, stride, relu):
    n = dy.shape[0] * dy.shape[1] * dy.shape[2]
    y = torch.full((n * co + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    y32 = torch.full((n * co + 64,), 3.0, device="cuda")
    dx = torch.full((x.numel() + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty_like(w)
    dims_c = (C.c_int * 3)(*dims)
    gpu_lib._check(L.lbm_nn_conv3d_fwd(_p(x), dims_c, ci, _p(w), _p(b), co, ks, stride, relu, _p(y), _p(y32), None))
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), dims_c, ci, _p(w), _p(scratch), co, ks, stride, _p(dy), _p(dx), None, None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    # nothing is written past the grid
    assert torch.all(y[n * co:] == 3.0) and torch.all(y32[n * co:] == 3.0) and torch.all(dx[x.numel():] == 3.0)
    return y[:n * co], y32[:n * co], dx[:x.numel()]


@pytest.mark.parametrize("ci,co,dims", [(16, 32, (16, 32, 48)), (64, 64, (17, 35, 21)), (32, 64, (40, 64, 64)), (64, 16, (1, 1, 1)),
                                        (32, 16, (6, 70, 33))])
def test_gpu_stride2_gradient_same_sums(gpu_lib, ci, co, dims):
    """The stride-2 input gradient by parity classes adds the taps and channels
    in the mma.sync kernel's order: equal bits."""
    L = gpu_lib.load()
    x, w, b, dy, _ = _data(ci, co, dims, 3, 2)
    auto = _run(L, gpu_lib, x, w, b, dy, dims, ci, co, 3, 2, 0)
    gpu_lib._check(L.lbm_nn_set_conv_engine(1))
    try:
        rows = _run(L, gpu_lib, x, w, b, dy, dims, ci, co, 3, 2, 0)
    finally:
        gpu_lib._check(L.lbm_nn_set_conv_engine(0))
    assert torch.equal(auto[2], rows[2])


@pytest.mark.parametrize("ci,co,dims", [(64, 64, (16, 8, 8)), (64, 64, (20, 15, 16)), (32, 64, (8, 8, 16))])
def test_gpu_low_grids_take_the_same_sums(gpu_lib, ci, co, dims):
    """Grids lower than a tensor-core block's 16 rows: both engines are the
    mma.sync kernel."""
    L = gpu_lib.load()
    x, w, b, dy, _ = _data(ci, co, dims, 3, 1)
    auto = _run(L, gpu_lib, x, w, b, dy, dims, ci, co, 3, 1, 1)
    gpu_lib._check(L.lbm_nn_set_conv_engine(1))
    try:
        rows = _run(L, gpu_lib, x, w, b, dy, dims, ci, co, 3, 1, 1)
    finally:
        gpu_lib._check(L.lbm_nn_set_conv_engine(0))
    assert all(torch.equal(a, r) for a, r in zip(auto, rows))
