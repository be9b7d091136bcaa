"""The mma.sync convolution (k_conv_gemm): steps pipelined across taps and
tiles, 16 columns a block or all of them, forward and input gradient, against
PyTorch in FP64 on BF16-exact values."""
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


@pytest.mark.parametrize("ci,co,dims,ks,stride", [
    (16, 16, (1, 1, 1), 3, 1), (64, 64, (16, 8, 8), 3, 1), (32, 64, (3, 5, 7), 3, 1), (64, 32, (13, 15, 101), 3, 1),
    (16, 64, (63, 14, 23), 3, 1), (16, 32, (5, 7, 9), 3, 2), (64, 64, (7, 33, 21), 3, 2), (32, 64, (64, 37, 44), 3, 2),
    (64, 32, (6, 17, 40), 3, 1), (32, 16, (9, 30, 44), 3, 2), (16, 16, (1, 1, 63), 1, 1), (64, 16, (1, 1, 64), 1, 1),
    (16, 32, (5, 13, 301), 1, 1), (32, 64, (9, 16, 151), 1, 1), (16, 16, (40, 60, 41), 1, 1)])
@pytest.mark.parametrize("relu", [0, 1])
def test_gpu_conv_rows_matches_fp64(gpu_lib, ci, co, dims, ks, stride, relu):
    """FP32 accumulation of BF16-exact products: 1e-5 of the output scale;
    the BF16 results are roundings of it (8e-3, as the other engine tests)."""
    L = gpu_lib.load()
    x, w, b, dy, od = _data(ci, co, dims, ks, stride)
    gpu_lib._check(L.lbm_nn_set_conv_engine(1))
    try:
        y, y32, dx = _run(L, gpu_lib, x, w, b, dy, dims, ci, co, ks, stride, relu)
    finally:
        gpu_lib._check(L.lbm_nn_set_conv_engine(0))
    wt = w.double().reshape(co, ks, ks, ks, ci).permute(0, 4, 1, 2, 3).contiguous()
    xt = x.double().permute(3, 0, 1, 2)[None].contiguous().requires_grad_(True)
    yt = torch.nn.functional.conv3d(xt, wt, b.double(), padding=ks // 2, stride=stride)
    yt.backward(dy.double().permute(3, 0, 1, 2)[None])
    ref = yt.detach()[0].permute(1, 2, 3, 0)
    ref = ref.relu() if relu else ref
    assert float((y32.double().reshape(*od, co) - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert torch.equal(y, y32.to(torch.bfloat16))
    dref = xt.grad[0].permute(1, 2, 3, 0)
    assert float((dx.double().reshape(*dims, ci) - dref).abs().max()) <= 8e-3 * float(dref.abs().max())
