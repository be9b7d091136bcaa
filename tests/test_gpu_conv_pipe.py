"""The stride-1 tensor-core convolution (k_conv3_pipe) on grids its blocks do
not tile and on grids with several blocks a CTA, forward and input gradient,
against PyTorch in FP64 on BF16-exact values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


SHAPES = [(16, 16, (1, 1, 1)), (16, 32, (4, 16, 8)), (32, 16, (5, 17, 9)), (64, 64, (3, 40, 23)), (16, 64, (9, 33, 20)),
          (64, 16, (2, 15, 7)), (32, 64, (6, 31, 41)), (64, 32, (7, 16, 65)), (16, 16, (21, 64, 163)),
          (32, 32, (20, 65, 160)), (64, 64, (17, 80, 104)), (64, 32, (24, 48, 168))]


@pytest.mark.parametrize("ci,co,dims", SHAPES)
@pytest.mark.parametrize("relu", [0, 1])
def test_gpu_conv_pipe_matches_fp64(gpu_lib, ci, co, dims, relu):
    """FP32 accumulation of BF16-exact products: 1e-5 of the output scale;
    the BF16 results are roundings of it (8e-3, as the other engine tests)."""
    L = gpu_lib.load()
    g = torch.Generator(device="cuda").manual_seed(ci + 3 * co + sum(dims))
    D, H, W = dims
    n = D * H * W

    def bf(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)

    x, w, dy = bf(D, H, W, ci), bf(co, 27, ci, scale=0.2), bf(D, H, W, co)
    b = torch.randn(co, generator=g, device="cuda") * 0.1
    wt = w.double().reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3).contiguous()
    xt = x.double().permute(3, 0, 1, 2)[None].contiguous().requires_grad_(True)
    yt = torch.nn.functional.conv3d(xt, wt, b.double(), padding=1)
    yt.backward(dy.double().permute(3, 0, 1, 2)[None])
    ref = yt.detach()[0].permute(1, 2, 3, 0)
    ref = ref.relu() if relu else ref
    y = torch.full((n * co + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    y32 = torch.full((n * co + 64,), 3.0, device="cuda")
    dx = torch.full((n * ci + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty_like(w)
    dims_c = (C.c_int * 3)(*dims)
    gpu_lib._check(L.lbm_nn_conv3d_fwd(_p(x), dims_c, ci, _p(w), _p(b), co, 3, 1, relu, _p(y), _p(y32), None))
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), dims_c, ci, _p(w), _p(scratch), co, 3, 1, _p(dy), _p(dx), None, None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    got = y32[:n * co].double().reshape(D, H, W, co)
    assert float((got - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert torch.equal(y[:n * co], y32[:n * co].to(torch.bfloat16))
    dref = xt.grad[0].permute(1, 2, 3, 0)
    assert float((dx[:n * ci].double().reshape(D, H, W, ci) - dref).abs().max()) <= 8e-3 * float(dref.abs().max())
    # nothing is written past the grid
    assert torch.all(y[n * co:] == 3.0) and torch.all(y32[n * co:] == 3.0) and torch.all(dx[n * ci:] == 3.0)
