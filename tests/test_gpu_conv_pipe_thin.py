"""The stride-1 tensor-core convolution (k_conv3_pipe takes grids of 16 rows or
more) on grids thinner than its 4 x 16 x 8 block in z and x, or one row over it,
forward and input gradient, against PyTorch in FP64 on BF16-exact values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("dims", [(1, 16, 1), (1, 17, 3), (2, 16, 7), (3, 31, 1), (1, 16, 8), (4, 33, 1), (5, 16, 2), (1, 64, 9)])
@pytest.mark.parametrize("ci,co", [(16, 16), (64, 64), (16, 64), (64, 32)])
def test_gpu_conv_pipe_thin_grids(gpu_lib, ci, co, dims):
    """FP32 accumulation of BF16-exact products: 1e-5 of the output scale; the
    BF16 gradients are roundings of it (8e-3), as the other convolution tests."""
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
    ref, dref = yt.detach()[0].permute(1, 2, 3, 0), xt.grad[0].permute(1, 2, 3, 0)
    y = torch.full((n * co + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    y32 = torch.full((n * co + 64,), 3.0, device="cuda")
    dx = torch.full((n * ci + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty_like(w)
    dims_c = (C.c_int * 3)(*dims)
    gpu_lib._check(L.lbm_nn_conv3d_fwd(_p(x), dims_c, ci, _p(w), _p(b), co, 3, 1, 0, _p(y), _p(y32), None))
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), dims_c, ci, _p(w), _p(scratch), co, 3, 1, _p(dy), _p(dx), None, None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    assert float((y32[:n * co].double().reshape(D, H, W, co) - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert torch.equal(y[:n * co], y32[:n * co].to(torch.bfloat16))
    assert float((dx[:n * ci].double().reshape(D, H, W, ci) - dref).abs().max()) <= 8e-3 * float(dref.abs().max())
    # nothing is written past the grid
    assert torch.all(y[n * co:] == 3.0) and torch.all(y32[n * co:] == 3.0) and torch.all(dx[n * ci:] == 3.0)
