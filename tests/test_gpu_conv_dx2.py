"""The stride-2 input gradient on the tensor cores (k_conv3_dx2) on even and
odd grids, below one block, ragged and with several blocks a CTA, against
PyTorch in FP64 on BF16-exact values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("ci,co,dims", [(16, 32, (1, 1, 1)), (16, 32, (2, 2, 2)), (16, 16, (3, 2, 1)), (32, 64, (4, 32, 16)),
                                        (64, 64, (5, 33, 17)), (16, 32, (7, 31, 18)), (64, 16, (6, 35, 50)),
                                        (32, 32, (3, 70, 34)), (16, 32, (64, 65, 130)), (32, 64, (41, 64, 96)),
                                        (64, 64, (40, 66, 63)), (16, 64, (33, 48, 80))])
def test_gpu_conv_dx2_matches_fp64(gpu_lib, ci, co, dims):
    """The BF16 result is a rounding of the FP64 one (8e-3 of the scale, as
    the other engine tests)."""
    L = gpu_lib.load()
    g = torch.Generator(device="cuda").manual_seed(ci + 3 * co + sum(dims))
    D, H, W = dims
    n = D * H * W
    x = torch.zeros(n * ci, dtype=torch.bfloat16, device="cuda")
    w = (torch.randn(co, 27, ci, generator=g, device="cuda") * 0.2).to(torch.bfloat16)
    wt = w.double().reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3).contiguous()
    xt = torch.zeros((1, ci, D, H, W), dtype=torch.float64, device="cuda", requires_grad=True)
    yt = torch.nn.functional.conv3d(xt, wt, None, stride=2, padding=1)
    dy = torch.randn(*yt.shape[2:], co, generator=g, device="cuda").to(torch.bfloat16)
    yt.backward(dy.double().permute(3, 0, 1, 2)[None])
    dx = torch.full((n * ci + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty_like(w)
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), (C.c_int * 3)(*dims), ci, _p(w), _p(scratch), co, 3, 2, _p(dy), _p(dx),
                                       None, None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    ref = xt.grad[0].permute(1, 2, 3, 0)
    got = dx[:n * ci].double().reshape(D, H, W, ci)
    assert float((got - ref).abs().max()) <= 8e-3 * float(ref.abs().max())
    assert torch.all(dx[n * ci:] == 3.0)  # nothing is written past the grid
