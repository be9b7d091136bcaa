"""Convolution gradients on either side of the lines of the dispatch: weight
gradients of few voxels (the plain kernel up to 96 output voxels at kernel size
3 and 24 at 1) and of grids thinner than a tile along z, input gradients at
stride 2 on columns of few voxels a plane, against PyTorch in FP64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


def _bf(a):
    return torch.as_tensor(a).to(torch.bfloat16).to(torch.float64)


@pytest.mark.parametrize("dims,ks,s", [((1, 1, 96), 3, 1), ((1, 1, 97), 3, 1), ((4, 8, 3), 3, 1), ((7, 2, 7), 3, 1),
                                       ((1, 1, 191), 3, 2), ((1, 1, 193), 3, 2), ((8, 8, 11), 3, 2), ((1, 1, 24), 1, 1),
                                       ((1, 5, 5), 1, 1), ((1, 20, 37), 3, 1), ((2, 9, 33), 3, 1), ((3, 17, 15), 3, 1),
                                       ((1, 20, 37), 3, 2), ((2, 33, 36), 3, 2), ((3, 18, 70), 3, 2), ((1, 11, 13), 1, 1)])
@pytest.mark.parametrize("ci,co", [(16, 16), (32, 64), (64, 16)])
def test_gpu_weight_gradient_small_grids(gpu_lib, ci, co, dims, ks, s):
    """FP32 sums of BF16-exact products: 1e-5 of the gradient's scale, the
    tolerance of the other weight-gradient tests."""
    L = gpu_lib.load()
    rng = np.random.default_rng(ci + 2 * co + sum(dims) + ks + s)
    x = _bf(rng.normal(size=(*dims, ci)))
    w = torch.zeros((co, ci, ks, ks, ks), dtype=torch.float64, requires_grad=True)
    y = torch.nn.functional.conv3d(x.permute(3, 0, 1, 2)[None], w, None, stride=s, padding=ks // 2)
    dy = _bf(rng.normal(size=(*y.shape[2:], co)))
    y.backward(dy.permute(3, 0, 1, 2)[None])
    ref = w.grad.permute(0, 2, 3, 4, 1).reshape(-1)
    xd, dyd = x.to(torch.bfloat16).cuda().reshape(-1), dy.to(torch.bfloat16).cuda().reshape(-1)
    wd = torch.zeros(ref.numel(), dtype=torch.bfloat16, device="cuda")
    dw = torch.full((ref.numel(),), 0.25, device="cuda")
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(xd), (C.c_int * 3)(*dims), ci, _p(wd), None, co, ks, s, _p(dyd), None, _p(dw),
                                       None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    assert float((dw.cpu().double() - 0.25 - ref).abs().max()) <= 1e-5 * float(ref.abs().max()) + 1e-6


@pytest.mark.parametrize("dims", [(40, 1, 1), (7, 4, 8), (6, 3, 5), (5, 6, 6), (9, 2, 17), (4, 16, 2)])
@pytest.mark.parametrize("ci,co", [(16, 16), (64, 64)])
def test_gpu_stride_two_input_gradient_columns(gpu_lib, ci, co, dims):
    """The two kernels' sums are the same: equal bits; 8e-3 of the scale against
    FP64 (BF16 roundings), as the other convolution tests."""
    L = gpu_lib.load()
    rng = np.random.default_rng(ci + co + sum(dims))
    od = [(d - 1) // 2 + 1 for d in dims]
    dy, w = _bf(rng.normal(size=(*od, co))), _bf(rng.normal(size=(co, 27, ci)) * 0.2)
    xt = torch.zeros((1, ci, *dims), dtype=torch.float64, requires_grad=True)
    wt = w.reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3).contiguous()
    torch.nn.functional.conv3d(xt, wt, None, stride=2, padding=1).backward(dy.permute(3, 0, 1, 2)[None])
    ref = xt.grad[0].permute(1, 2, 3, 0)
    dyd, wd = dy.to(torch.bfloat16).cuda().reshape(-1), w.to(torch.bfloat16).cuda().reshape(-1)
    xd, scratch, got = torch.zeros(ref.numel(), dtype=torch.bfloat16, device="cuda"), torch.empty_like(wd), []
    for engine in (0, 1):
        gpu_lib._check(L.lbm_nn_set_conv_engine(engine))
        try:
            dx = torch.full((ref.numel() + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
            gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(xd), (C.c_int * 3)(*dims), ci, _p(wd), _p(scratch), co, 3, 2, _p(dyd), _p(dx),
                                               None, None, None))
            torch.cuda.synchronize()
            gpu_lib._check(L.lbm_nn_conv_status())
        finally:
            gpu_lib._check(L.lbm_nn_set_conv_engine(0))
        assert torch.all(dx[ref.numel():] == 3.0)
        got.append(dx[:ref.numel()])
    assert torch.equal(*got)
    assert float((got[0].cpu().double().reshape(ref.shape) - ref).abs().max()) <= 8e-3 * float(ref.abs().max())
