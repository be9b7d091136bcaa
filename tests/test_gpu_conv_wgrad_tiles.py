"""The tile weight gradient (k_conv_wgrad_tiles) at the edges of its tiles:
grids below one tile, one voxel over, ragged in every axis, odd strided
grids and 1x1x1 layers, against a PyTorch FP64 gradient of the same values;
dw is accumulated into."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


CASES = [(16, 16, (1, 1, 1), 3, 1), (16, 16, (4, 8, 32), 3, 1), (16, 16, (5, 9, 33), 3, 1), (32, 16, (7, 3, 70), 3, 1),
         (64, 32, (5, 9, 17), 3, 1), (16, 64, (3, 17, 15), 3, 1), (64, 64, (9, 8, 16), 3, 1), (16, 32, (8, 16, 64), 3, 2),
         (32, 64, (7, 9, 35), 3, 2), (64, 16, (3, 2, 1), 3, 2), (16, 16, (5, 9, 33), 1, 1), (64, 32, (4, 8, 16), 1, 1),
         (32, 64, (3, 25, 47), 1, 1), (16, 16, (40, 33, 65), 3, 1)]


@pytest.mark.parametrize("ci,co,dims,ks,s", CASES)
def test_gpu_weight_gradient_tile_edges(gpu_lib, ci, co, dims, ks, s):
    """FP32 sums of BF16-exact products over n voxels: 1e-5 of the
    gradient's scale, the tolerance of the other weight-gradient tests."""
    L = gpu_lib.load()
    rng = np.random.default_rng(ci + 2 * co + sum(dims) + ks + s)

    def bf(a):
        return torch.as_tensor(a).to(torch.bfloat16).to(torch.float64)

    x = bf(rng.normal(size=(*dims, ci)))
    w = torch.zeros((co, ci, ks, ks, ks), dtype=torch.float64, requires_grad=True)
    y = torch.nn.functional.conv3d(x.permute(3, 0, 1, 2)[None], w, None, stride=s, padding=ks // 2)
    dy = bf(rng.normal(size=(*y.shape[2:], co)))
    y.backward(dy.permute(3, 0, 1, 2)[None])
    ref = w.grad.permute(0, 2, 3, 4, 1).reshape(-1)
    xd = x.to(torch.bfloat16).cuda().reshape(-1)
    dyd = dy.to(torch.bfloat16).cuda().reshape(-1)
    wd = torch.zeros(ref.numel(), dtype=torch.bfloat16, device="cuda")
    dw = torch.full((ref.numel(),), 0.25, device="cuda")
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(xd), (C.c_int * 3)(*dims), ci, _p(wd), None, co, ks, s, _p(dyd), None, _p(dw),
                                       None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    got = dw.cpu().double() - 0.25
    assert float((got - ref).abs().max()) <= 1e-5 * float(ref.abs().max()) + 1e-6
