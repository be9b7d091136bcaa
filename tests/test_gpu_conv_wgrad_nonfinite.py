"""The tile weight gradient with infinities in the activations of the grid's
last layers: only the taps and channels whose sums meet one are not finite, as
in a sum over the output voxels alone, also where a tile reaches past the grid."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


CASES = [(16, 16, (4, 8, 32), 3, 1), (16, 16, (5, 9, 33), 3, 1), (16, 16, (2, 3, 17), 3, 1), (32, 32, (6, 13, 29), 3, 1),
         (64, 64, (3, 17, 15), 3, 1), (16, 32, (6, 10, 36), 3, 2), (32, 16, (8, 14, 22), 3, 2), (16, 64, (7, 9, 35), 3, 2),
         (16, 16, (3, 5, 37), 1, 1), (32, 32, (3, 5, 19), 1, 1)]


@pytest.mark.parametrize("ci,co,dims,ks,s", CASES)
def test_gpu_weight_gradient_infinities(gpu_lib, ci, co, dims, ks, s):
    """Finite elements: FP32 sums of BF16-exact products, 1e-5 of the gradient's
    scale as in the other weight-gradient tests."""
    L = gpu_lib.load()
    rng = np.random.default_rng(ci + 2 * co + sum(dims) + ks + s)
    bf = lambda a: torch.as_tensor(a).to(torch.bfloat16).to(torch.float64)
    x = bf(rng.normal(size=(*dims, ci)))
    bad = torch.zeros_like(x)
    bad[-1, :, :, 1] = bad[:, -1, :, 2] = bad[:, :, -1, 3] = bad[0, 0, 0, 4] = 1.0
    x[bad > 0] = 0.0

    def gradient(v, d):
        w = torch.zeros((co, ci, ks, ks, ks), dtype=torch.float64, requires_grad=True)
        torch.nn.functional.conv3d(v.permute(3, 0, 1, 2)[None], w, None, stride=s, padding=ks // 2).backward(
            d.permute(3, 0, 1, 2)[None])
        return w.grad.permute(0, 2, 3, 4, 1).reshape(-1)

    od = [(d - 1) // s + 1 for d in dims]
    dy = bf(rng.normal(size=(*od, co)))
    dy[dy == 0] = 1.0
    ref, meets = gradient(x, dy), gradient(bad, torch.ones_like(dy)) > 0
    xd = x.masked_fill(bad > 0, float("inf")).to(torch.bfloat16).cuda().reshape(-1)
    dyd = dy.to(torch.bfloat16).cuda().reshape(-1)
    wd = torch.zeros(ref.numel(), dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros(ref.numel(), device="cuda")
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(xd), (C.c_int * 3)(*dims), ci, _p(wd), None, co, ks, s, _p(dyd), None, _p(dw),
                                       None, None))
    torch.cuda.synchronize()
    gpu_lib._check(L.lbm_nn_conv_status())
    got = dw.cpu().double()
    assert torch.equal(torch.isfinite(got), ~meets)
    assert float((got - ref)[~meets].abs().max()) <= 1e-5 * float(ref.abs().max()) + 1e-6
