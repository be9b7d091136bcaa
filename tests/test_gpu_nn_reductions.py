"""The network's reductions -- bias gradient and masked squared error -- at
sizes around their blocks, against FP64 sums of the same values."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 1, 31), (2, 3, 43), (5, 7, 147), (9, 64, 301)])
@pytest.mark.parametrize("co", [16, 32, 64])
def test_gpu_bias_gradient_sizes(gpu_lib, dims, co):
    """A thread adds at most rows co / 8 / (608 256) + 1 values and the rest
    is a tree: the FP32 sum is within 64 eps of the sum of magnitudes."""
    g = torch.Generator(device="cuda").manual_seed(co + dims[2])
    rows = int(np.prod(dims))
    x = torch.randn(rows * 16, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(co * 16, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(rows * co, generator=g, device="cuda").to(torch.bfloat16)
    db = torch.full((co,), 0.5, device="cuda")
    L = gpu_lib.load()
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), (C.c_int * 3)(*dims), 16, _p(w), None, co, 1, 1, _p(dy), None, None,
                                       _p(db), None))
    d = dy.double().reshape(rows, co)
    ref, mag = d.sum(0) + 0.5, d.abs().sum(0) + 0.5
    assert torch.all((db.double() - ref).abs() <= 64 * 2.0 ** -24 * mag)


@pytest.mark.parametrize("nvox", [1, 255, 257, 40000, 400003])
@pytest.mark.parametrize("c,nc,shift", [(16, 4, 0), (16, 4, 1), (16, 16, 0), (8, 3, 0), (5, 2, 0)])
def test_gpu_masked_error_sizes(gpu_lib, nvox, c, nc, shift):
    """shift: the prediction off 16-byte alignment (the general kernel)."""
    g = torch.Generator(device="cuda").manual_seed(nvox + c)
    pred = torch.randn(nvox * c + shift, generator=g, device="cuda")[shift:]
    tgt = torch.randn(nvox * nc, generator=g, device="cuda")
    mask = (torch.rand(nvox, generator=g, device="cuda") < 0.6).to(torch.uint8)
    p2 = pred.reshape(nvox, c)
    p2[mask == 0] = float("nan")  # values outside the mask count nowhere
    inv = 1.0 / max(1, 4 * int(mask.sum()))
    dpred = torch.full((nvox * c,), 7.0, dtype=torch.bfloat16, device="cuda")
    loss = torch.full((1,), 0.25, device="cuda")
    L = gpu_lib.load()
    gpu_lib._check(L.lbm_nn_mse(_p(pred), _p(tgt), _p(mask), nvox, c, nc, inv, _p(dpred), _p(loss), None))
    d = torch.zeros((nvox, c), device="cuda")
    on = mask.bool()
    d[on, :nc] = p2[on, :nc] - tgt.reshape(nvox, nc)[on]
    inv32 = torch.tensor(inv, dtype=torch.float32, device="cuda")
    assert torch.equal(dpred.reshape(nvox, c), (2.0 * d * inv32).to(torch.bfloat16))
    ref = (d.double() ** 2).sum() * inv + 0.25
    # up to 8 c values a thread, then a tree and one addition a block
    assert abs(float(loss) - float(ref)) <= 1e-4 * float(ref)
