"""The gradient at a layer's output in one pass (lbm_nn_layer_grad) against the
passes that it stands for: sum, copy, ReLU (equal bits) and bias gradient."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("c", [16, 32, 64])
@pytest.mark.parametrize("rows", [1, 31, 257, 20011])
@pytest.mark.parametrize("add,copy", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_gpu_layer_grad_matches_passes(gpu_lib, c, rows, add, copy):
    L = gpu_lib.load()
    g = torch.Generator(device="cuda").manual_seed(rows + c)

    def bf():
        return torch.randn(rows * c, generator=g, device="cuda").to(torch.bfloat16)

    y, dy, other = bf().relu(), bf(), bf()
    y[:3], dy[1] = torch.tensor([float("nan"), float("inf"), -0.0]), -0.0
    ref = dy.clone()
    if add:
        gpu_lib._check(L.lbm_nn_add(_p(ref), _p(other), _p(ref), rows * c, None))
    ref_copy = ref.clone()
    gpu_lib._check(L.lbm_nn_relu_bwd(_p(y), _p(ref), rows * c, None))
    db = torch.full((c + 8,), 0.5, device="cuda")
    out = torch.zeros_like(dy) if copy else None
    gpu_lib._check(L.lbm_nn_layer_grad(_p(y), _p(other) if add else None, _p(dy), _p(out), _p(db), rows, c, None))
    torch.cuda.synchronize()
    assert torch.equal(dy.view(torch.int16), ref.view(torch.int16))
    if copy:
        assert torch.equal(out.view(torch.int16), ref_copy.view(torch.int16))
    want = ref.double().reshape(rows, c).sum(0) + 0.5
    # FP32 additions, at most rows of them in a chain of partial sums: 2^-24 per level of the terms' total
    scale = ref.double().abs().reshape(rows, c).sum(0) + 0.5
    assert torch.all((db[:c].double() - want).abs() <= 2e-6 * scale) and torch.all(db[c:] == 0.5)


def test_gpu_layer_grad_refuses(gpu_lib):
    L = gpu_lib.load()
    t = torch.zeros(64, dtype=torch.bfloat16, device="cuda")
    db = torch.zeros(64, device="cuda")
    off = C.c_void_p(t.data_ptr() + 2)
    assert L.lbm_nn_layer_grad(_p(t), None, _p(t), None, _p(db), 1, 24, None) != 0
    assert L.lbm_nn_layer_grad(off, None, _p(t), None, _p(db), 1, 16, None) != 0
    assert L.lbm_nn_layer_grad(None, None, _p(t), None, _p(db), 1, 16, None) != 0
    assert L.lbm_nn_layer_grad(_p(t), None, _p(t), None, _p(db), 0, 16, None) == 0
