"""1x1x1 layers with 64 columns in a block (two stages; with 16 channels one
tile a block, else a grid of resident blocks): forward with and without the FP32
output, and input gradient, around the tile of 64 rows and the line at 152 tiles,
against FP64 products of BF16-exact values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("rows", [152 * 64 - 1, 152 * 64, 152 * 64 + 1, 152 * 64 * 7 + 33])
@pytest.mark.parametrize("ci,co", [(16, 64), (32, 64), (64, 64), (64, 16), (64, 32)])
def test_gpu_1x1_columns(gpu_lib, ci, co, rows):
    """FP32 accumulation of BF16-exact products: 1e-5 of the output scale; the
    BF16 gradients are roundings of it (8e-3), as the other convolution tests."""
    L = gpu_lib.load()
    g = torch.Generator(device="cuda").manual_seed(ci + 3 * co + rows)

    def bf(*shape):
        return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)

    x, w, dy = bf(rows, ci), bf(co, ci), bf(rows, co)
    b = torch.randn(co, generator=g, device="cuda")
    ref = (x.double() @ w.double().T + b.double()).relu()
    dref = dy.double() @ w.double()
    dims, scratch = (C.c_int * 3)(1, 1, rows), torch.empty_like(w)
    y32 = torch.full((rows * co + 64,), 3.0, device="cuda")
    ys = []
    for out32 in (None, y32):
        y = torch.full((rows * co + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
        gpu_lib._check(L.lbm_nn_conv3d_fwd(_p(x), dims, ci, _p(w), _p(b), co, 1, 1, 1, _p(y), _p(out32), None))
        ys.append(y)
    dx = torch.full((rows * ci + 64,), 3.0, dtype=torch.bfloat16, device="cuda")
    gpu_lib._check(L.lbm_nn_conv3d_bwd(_p(x), dims, ci, _p(w), _p(scratch), co, 1, 1, _p(dy), _p(dx), None, None, None))
    torch.cuda.synchronize()
    n = rows * co
    assert float((y32[:n].double().reshape(rows, co) - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[1][:n], y32[:n].to(torch.bfloat16))
    assert float((dx[:rows * ci].double().reshape(rows, ci) - dref).abs().max()) <= 8e-3 * float(dref.abs().max())
    # nothing is written past the grid
    assert torch.all(ys[0][n:] == 3.0) and torch.all(y32[n:] == 3.0) and torch.all(dx[rows * ci:] == 3.0)
