"""The launch shape a handle starts on and the compact shapes (variants 3, 4)
against the flat step kernel (variant 0), at node counts on both sides of each
line of the rule -- the blocks of 256, the shapes for buffers from 32 MB on,
evict-first loads up to 138 MB and the other block order from 86 MB on: the same
arithmetic on the same loads, so the distributions are bit-identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (Q, format, box of active nodes, [z][y][x])
CASES = [
    (19, "f32", (3, 5, 7)),
    (19, "f32", (12, 40, 25)),     # 12,000: blocks of 256
    (27, "bf16", (11, 31, 37)),    # 12,617
    (19, "f32", (60, 83, 84)),     # 31.8 MB a buffer
    (19, "f32", (61, 83, 84)),     # 32.3 MB
    (19, "f16", (101, 91, 93)),    # 32.5 MB
    (19, "bf16", (139, 128, 129)),  # 87 MB: evict-first, the other order
    (19, "f32", (151, 110, 111)),  # 140 MB: the other order alone
    (27, "f32", (111, 91, 81)),    # 88 MB
]


def _run(capi, Q, prec, box, variant):
    mask = np.zeros([b + 2 for b in box], np.uint8)
    mask[1:-1, 1:-1, 1:-1] = 1
    mask[1, 1, 1] = 0
    s = capi.Solver(Q, prec, capi.LBM_PHYSICS, 0.6, 1.0, (0.0, 0.0, 0.0), 1.0, 1.0)
    s.set_geometry(mask, [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", 1, 0.05), capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", box[0], 1.002)])
    if variant is not None:
        s.set_variant(variant)
    s.step(5)
    f = s.distributions()
    s.close()
    return f


@pytest.mark.parametrize("Q,prec,box", CASES)
def test_default_shape_bit_identical_to_flat(gpu_lib, Q, prec, box):
    ref = _run(gpu_lib, Q, prec, box, 0)
    assert np.isfinite(ref).all()
    for v in (None, 3, 4):
        assert np.array_equal(_run(gpu_lib, Q, prec, box, v), ref), v
