"""Lattices whose steps share the device's L2 with others': the launch shape and
loads that a handle uses change with the steps of others in flight -- also under
captured graphs -- and its results do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(capi, box, Q=19, prec="f32"):
    mask = np.zeros([b + 2 for b in box], np.uint8)
    mask[1:-1, 1:-1, 1:-1] = 1
    mask[1, 1, 1] = 0
    s = capi.Solver(Q, prec, capi.LBM_PHYSICS, 0.6, 1.0, (0.0, 0.0, 0.0), 1.0, 1.0)
    s.set_geometry(mask, [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", 1, 0.05), capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", box[0], 1.002)])
    return s


def _state(s):
    w = s.wss()  # (no normals are set: no stress, and OSI 0 / 0)
    return [s.distributions(), w["wss"], w["osi"], w["tawss"]]


@pytest.mark.parametrize("Q,prec", [(19, "f32"), (19, "f16"), (27, "f32"), (19, "f64")])
@pytest.mark.parametrize("graph", [0, 4])
@pytest.mark.parametrize("tune", [False, True])
def test_gpu_step_beside_other_lattices(gpu_lib, Q, prec, graph, tune):
    box = (40, 33, 31)
    alone = _solver(gpu_lib, box, Q, prec)
    alone.set_graph_steps(graph)
    alone.step(33)
    ref = _state(alone)
    alone.close()
    s = _solver(gpu_lib, box, Q, prec)
    if tune:
        s.autotune(2)
    s.set_graph_steps(graph)
    s.step(11)
    other = _solver(gpu_lib, (140, 128, 109))  # 148 MB a buffer: both together beyond the L2
    other.step_async(20)
    s.step_async(11)  # beside the other's steps
    s.sync()
    s.step_async(1)
    other.sync()
    s.sync()
    s.step(10)
    other.close()
    got = _state(s)
    s.close()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b, equal_nan=True)
