"""The FP64 step's forms with fewer operations against the oracle, bit for
bit where the reference's rounding is kept: quotients by one reciprocal at
states whose momenta are zero, of either sign, tiny or ordinary, and the
stress of blocks of next-to-wall nodes through graphs and single steps."""
import numpy as np
import pytest

from helpers import classify, fixtures, load, sim_bcs, wss_C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.0, 1e-300, 1e-160, 1e-17, 1e-9, 1e-2])
@pytest.mark.parametrize("steps,graph", [(1, 0), (2, 0), (19, 4)])
def test_gpu_f64_parity_from_any_momentum(gpu_lib, oracle_lib, scale, steps, graph):
    d = load(fixtures("sim")[0])
    capi = gpu_lib
    mask, desc = capi.voxelize(d["tri12"], float(d["spacing"]))
    bb = np.array(desc.bbox[:])
    org, sp, tau = (bb[0], bb[2], bb[4]), float(d["spacing"]), float(d["tau"])
    bcs = sim_bcs(d)
    C = wss_C(float(d["dt"]), sp)
    s = capi.Solver(19, capi.LBM_F64, capi.LBM_PARITY, tau, sp, org, C, 0.9)
    s.set_geometry(mask, [capi.bc_spec(**spec) for _, spec in bcs])
    s.set_normals(d["tri12"])
    s.set_inlet_table(d["amp"])
    s.set_graph_steps(graph)
    o = oracle_lib.Sim(19, oracle_lib.PARITY, classify(mask, [(a, spec["plane"]) for a, spec in bcs]), org, sp, tau,
                       [spec for _, spec in bcs])
    o.set_amplitude(d["amp"])
    o.set_wss(C, 0.9)
    o.compute_normals(d["tri12"])
    c, w, _ = oracle_lib.lattice(19)
    rng = np.random.default_rng(int(steps))
    n = s.counts()["active"]
    f = np.tile(np.asarray(w, float)[None], (n, 1))
    # momenta of magnitude `scale` in populations that can hold it, some densities near the mantissa's end
    f *= 1.0 + rng.choice([0.0, 1.0, -1.0], (n, 19)) * scale
    f[::7] *= 1.0 - 2.0 ** -53 * rng.integers(0, 3, (len(f[::7]), 1))
    s.set_distributions(f)
    o.set_f(f)
    s.step(steps)
    o.step(steps)
    fo, _, _ = o.f()
    assert np.array_equal(s.distributions(), fo)
    g, r = s.wss(), o.nw()
    assert np.array_equal(g["pt"], r["pt"])
    for key in ("wss", "acc", "acc_mag"):
        np.testing.assert_allclose(g[key], r[key], rtol=1e-11, atol=1e-13 * max(np.abs(r[key]).max(), 1e-300))
