"""The bounds-checked build (-DLBM_CHECK) on the compact kernel's launch shapes
of small and mid-sized lattices (blocks of 256, and (128, 8)) and on the shape
that a handle starts on: no index outside its array, results bit-identical to
the normal build.  In a child process, bound through LBM_LIBRARY."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys, numpy as np
sys.path.insert(0, {root!r})
from pv_dec_original_gb300 import capi
capi.load(build_if_missing=False)
out = {{}}
for nz, n in ((9, 20), (40, 33)):
    z, y, x = np.indices((nz + 2, n + 2, n + 2))
    mask = (((y - n / 2 - .5) ** 2 + (x - n / 2 - .5) ** 2 < (n / 2) ** 2) & (z > 0) & (z <= nz)).astype(np.uint8)
    for Q, prec in ((19, "f32"), (19, "f16"), (27, "bf16")):
        for v in (None, 3, 4):
            s = capi.Solver(Q, prec, capi.LBM_PHYSICS, 0.6, 1.0, (0.0, 0.0, 0.0), 1.0, 1.0)
            s.set_geometry(mask, [capi.bc_spec(capi.LBM_BC_VELOCITY, "z-", 1, 0.05),
                                  capi.bc_spec(capi.LBM_BC_PRESSURE, "z+", nz, 1.002)])
            if v is not None:
                s.set_variant(v)
            s.step(19)
            out[f"{{nz}}_{{Q}}_{{prec}}_{{v}}"] = s.distributions()
            s.close()
np.savez({path!r}, **out)
"""


def _child(lib, path):
    env = dict(os.environ)
    if lib:
        env["LBM_LIBRARY"] = lib
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, path=path)], env=env, capture_output=True, text=True,
                       timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return dict(np.load(path))


def test_checked_build_small_lattice_shapes(gpu_lib, tmp_path):
    from pv_dec_original_gb300 import build
    lib = build.build_checked()
    plain = _child(None, str(tmp_path / "plain.npz"))
    checked = _child(lib, str(tmp_path / "checked.npz"))
    assert set(plain) == set(checked) and len(plain) == 18
    for k in plain:
        assert np.isfinite(plain[k]).all() and np.array_equal(plain[k], checked[k]), k
