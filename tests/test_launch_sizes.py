"""Grids that depend on the number of SMs take it from the device: no launcher
or kernel writes it out."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pv_dec_original_gb300", "csrc")


def test_no_written_out_sm_count():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            for n, line in enumerate(f, 1):
                if re.search(r"\b(148|152)\b", re.sub(r"//.*", "", line)):
                    found.append("%s:%d: %s" % (os.path.basename(path), n, line.strip()))
    assert not found, "\n".join(found)
