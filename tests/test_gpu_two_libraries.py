"""The two- and the three-material library in one process, in either order: the FP64_FMA
path's row sort asks for more shared memory than a kernel has by default, in each
library for itself.  Child processes, so that the order of loading is known."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import sys
from pgdg_p2_gb300 import mpm as M
for cid in map(int, sys.argv[1:]):
    cs, p, c = M.make_case(cid, (40, 17))
    for prec in (2, 1, 0):
        g = M.MPM(cs, prec)
        if prec == 2:
            g.tune("pst", 0)
        g.upload_particles(p)
        g.upload_cells(c)
        g.advance(2)
        g.sync()
        g.close()
"""


@pytest.mark.parametrize("order", [("1", "5"), ("5", "1")])
def test_both_libraries_run(gpu_mod, order):
    r = subprocess.run([sys.executable, "-c", CODE, *order], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
