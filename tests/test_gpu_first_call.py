"""The first small solve of a process does not pin buffers for large ones.

The staging buffers are 64 MB each and are pinned when something is staged that needs
them; pinned memory of this size shows as shared resident memory of the process.
"""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np
import __graft_entry__ as ge
tp = ge.load_package()
def pinned():
    return next(int(l.split()[1]) for l in open("/proc/self/status") if l.startswith("RssShmem"))
MOMENT = (0.0, 0.0, -8.0e22)
u0 = np.array([[4 * tp.Re], [0.0], [0.0], [1.0e5], [1.0e5], [1.0e5]])
full = tp.TraceProblem(u0, (0.0, 1.0), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT)))
tp.solve(full, tp.Boris(), tp.EnsembleB200(), dt=0.01, trajectories=1)
before = pinned()
x = np.array([[4 * tp.Re], [0.0], [0.0], [1.0e6]])
gc = tp.TraceGCProblem(x, (0.0, 5.0), (tp.qi, tp.qi / tp.mi, 1.0e-10, tp.ZeroField(), tp.DipoleField(MOMENT)))
tp.solve(gc, tp.EnsembleB200(), alg="rk4", dt=0.5, trajectories=1)
tp.solve(full, tp.AdaptiveBoris(0.1), tp.EnsembleB200(), trajectories=1)
print(pinned() - before)
"""


def test_first_small_solves():
    out = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout.split()[-1]) < 16 << 10  # KB
