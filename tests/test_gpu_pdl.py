"""GPU: the cycle with programmatic dependent launch (AGB_PDL=1, read once a
process) against the default.  The kernels and their order are the same, and on
a box with no periodic direction no sum depends on the order of blocks (norms
are maxima), so the solutions agree bit for bit.  48 and 64 cells an edge lie on
either side of the FP64 column kernel's smallest box."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOLVE = """
import sys
import numpy as np
from alamo_gb300 import Elastic, Linear, TensionTest
from alamo_gb300 import microstructure as M
n, mixed, sym, path = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3], sys.argv[4]
op = Elastic([n] * 3, None, sym)
op.SetBC(TensionTest("uniaxial_stress", disp=0.01))
N = op.nodes()
r = np.random.default_rng(7)
if sym == "isotropic":
    ddw = r.uniform(0.9, 1.3, size=2 * N)
else:
    one = M.cubic(1.68, 1.21, 0.75, M.quat_to_rot([1.0, 0.4, -0.2, 0.3]))
    ddw = (one[None, :] * r.uniform(1.0, 1.1, size=(N, 1))).reshape(-1)
op.SetModel(ddw)
rhs = op.BCInit(np.zeros(3 * N))
out = [op.Fapply(0, r.uniform(-1, 1, 3 * N))]
s = Linear(op, precision=mixed)
for _ in range(2):
    x = np.zeros(3 * N)
    s.solve(x, rhs, 1e-8, 0.0)
    out.append(x)
np.save(path, np.concatenate(out))
"""


@pytest.mark.parametrize("n,mixed,sym", [(48, 0, "majorminor"), (64, 0, "majorminor"), (64, 0, "isotropic"),
                                         (64, 1, "majorminor")])
def test_dependent_launch_solves_the_same(gpu_lib, tmp_path, n, mixed, sym):
    got = []
    for pdl in ("0", "1"):
        path = str(tmp_path / ("x%s.npy" % pdl))
        env = dict(os.environ, AGB_PDL=pdl, PYTHONPATH=ROOT)
        subprocess.run([sys.executable, "-c", SOLVE, str(n), str(mixed), sym, path], check=True, timeout=300, cwd=ROOT,
                       env=env)
        got.append(np.load(path))
    assert np.array_equal(got[0], got[1])
