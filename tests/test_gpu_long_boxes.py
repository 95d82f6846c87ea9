"""GPU: boxes longer than 65535 blocks of a kernel's tile in y or z.  All fields
repeat along the long direction every 32 cells, so a result away from its ends is
that of a box of 96 cells (the oracle's), repeated; FP64 sums as in the other
operator tests (1e-12), transfers 1e-14."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def repeated(block, axis, n):
    """block (one period of 32 nodes along `axis`) repeated to n + 1 nodes."""
    import torch
    idx = torch.arange(n + 1, device=block.device) % 32
    return block.index_select(axis, idx).contiguous()


def check_repeats(out, want, axis):
    """Largest difference of out, but for a period at both ends, from the middle of want's three periods."""
    period = want.shape[axis] // 3
    mid = want.narrow(axis, period, period)
    n = (out.shape[axis] - 1) // period
    a = out.narrow(axis, period, (n - 2) * period).unflatten(axis, (n - 2, period))
    err = (a - mid.unsqueeze(axis)).abs().max()
    return float(err / want.abs().max())


@pytest.mark.parametrize("n", [(40, 4, 87424)])
def test_transfers_of_a_long_box(gpu_lib, n):
    import torch
    from alamo_gb300 import Elastic
    op = Elastic(list(n), [0.1] * 3, "isotropic")
    c = [v // 2 for v in n]
    gen = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) - 0.5  # noqa: E731
    small = (n[0], n[1], 96)
    g = O.make_grid(small, dx=[0.1] * 3)
    cpu = lambda t: np.ascontiguousarray(t.cpu().numpy().reshape(-1))  # noqa: E731
    # restriction: a period of 32 fine nodes is one of 16 coarse nodes
    block = rnd(3, 32, n[1] + 1, n[0] + 1)
    fine = repeated(block, 1, n[2])
    crse = torch.empty(3, c[2] + 1, c[1] + 1, c[0] + 1, dtype=torch.float64, device="cuda")
    op.restriction(1, fine, crse)
    want = torch.from_numpy(O.restriction(g, cpu(repeated(block, 1, 96)))).cuda()
    want = want.reshape(3, 49, c[1] + 1, c[0] + 1)[:, :48]
    assert check_repeats(crse, want, 1) < 1e-14
    # interpolation (added to the fine field)
    cb = rnd(3, 16, c[1] + 1, c[0] + 1)
    ci = torch.arange(c[2] + 1, device="cuda") % 16
    op.interpolation(0, fine, cb.index_select(1, ci).contiguous())
    want = O.interpolation(g, cpu(repeated(block, 1, 96)), cpu(cb.index_select(1, torch.arange(49, device="cuda") % 16)))
    want = torch.from_numpy(want).cuda().reshape(3, 97, n[1] + 1, n[0] + 1)[:, :96]
    assert check_repeats(fine, want, 1) < 1e-14
    op.close()


FAPPLY = """
import sys
sys.path[:0] = [%r, %r]
import numpy as np
import torch
import oracle as O
from alamo_gb300 import Constant, Elastic
from test_gpu_long_boxes import check_repeats, repeated
n, small = (4, 131104, 16), (4, 96, 16)
gen = torch.Generator(device="cuda").manual_seed(1)
u = torch.rand(3, 17, 32, 5, dtype=torch.float64, device="cuda", generator=gen) - 0.5
c = torch.rand(2, 17, 32, 5, dtype=torch.float64, device="cuda", generator=gen) + 0.5
op = Elastic(list(n), [0.1] * 3, "isotropic", max_coarsening_level=0)
op.SetBC(Constant())
op.SetModel(repeated(c, 2, n[1]), layout="soa")
f = torch.empty(3, 17, n[1] + 1, 5, dtype=torch.float64, device="cuda")
op.Fapply(0, repeated(u, 2, n[1]), f)
g = O.make_grid(small, dx=[0.1] * 3)
cs = repeated(c, 2, 96).permute(1, 2, 3, 0).contiguous().cpu().numpy().reshape(-1)
want = O.fapply(g, cs, repeated(u, 2, 96).cpu().numpy().reshape(-1))
want = torch.from_numpy(want).cuda().reshape(3, 17, 97, 5)[:, :, :96]
assert check_repeats(f, want, 2) < 1e-12
"""


def test_rows_of_a_long_box(gpu_lib):
    """In a process whose column kernel takes boxes from 4 cells in x on."""
    env = dict(os.environ, AGB_MARCH_MIN_CELLS="4", PYTHONPATH=ROOT)
    src = FAPPLY % (os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests"))
    subprocess.run([sys.executable, "-c", src], check=True, timeout=300, cwd=ROOT, env=env)
