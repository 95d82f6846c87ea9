"""GPU: the exact coarsest solve at the sizes where its paths change: the
largest dense level (128 unknowns at most: 3 x 4 x 3 nodes), the smallest one
of the panel elimination, remainders of its eight columns and its tiles of 32,
the two-row panel kernel (above 1024 unknowns), its largest level (1536) and
the first above it, which keeps BiCGStab.  Each solve is checked by the
oracle's residual and against the oracle's solve: both stop at 1e-10 of the
same residual norm, and the displacement follows the residual by the
operator's condition in that norm, about 1 (1e-8 bar)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_err, tension_bc_arrays

pytestmark = pytest.mark.gpu

# cells of the box: one coarsening to half of it; nodes of the coarse level
BOXES = [(4, 6, 4), (6, 6, 6), (14, 10, 6), (10, 10, 18), (14, 14, 14), (14, 14, 18)]


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
@pytest.mark.parametrize("mixed", [False, True])
def test_exact_bottom_solves(gpu_lib, n, sym, mixed):
    from alamo_gb300 import Elastic, Linear, TensionTest
    dx = [1.0 / max(n)] * 3
    bt, bv = tension_bc_arrays(0.01)
    g = O.make_grid(n, dx=dx, sym=sym, bc_type=bt, bc_val=bv)
    N = O.nodes(g)
    r = np.random.default_rng(5)
    if sym == O.ISO:
        ddw = r.uniform(1.0, 1.3, size=2 * N)
    else:
        from alamo_gb300 import microstructure as M
        one = M.cubic(1.68, 1.21, 0.75, M.quat_to_rot([1.0, 0.4, -0.2, 0.3]))
        ddw = (one[None, :] * r.uniform(1.0, 1.1, size=(N, 1))).reshape(-1)
    rhs = O.bc_init(g, np.zeros(3 * N))
    xo, _ = O.solve(g, ddw, rhs, tol_rel=1e-10, tol_abs=0.0)
    op = Elastic(list(n), dx, "isotropic" if sym == O.ISO else "majorminor")
    assert op.NumLevels() == 2
    op.SetBC(TensionTest("uniaxial_stress", disp=0.01))
    op.SetModel(ddw)
    s = Linear(op, precision=1, krylov=8) if mixed else Linear(op)
    for _ in range(2):   # the second solve replays the captured cycles
        x = np.zeros_like(rhs)
        s.solve(x, rhs, 1e-10, 0.0)
        assert np.abs(O.residual(g, ddw, x, rhs)).max() <= 1e-10 * np.abs(rhs).max() * 1.0000001
        assert rel_err(x, xo) < 1e-8
    s.Clear()
    op.close()
