"""GPU: rows from the node's own moduli (k_rows, k_column) against the oracle
at the edges of their tiles: boxes just above and below the column kernel's
smallest, x extents of one tile more or less one node, odd y extents, k
extents that leave a remainder of the chunk, the smallest box, periodic
directions, cubic and other cells.

Bars: the row is a sum of at most 171 products of FP64 values, each formed from
differences of at most four displacements, so its rounding error is at most
about 200 units of 1.1e-16 of the sum of its terms' magnitudes; on uniformly
random fields that sum is below 30 times the largest entry: 1e-12 (the bar of
the other FP64 operator tests) covers it.  FP32: the same with 6e-8: 1e-5
covers the random error of such sums (sqrt(200) * 6e-8 * 10)."""
import numpy as np
import pytest

import oracle as O
from helpers import random_bc, random_ddw, random_field, rel_err

pytestmark = pytest.mark.gpu

BOXES = [([2, 2, 2], (0, 0, 0)), ([63, 17, 16], (0, 0, 0)), ([64, 17, 16], (0, 0, 0)), ([65, 16, 19], (0, 0, 0)),
         ([98, 19, 33], (0, 0, 0)), ([66, 18, 17], (0, 1, 0)), ([7, 5, 6], (1, 1, 0)), ([64, 16, 16], (1, 1, 1))]


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
@pytest.mark.parametrize("cube", [True, False])
def test_rows_match_oracle(gpu_lib, box, sym, cube):
    from alamo_gb300 import Constant, Elastic
    n, per = box
    dx = [1.0 / max(n)] * 3 if cube else [1.0 / n[0], 0.7 / n[1], 1.3 / n[2]]
    bt, bv = random_bc(41, ("disp", "trac", "neumann"))
    g = O.make_grid(n, dx=dx, sym=sym, periodic=per, bc_type=bt, bc_val=bv)
    op = Elastic(n, dx, "isotropic" if sym == O.ISO else "majorminor", per)
    bc = Constant()
    bc.type[:] = bt
    bc.val[:] = bv
    op.SetBC(bc)
    ddw = random_ddw(n, sym, 42, per)
    op.SetModel(ddw)
    u, b = random_field(n, 43, per), random_field(n, 44, per)
    ref = O.fapply(g, ddw, u)
    assert rel_err(op.Fapply(0, u), ref) < 1e-12
    assert rel_err(op.solutionResidual(0, u, b), O.residual(g, ddw, u, b)) < 1e-12
    d = O.diagonal(g, ddw)
    assert rel_err(op.Diagonal(0), d) < 1e-12
    if np.abs(d).min() > 0:
        assert rel_err(op.Fsmooth(0, u.copy(), b), O.fsmooth(g, ddw, d, u, b)) < 1e-12
    f32 = op.Fapply(0, u.astype(np.float32)).astype(np.float64)
    ref32 = O.fapply(g, ddw.astype(np.float32).astype(np.float64), u.astype(np.float32).astype(np.float64))
    assert rel_err(f32, ref32) < 1e-5
    op.SetUniform(True)
    g.uniform = 1
    assert rel_err(op.Fapply(0, u), O.fapply(g, ddw, u)) < 1e-12
    op.close()


@pytest.mark.parametrize("n,sym", [([100, 61, 60], O.MAJORMINOR), ([130, 101, 95], O.ISO)])
@pytest.mark.parametrize("uniform", [False, True])
def test_fp32_tiled_boxes(gpu_lib, n, sym, uniform):
    """The smallest ragged boxes whose FP32 sweep exceeds half of the L2 and so
    goes to the tiled kernels; the FP32 bar of the other operator tests."""
    from alamo_gb300 import Constant, Elastic
    dx = [1 / 100, 1 / 61, 1 / 90]
    bt, bv = random_bc(51, ("disp",))
    g = O.make_grid(n, dx=dx, sym=sym, bc_type=bt, bc_val=bv)
    op = Elastic(n, dx, "isotropic" if sym == O.ISO else "majorminor")
    bc = Constant()
    bc.type[:] = bt
    bc.val[:] = bv
    op.SetBC(bc)
    ddw = random_ddw(n, sym, 52)
    op.SetModel(ddw)
    if uniform:
        op.SetUniform(True)
        g.uniform = 1
    d32 = ddw.astype(np.float32).astype(np.float64)
    u = random_field(n, 53, dtype=np.float32)
    b = random_field(n, 54, dtype=np.float32)
    assert rel_err(op.Fapply(0, u).astype(np.float64), O.fapply(g, d32, u.astype(np.float64))) < 1e-5
    x = op.Fsmooth(0, u.copy(), b).astype(np.float64)
    assert rel_err(x, O.fsmooth(g, d32, O.diagonal(g, d32), u.astype(np.float64), b.astype(np.float64))) < 1e-5
    op.close()
