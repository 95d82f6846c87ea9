"""GPU: which coarsest solve the cycles take does not depend on the units of the
moduli and the box, and an operator without an inverse still gets BiCGStab.

The limit on BiCGStab's iterations tells the two apart: with it at 1 or 200 a
cycle on the exact product is the same bit for bit (on these boxes no sum
depends on the order of blocks), one on BiCGStab is not.  Levels of 81 unknowns
(one-CTA inversion) and of 192 and 1536 (panels)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_err

pytestmark = pytest.mark.gpu

BOXES = [(4, 4, 4), (6, 6, 6), (14, 14, 14)]   # cells; one coarsening to half of it


def run(op, rhs, mixed, limit, **kw):
    from alamo_gb300 import AgbError, Linear
    s = Linear(op, precision=mixed, bottom_max_iter=limit, **kw)
    x = np.zeros_like(rhs)
    try:
        s.solve(x, rhs, 1e-8, 0.0)
    except AgbError as e:
        assert "AGB_MAXITER" in str(e) or "AGB_STALL" in str(e)
    n = s.report.iterations
    s.Clear()
    return x, n


def moduli(sym, N, scale):
    r = np.random.default_rng(5)
    if sym == O.ISO:
        return scale * r.uniform(1.0, 1.3, size=2 * N)
    from alamo_gb300 import microstructure as M
    one = M.cubic(1.68, 1.21, 0.75, M.quat_to_rot([1.0, 0.4, -0.2, 0.3]))
    return scale * (one[None, :] * r.uniform(1.0, 1.1, size=(N, 1))).reshape(-1)


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("scale,edge", [(1.0, 1.0), (1e11, 1e-3), (1e-9, 1e3)])
def test_exact_solve_in_any_units(gpu_lib, n, sym, mixed, scale, edge):
    from alamo_gb300 import Constant, Elastic
    dx = [edge / max(n)] * 3
    g = O.make_grid(n, dx=dx, sym=sym, bc_type=np.full((26, 3), O.DISP, np.int32), bc_val=np.zeros((26, 3)))
    N = O.nodes(g)
    ddw = moduli(sym, N, scale)
    F0 = np.random.default_rng(6).uniform(-1e-3, 1e-3, size=9 * N)
    rhs = O.newton_rhs(g, ddw, F0, np.zeros(3 * N), np.zeros(3 * N))
    op = Elastic(list(n), dx, "isotropic" if sym == O.ISO else "majorminor")
    op.SetBC(Constant())
    op.SetModel(ddw)
    one, few = run(op, rhs, mixed, 200), run(op, rhs, mixed, 1)
    assert one[1] == few[1] and np.array_equal(one[0], few[0])
    # both stop at 1e-8 of the same residual norm; the displacement follows it
    xo, _ = O.solve(g, ddw, rhs, tol_rel=1e-8, tol_abs=0.0)
    assert rel_err(one[0], xo) < 1e-6
    op.close()


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
def test_singular_level_keeps_bicgstab(gpu_lib, monkeypatch, n, sym):
    """Tractions on every face: rigid motions make the level singular, its last
    pivots are rounding (5e-16 of the scaled rows and less), and the cycles are
    those of an operator that never makes the inverse."""
    from alamo_gb300 import Constant, Elastic
    dx = [1.0 / max(n)] * 3
    bc = Constant()
    bc.type[:] = O.TRAC
    got = []
    for exact in ("1", "0"):
        monkeypatch.setenv("AGB_BOTTOM_EXACT", exact)
        op = Elastic(list(n), dx, "isotropic" if sym == O.ISO else "majorminor")
        op.SetBC(bc)
        op.SetModel(moduli(sym, op.nodes(), 1.0))
        rhs = np.random.default_rng(8).uniform(-1, 1, size=3 * op.nodes())
        got.append(run(op, rhs, 0, 20, max_iter=4))
        op.close()
    assert got[0][1] == got[1][1] and np.array_equal(got[0][0], got[1][0], equal_nan=True)
