"""GPU: the coarsest solve of FP32 cycles above the 128 unknowns of the dense
level is FP64 arithmetic, rounded once.

Without smoothing a V-cycle is x = P A_c^-1 R r, and P copies the coarse values to
the fine nodes with even indices, so one cycle of a mixed solve shows the
coarsest solve itself.  Moduli, cell sizes and the right-hand side (small
integers over a power of two) make the coarse operator and R r exact in 24 bits.
The bar: half a unit of FP32 of each value, and FP64's 1.1e-16 times the condition
number in the maximum norm (numpy's inverse has the same error, hence twice).  A
product in FP32 is off by 6e-8 of the sum of the terms' magnitudes, which
exceed the value of a slender box's row many times over."""
import numpy as np
import pytest

import oracle as O
from helpers import FACES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(6, 6, 6), (6, 6, 24), (8, 8, 36), (14, 14, 14)])
def test_bottom_of_fp32_cycles(gpu_lib, n):
    from alamo_gb300 import Constant, Elastic, Linear
    bc = Constant()
    bc.type[:] = O.TRAC
    for f in [i for i, name in enumerate(FACES) if "zlo" in name]:
        bc.type[f] = O.DISP
    dx = [0.125] * 3
    op = Elastic(list(n), dx, "isotropic", max_coarsening_level=1)
    assert op.NumLevels() == 2
    op.SetBC(bc)
    N = op.nodes()
    op.SetModel(np.ones(2 * N))
    rhs = (np.random.default_rng(3).integers(-8, 9, size=3 * N) / 8.0)
    rhs[0] = 1.0   # the max norm, by which the cycle's right-hand side is scaled, is 1
    s = Linear(op, precision=1, max_fmg_iter=0, pre_smooth=0, post_smooth=0, inner_max_iter=1, max_refine=1)
    x = np.zeros(3 * N)
    s.solve(x, rhs, 1e-14, 0.0, raise_on_fail=False)
    s.Clear()
    op.close()

    c = [v // 2 for v in n]
    gc = O.make_grid(c, dx=[0.25] * 3, sym=O.ISO, bc_type=bc.type, bc_val=np.zeros((26, 3)))
    gf = O.make_grid(n, dx=dx, sym=O.ISO, bc_type=bc.type, bc_val=np.zeros((26, 3)))
    M = 3 * O.nodes(gc)
    assert 128 < M <= 1536
    A, e = np.empty((M, M)), np.zeros(M)
    for j in range(M):
        e[j] = 1.0
        A[:, j] = O.fapply(gc, np.ones(2 * M // 3), e)
        e[j] = 0.0
    r = O.restriction(gf, rhs)
    inv = np.linalg.inv(A)
    want = np.linalg.solve(A, r)
    got = x.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)[:, ::2, ::2, ::2].reshape(-1)
    cond = np.abs(A).sum(1).max() * np.abs(inv).sum(1).max()
    fp64 = 2 * 1.1e-16 * cond * np.abs(want).max()
    assert fp64 < 1e-8 * np.abs(want).max()   # the bar below is FP32's
    assert (np.abs(got - want) <= 2.0 ** -24 * np.abs(want) * 1.0001 + fp64).all()
