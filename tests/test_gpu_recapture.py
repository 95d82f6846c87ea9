"""GPU: a solver that has captured its cycles follows what is set on its operator
afterwards: other types of boundary conditions, another omega, other moduli.  The
expected solution is a new operator's, bit for bit (no sum of these cycles depends
on the order of blocks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 16


def conditions(kind):
    from alamo_gb300 import Constant, TensionTest
    if kind == "tension":
        return TensionTest("uniaxial_stress", disp=0.01)
    bc = Constant()
    bc.set_face("xhi", ["disp"] * 3, [0.01, 0.0, 0.0])
    return bc


def moduli(seed):
    return np.random.default_rng(seed).uniform(1.0, 1.3, size=2 * (N + 1) ** 3)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("graph", [0, 1])
def test_solver_follows_its_operator(gpu_lib, mixed, graph):
    from alamo_gb300 import Elastic, Linear

    def setup(op, kind, omega, seed):
        op.SetBC(conditions(kind))
        op.SetOmega(omega)
        op.SetModel(moduli(seed))

    def solve(op, s):
        rhs = op.BCInit(np.zeros(3 * (N + 1) ** 3))
        x = np.zeros_like(rhs)
        s.solve(x, rhs, 1e-8, 0.0)
        return x, s.report.iterations

    steps = [("tension", 2 / 3, 1), ("fixed", 2 / 3, 1), ("fixed", 0.5, 1), ("tension", 0.5, 2), ("tension", 0.6, 1)]
    op = Elastic([N] * 3, None, "isotropic")
    setup(op, *steps[0])
    s = Linear(op, precision=mixed, use_graph=graph)
    for step in steps:
        setup(op, *step)
        x, n = solve(op, s)
        fresh = Elastic([N] * 3, None, "isotropic")
        setup(fresh, *step)
        f = Linear(fresh, precision=mixed, use_graph=graph)
        y, m = solve(fresh, f)
        assert n == m and np.array_equal(x, y), step
        f.Clear(), fresh.close()
    s.Clear(), op.close()
