"""GPU: operators without the divergence field of general moduli, from the start
(AGB_DIV=0) or because a later allocation took its memory, and the fields that
uniform moduli do not need.  AGB_OP_BYTES_MAX, the most device memory an operator
may hold, stands in for a device that is full."""
import numpy as np
import pytest

import oracle as O
from helpers import random_bc, random_ddw, random_field, rel_err

pytestmark = pytest.mark.gpu

N = 48


def field_bytes(n, elem):
    """Bytes of the fields of every level (rows hold 36 nodes from each multiple of 32
    on and are a multiple of 8 long, planes together a multiple of 64)."""
    total = 0
    while True:
        row = (max(n + 1, 32 * ((n - 2) // 32) + 36) + 7) // 8 * 8
        total += 18 * elem * ((row * (n + 1) ** 2 + 63) // 64 * 64)
        if n % 2 or n // 2 < 2:
            return total
        n //= 2


def cubic(n, seed=1):
    from alamo_gb300 import microstructure as M
    one = M.cubic(1.68, 1.21, 0.75, M.quat_to_rot([1.0, 0.4, -0.2, 0.3]))
    return (one[None, :] * np.random.default_rng(seed).uniform(1.0, 1.1, size=((n + 1) ** 3, 1))).reshape(-1)


def make_op(n=N, model=True):
    from alamo_gb300 import Elastic, TensionTest
    op = Elastic([n] * 3, None, "majorminor")
    op.SetBC(TensionTest("uniaxial_stress", disp=0.01))
    if model:
        op.SetModel(cubic(n))
    return op


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("box", [([2, 2, 2], (0, 0, 0)), ([64, 17, 16], (0, 0, 0)), ([41, 20, 9], (0, 0, 0)),
                                 ([66, 18, 17], (0, 1, 0)), ([6, 4, 6], (1, 1, 1))])
@pytest.mark.parametrize("cube", [True, False])
def test_rows_without_the_field(gpu_lib, monkeypatch, box, cube):
    """The bars of the rows that read the field (1e-12, FP32 1e-5)."""
    from alamo_gb300 import Constant, Elastic
    monkeypatch.setenv("AGB_DIV", "0")
    n, per = box
    dx = [1.0 / max(n)] * 3 if cube else [1.0 / n[0], 0.7 / n[1], 1.3 / n[2]]
    bt, bv = random_bc(41, ("disp", "trac", "neumann"))
    g = O.make_grid(n, dx=dx, sym=O.MAJORMINOR, periodic=per, bc_type=bt, bc_val=bv)
    op = Elastic(n, dx, "majorminor", per)
    bc = Constant()
    bc.type[:] = bt
    bc.val[:] = bv
    op.SetBC(bc)
    ddw = random_ddw(n, O.MAJORMINOR, 42, per)
    op.SetModel(ddw)
    u, b = random_field(n, 43, per), random_field(n, 44, per)
    assert rel_err(op.Fapply(0, u), O.fapply(g, ddw, u)) < 1e-12
    assert rel_err(op.solutionResidual(0, u, b), O.residual(g, ddw, u, b)) < 1e-12
    d = O.diagonal(g, ddw)
    if np.abs(d).min() > 0:
        assert rel_err(op.Fsmooth(0, u.copy(), b), O.fsmooth(g, ddw, d, u, b)) < 1e-12
    f32 = op.Fapply(0, u.astype(np.float32)).astype(np.float64)
    ref = O.fapply(g, ddw.astype(np.float32).astype(np.float64), u.astype(np.float32).astype(np.float64))
    assert rel_err(f32, ref) < 1e-5
    op.close()


def solve(op, rhs, **kw):
    from alamo_gb300 import Linear
    s = Linear(op, **kw)
    x = np.zeros_like(rhs)
    s.solve(x, rhs, 1e-8, 0.0)
    return s, x


def least(monkeypatch, run):
    """The smallest AGB_OP_BYTES_MAX (to 64 KB) with which run() finds its memory."""
    from alamo_gb300 import AgbError
    lo, hi = 0, 4 << 30
    while hi - lo > 1 << 16:
        mid = (lo + hi) // 2
        monkeypatch.setenv("AGB_OP_BYTES_MAX", str(mid))
        try:
            run()
            hi = mid
        except AgbError as e:
            assert "AGB_NOMEM" in str(e)
            lo = mid
    return hi


@pytest.mark.parametrize("kw", [{"precision": 1, "krylov": 8}, {"precision": 0}])
def test_allocations_take_the_field(gpu_lib, monkeypatch, kw):
    """Limits that solves without the fields keep: they are kept, at the second solve
    from captured cycles, and when a second solver's vectors take the fields that the
    first one's captured cycles held.  All solutions have the residual asked for, so
    they agree to the condition of the system times 1e-8 (1e-6, as in the solve tests)."""
    rhs = make_op().BCInit(np.zeros(3 * (N + 1) ** 3))

    def solves(count):
        op = make_op()
        s, out = [], []
        for _ in range(count):
            q, x = solve(op, rhs, **kw)
            s.append(q)
            out.append(x)
        for q in s + s[::-1]:   # from captured cycles
            x = np.zeros_like(rhs)
            q.solve(x, rhs, 1e-8, 0.0)
            out.append(x)
        for q in s:
            q.Clear()
        op.close()
        return out

    ref = solves(1)[0]
    monkeypatch.setenv("AGB_DIV", "0")
    one, two = least(monkeypatch, lambda: solves(1)), least(monkeypatch, lambda: solves(2))
    monkeypatch.delenv("AGB_DIV")
    fields = field_bytes(N, 8) if kw["precision"] == 0 else field_bytes(N, 4) + 18 * 8 * 72 * 49 * 49
    told = gpu_lib.agb_last_error()
    # room for a part of the fields; for all of them until the second solver comes
    # (4 MB: the coarsest solve's inverse, less than a solver's vectors)
    for count, limit in ((1, one), (1, one + fields // 2), (2, max(two, one + fields) + (4 << 20))):
        monkeypatch.setenv("AGB_OP_BYTES_MAX", str(limit))
        for x in solves(count):
            assert rel_err(x, ref) < 1e-6
    assert gpu_lib.agb_last_error() == told   # calls that succeed leave no message


def test_no_memory_is_still_an_error(gpu_lib, monkeypatch):
    from alamo_gb300 import AgbError
    monkeypatch.setenv("AGB_OP_BYTES_MAX", str(1 << 20))
    with pytest.raises(AgbError) as e:
        make_op()
    assert "AGB_NOMEM" in str(e.value)


def test_uniform_moduli_need_no_field(gpu_lib):
    """No memory for it while the moduli are uniform, and the right rows before and
    after the switch, by hand and in a solver's captured cycles."""
    n, sizes = 64, {}
    for uniform in (True, False):
        before = used()
        op = make_op(n)
        op.SetUniform(uniform)
        op.prepareForSolve()
        sizes[uniform] = used() - before
        op.close()
    assert sizes[False] - sizes[True] > 18 * 8 * 65 ** 3 * 0.9

    n = 16
    one = cubic(n).reshape(-1, 21)[0]
    model = np.ascontiguousarray(np.tile(one, (n + 1) ** 3))
    op = make_op(n, model=False)
    g = O.make_grid([n] * 3, sym=O.MAJORMINOR, bc_type=op.bc.type, bc_val=op.bc.val)
    rhs = O.bc_init(g, np.zeros(3 * op.nodes()))
    u = random_field([n] * 3, 3)
    op.SetModel(cubic(n, 5))
    s, x = solve(op, rhs)   # captures cycles with the field of these moduli
    assert np.abs(O.residual(g, cubic(n, 5), x, rhs)).max() <= 1e-8 * np.abs(rhs).max() * 1.0001
    for uniform, ddw in ((True, model), (False, cubic(n, 6)), (True, model)):
        op.SetModel(ddw)
        op.SetUniform(uniform)
        assert rel_err(op.Fapply(0, u), O.fapply(g, ddw, u)) < 1e-12
        x = np.zeros_like(rhs)
        s.solve(x, rhs, 1e-8, 0.0)
        assert np.abs(O.residual(g, ddw, x, rhs)).max() <= 1e-8 * np.abs(rhs).max() * 1.0001
    s.Clear()
    op.close()
