"""GPU: stress, strain and energy written into device buffers that overlap the
displacement they are computed from: u at the start of the output, in its
middle, at its end and astride its last value.  The expected fields are the same calls'
into separate buffers; the arithmetic of a node is the same either way, so they
agree bit for bit.  The box has more nodes than blocks in flight, so that a
block's writes would reach nodes that later blocks still read."""
import ctypes

import numpy as np
import pytest

import oracle as O
from helpers import random_ddw, random_field

pytestmark = pytest.mark.gpu

N_CELLS = [95, 79, 63]


@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
@pytest.mark.parametrize("per", [(0, 0, 0), (0, 1, 0)])
def test_outputs_overlapping_u(gpu_lib, sym, per):
    import torch
    from alamo_gb300 import Constant, Elastic
    from alamo_gb300._lib import check, lib
    n = [N_CELLS[0], 80 if per[1] else N_CELLS[1], N_CELLS[2]]
    op = Elastic(n, [0.1, 0.07, 0.13], "isotropic" if sym == O.ISO else "majorminor", per)
    op.SetBC(Constant())
    op.SetModel(random_ddw(n, sym, 3, per))
    N = op.nodes()
    u = torch.from_numpy(random_field(n, 4, per)).cuda()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    ref = {k: torch.zeros(m * N, dtype=torch.float64, device="cuda") for k, m in (("s", 9), ("e", 9), ("w", 1))}
    check(lib().agb_stress(op.h, None, p(u), p(ref["s"]), 1))
    check(lib().agb_strain_energy(op.h, p(u), p(ref["e"]), p(ref["w"]), 1))
    buf = torch.zeros(12 * N, dtype=torch.float64, device="cuda")
    for at in (0, 3 * N, 6 * N, 9 * N - 1):   # u inside buf; the 9 N outputs from 0
        buf[at:at + 3 * N] = u
        check(lib().agb_stress(op.h, None, p(buf[at:]), p(buf), 1))
        assert torch.equal(buf[:9 * N], ref["s"]), at
        buf[at:at + 3 * N] = u
        check(lib().agb_strain_energy(op.h, p(buf[at:]), p(buf), None, 1))
        assert torch.equal(buf[:9 * N], ref["e"]), at
    for at in (0, N, 2 * N, 3 * N - 1):       # the N energies inside u
        buf[:3 * N] = u
        check(lib().agb_strain_energy(op.h, p(buf), None, p(buf[at:]), 1))
        assert torch.equal(buf[at:at + N], ref["w"]), at
    assert np.isfinite(ref["w"].cpu().numpy()).all()
    op.close()
