"""GPU: stress, strain, energy and traction computed in place in device memory
(caller layout, periodic images) against the oracle: boxes whose node count is
below, at and above the 128 nodes of a block, with and without an eigenstrain.
FP64 sums of at most 9 + 18 products: 1e-12 as for the other FP64 fields."""
import ctypes

import numpy as np
import pytest

import oracle as O
from helpers import random_ddw, random_field, rel_err

pytestmark = pytest.mark.gpu

BOXES = [([2, 2, 2], (0, 0, 0)), ([3, 3, 7], (0, 0, 0)), ([42, 2, 2], (0, 0, 0)), ([17, 20, 9], (0, 0, 0)),
         ([6, 8, 4], (0, 1, 1)), ([4, 6, 8], (0, 1, 0)), ([6, 4, 6], (1, 1, 1))]


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("sym", [O.ISO, O.MAJORMINOR])
@pytest.mark.parametrize("eig", [False, True])
def test_post_in_device_memory(gpu_lib, box, sym, eig):
    import torch
    from alamo_gb300 import Constant, Elastic
    from alamo_gb300._lib import check, lib
    n, per = box
    dx = [0.1, 0.07, 0.13]
    g = O.make_grid(n, dx=dx, sym=sym, periodic=per)
    op = Elastic(n, dx, "isotropic" if sym == O.ISO else "majorminor", per)
    op.SetBC(Constant())
    ddw = random_ddw(n, sym, 3, per)
    op.SetModel(ddw)
    u = random_field(n, 4, per)
    N = O.nodes(g)
    F0 = np.tile(np.array([1e-1, 2e-2, 0, 2e-2, -1e-1, 0, 0, 0, 5e-2]), N) if eig else None
    d = lambda a: None if a is None else torch.from_numpy(a).cuda()  # noqa: E731
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    ud, Fd = d(u), d(F0)
    out = {k: torch.full((m * N,), 7.0, dtype=torch.float64, device="cuda") for k, m in (("s", 9), ("e", 9), ("w", 1))}
    check(lib().agb_stress(op.h, p(Fd), p(ud), p(out["s"]), 1))
    check(lib().agb_strain_energy(op.h, p(ud), p(out["e"]), p(out["w"]), 1))
    assert rel_err(out["s"].cpu().numpy(), O.stress(g, ddw, F0, u)) < 1e-12
    eo, wo = O.strain_energy(g, ddw, u)
    assert rel_err(out["e"].cpu().numpy(), eo) < 1e-12
    assert rel_err(out["w"].cpu().numpy(), wo) < 1e-12
    if not per[0]:
        t = (ctypes.c_double * 3)()
        check(lib().agb_traction_xhi(op.h, p(Fd), p(ud), t, 1))
        assert np.abs(np.array(list(t)) - O.traction_xhi(g, ddw, F0, u)).max() < 1e-12 * np.abs(
            O.stress(g, ddw, F0, u)).max()
    op.close()
