"""GPU: field import and export by rows, and the masked update by eight channels.

A field that is imported and exported comes back unchanged on boxes whose rows are shorter than a warp, exactly a warp's
unrolled copy (256 nodes) and one node longer, with and without periodic
directions.  The masked update equals the same expression in FP32 rounded once
to BF16, bit for bit, on the eight-channel form and on slices that do not allow
it (offset or width no multiple of 8)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4, 6, 8), (32, 4, 4), (255, 3, 2), (256, 2, 5), (300, 4, 3)])
@pytest.mark.parametrize("periodic", [(0, 0, 0), (1, 0, 1), (1, 1, 1)])
def test_import_export_rows(gpu_lib, n, periodic):
    from alamo_gb300 import Constant, Elastic, _lib
    if any(p and k % 2 for p, k in zip(periodic, n)):
        n = tuple(k + k % 2 for k in n)
    op = Elastic(list(n), None, "isotropic", list(periodic), max_coarsening_level=0)
    rng = np.random.default_rng(3)
    m = rng.uniform(1.0, 2.0, (2, n[2] + 1, n[1] + 1, n[0] + 1))   # component planes
    if periodic[0]:
        m[..., -1] = m[..., 0]
    if periodic[1]:
        m[:, :, -1] = m[:, :, 0]
    if periodic[2]:
        m[:, -1] = m[:, 0]
    op.SetBC(Constant())
    op.SetModel(m.reshape(-1), layout="soa")
    out = np.zeros(m.size)
    _lib.check(_lib.lib().agb_op_get_model(op.h, 0, ctypes.c_void_p(out.ctypes.data), _lib.AGB_LAYOUT_SOA,
                                           _lib.AGB_MEM_HOST))
    assert np.array_equal(out, m.reshape(-1))
    aos = np.asarray(op.GetModel(0)).reshape(-1, 2)
    assert np.array_equal(aos, m.reshape(2, -1).T)
    op.close()


@pytest.mark.parametrize("C,cs,c0", [(8, 8, 0), (16, 48, 16), (24, 32, 8), (8, 24, 4), (12, 16, 0), (3, 3, 0)])
@pytest.mark.parametrize("has_b,has_m", [(True, True), (True, False), (False, True), (False, False)])
def test_axpby_mask(gpu_lib, C, cs, c0, has_b, has_m):
    torch = pytest.importorskip("torch")
    from alamo_gb300 import _lib
    V = 333
    gen = torch.Generator().manual_seed(C + cs)
    a, b, m, y = [torch.randn(V, cs, generator=gen).to(torch.bfloat16).cuda() for _ in range(4)]
    m[5, c0] = float("nan")
    m[6, c0] = 0.0
    keep = y.clone()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    s = slice(c0, c0 + C)
    beta = 0.75
    _lib.check(_lib.lib().agb_axpby_mask(V, C, p(y), cs, c0, p(a), cs, c0, p(b) if has_b else None, cs, c0, beta,
                                         p(m) if has_m else None, cs, c0, None))
    torch.cuda.synchronize()
    r = a[:, s].float()
    if has_b:   # 0.75 b is exact in FP32: one rounding, fused or not
        r = (r.double() + beta * b[:, s].double()).float()
    if has_m:
        r = torch.where(m[:, s].float() > 0, r, torch.zeros_like(r))
    keep[:, s] = r.to(torch.bfloat16)
    assert torch.equal(y, keep)
