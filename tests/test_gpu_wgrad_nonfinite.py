"""GPU: a NaN or an infinity in the input reaches the weight gradients of the taps
that use it and no others, on lines that fill their last 16 voxels and lines
that end inside them (one tile of a line and several).  The finite entries keep
the bar of the other weight gradients, 1e-5 of the largest."""
import ctypes

import pytest

from test_gpu_wgrad_tc import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [(1, 2, 2), (15, 3, 2), (16, 4, 3), (17, 9, 5), (65, 6, 4), (128, 3, 2), (129, 2, 3),
                               (250, 3, 2)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 32), (32, 64)])
def test_nonfinite_inputs_stay_in_their_taps(gpu_lib, g, cin, cout):
    import torch
    from alamo_gb300._lib import check, lib
    nx, ny, nz = g
    gen = torch.Generator(device="cuda").manual_seed(nx + cout)
    x = torch.randn(nz, ny, nx, cin, device="cuda", generator=gen).to(torch.bfloat16)
    dy = torch.randn(nx * ny * nz, cout, device="cuda", generator=gen).to(torch.bfloat16)
    x[0, ny - 1, nx - 1, 3] = float("nan")
    x[nz - 1, 0, nx - 1, 5] = float("inf")
    x[0, 0, 0, 9] = float("-inf")
    x[nz - 1, ny - 1, 0, 12] = float("nan")
    x = x.reshape(-1, cin)
    dw = torch.zeros(27, cout, cin, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    check(lib().agb_conv3_wgrad0((ctypes.c_int * 3)(*g), cin, cout, p(x), cin, 0, p(dy), cout, 0, p(dw), None, None))
    torch.cuda.synchronize()
    ref, _ = reference(g, x, dy)
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(dw), fin)
    assert torch.equal(torch.isnan(dw), torch.isnan(ref))
    inf = torch.isinf(ref)
    assert torch.equal(dw[inf].sign().double(), ref[inf].sign())
    assert float((dw[fin].double() - ref[fin]).abs().max()) < 1e-5 * max(1.0, float(ref[fin].abs().max()))
