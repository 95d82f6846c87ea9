"""GPU: weight and bias gradients of the 3x3x3 convolutions against FP64 sums,
at the edges of the tensor-core kernel: one voxel, line tiles of 16 voxels
more or less one, two tiles of a line, a remainder of the four lines of a
batch, one plane, every channel block, channel slices; and the scalar kernel
that slices without 16-byte alignment take.

Bar: an accumulator sums at most 32 tensor-core steps (4 lines of 128 voxels, 16
a step), each off by at most 2^-23 of the running sum (truncation), and at most
a few hundred of these are added in FP32: below 1e-5 of the largest gradient."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (15, 3, 2), (16, 4, 3), (17, 9, 5), (65, 6, 4), (127, 5, 1), (129, 2, 3), (257, 3, 2), (33, 33, 33)]
CHANNELS = [(16, 16), (32, 32), (48, 16), (96, 32), (32, 64), (64, 64), (16, 48)]


def reference(g, x, dy):
    import torch
    nx, ny, nz = g
    xp = torch.nn.functional.pad(x.double().reshape(nz, ny, nx, -1), (0, 0, 1, 1, 1, 1, 1, 1))
    d = dy.double()
    rows = []
    for t in range(27):
        dz, dyy, dx = t // 9, t // 3 % 3, t % 3
        rows.append(d.T @ xp[dz:dz + nz, dyy:dyy + ny, dx:dx + nx].reshape(nx * ny * nz, -1))
    return torch.stack(rows), d.sum(0)


def run(g, cin, cout, x_pad, dy_pad):
    """Slices of buffers with x_pad (dy_pad) channels before and 8 after them."""
    import torch
    from alamo_gb300._lib import check, lib
    V = g[0] * g[1] * g[2]
    gen = torch.Generator(device="cuda").manual_seed(V + cin + cout)
    x = torch.randn(V, x_pad + cin + 8, device="cuda", generator=gen).to(torch.bfloat16)
    dy = torch.randn(V, dy_pad + cout + 8, device="cuda", generator=gen).to(torch.bfloat16)
    dw0 = torch.randn(27, cout, cin, device="cuda", generator=gen)
    db0 = torch.randn(cout, device="cuda", generator=gen)
    dw, db = dw0.clone(), db0.clone()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    check(lib().agb_conv3_wgrad0((ctypes.c_int * 3)(*g), cin, cout, p(x), x.shape[1], x_pad, p(dy), dy.shape[1], dy_pad,
                                 p(dw), p(db), None))
    torch.cuda.synchronize()
    flag = ctypes.c_int()
    check(lib().agb_conv3_tc_error(ctypes.byref(flag)))
    assert flag.value == 0
    rw, rb = reference(g, x[:, x_pad:x_pad + cin], dy[:, dy_pad:dy_pad + cout])
    assert float((dw.double() - dw0.double() - rw).abs().max() / rw.abs().max().clamp(min=1)) < 1e-5
    assert float((db.double() - db0.double() - rb).abs().max() / rb.abs().max().clamp(min=1)) < 1e-5


@pytest.mark.parametrize("g", GRIDS)
@pytest.mark.parametrize("cin,cout", CHANNELS)
def test_wgrad_matches_fp64(gpu_lib, g, cin, cout):
    run(g, cin, cout, 8, 16)


@pytest.mark.parametrize("pads", [(4, 8), (8, 3), (0, 0)])
def test_wgrad_slices(gpu_lib, pads):
    run((18, 5, 6), 32, 16, *pads)
