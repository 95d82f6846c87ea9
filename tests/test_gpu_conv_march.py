"""GPU: the convolution that marches by planes against FP64 sums: one voxel, one
plane, rows whose flat tiles of 128 end inside and at the end of a line, several
runs of planes, every block of output channels, slices, FP32 and BF16 output;
and the shapes the line kernel keeps (few lines, more than 96 input channels, long
rows).

Bars: an output sums 27 cin / 16 tensor-core steps (162 at most here; 216 in the
line kernel's case), each off by at most 2^-23 of the running sum
(truncation): below 2.6e-5 of the largest output; BF16 output rounds to 2^-8."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# the first nine march; the others are the line kernel's
SHAPES = [((1, 20, 20), 16, 16), ((5, 31, 11), 32, 64), ((126, 21, 16), 16, 48), ((33, 20, 20), 96, 32),
          ((65, 31, 12), 32, 32), ((129, 17, 10), 48, 16), ((14, 64, 40), 16, 64), ((257, 11, 10), 32, 48),
          ((30, 16, 70), 64, 64), ((1, 1, 1), 16, 16), ((17, 17, 17), 64, 64), ((700, 3, 2), 16, 16),
          ((20, 26, 15), 128, 16)]


@pytest.mark.parametrize("n,cin,cout", SHAPES)
@pytest.mark.parametrize("out_f32,relu,pad", [(True, False, 0), (False, True, 8)])
def test_conv_march_matches_fp64(gpu_lib, n, cin, cout, out_f32, relu, pad):
    import torch
    from alamo_gb300._lib import check, lib
    L = lib()
    nx, ny, nz = n
    V = nx * ny * nz
    g = torch.Generator(device="cuda").manual_seed(V + cin)
    x = torch.randn(V, pad + cin + pad, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", generator=g)
    out = torch.full((V, pad + cout + pad), 7.0, device="cuda", dtype=torch.float32 if out_f32 else torch.bfloat16)
    wp = torch.empty(27 * cout * cin, dtype=torch.bfloat16, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    check(L.agb_conv3_tc_pack(cin, cout, p(w), cout, 0, p(wp), None))
    for _ in range(2):
        check(L.agb_conv3_tc((ctypes.c_int * 3)(*n), cin, cout, p(x), x.shape[1], pad, p(wp), p(b), p(out),
                             out.shape[1], pad, int(out_f32), int(relu), None))
    torch.cuda.synchronize()
    flag = ctypes.c_int()
    check(L.agb_conv3_tc_error(ctypes.byref(flag)))
    assert flag.value == 0
    xp = torch.nn.functional.pad(x[:, pad:pad + cin].double().reshape(nz, ny, nx, cin), (0, 0, 1, 1, 1, 1, 1, 1))
    ref = b.double()
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        ref = ref + xp[dz:dz + nz, dy:dy + ny, dx:dx + nx] @ w[t].double().T
    ref = (torch.relu(ref) if relu else ref).reshape(V, cout)
    err = float((out[:, pad:pad + cout].double() - ref).abs().max() / ref.abs().max())
    assert err < (2.6e-5 if out_f32 else 2.0 ** -8)
    assert bool((out[:, :pad] == 7).all()) and bool((out[:, pad + cout:] == 7).all())
