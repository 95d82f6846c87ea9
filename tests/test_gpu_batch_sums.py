"""GPU: the sums of the batched FP32 cycles do not lose bits with the size of the
batch: a thread adds at most the 16 elements of a segment in FP32, the rest in FP64 or
its equal.

The kernels are called through the library's own launchers, on one problem of
2000 segments shared by two CTAs, with all terms positive and their exact sum
from FP64.  Bar: a partial sum of 16 terms is off by at most 9 roundings of
2^-24 (products and adds), independent between the 512000 partial sums:
5.4e-7 / sqrt(512000) = 7.5e-10 of the total; four times that.  A sum in FP32
over all 16000 elements of a thread is off by some 1e-6, 4e-8 over 512 threads."""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

BSEG, NSEG, GRID, BAR = 4096, 2000, 2, 3e-9
vp = ctypes.c_void_p


class SegList(ctypes.Structure):
    _fields_ = [("d", vp), ("n", vp), ("max", ctypes.c_int)]


class Vecs(ctypes.Structure):
    _fields_ = [("v", vp * 16)]


def launcher(name, args):
    from alamo_gb300 import _lib
    out = subprocess.run(["nm", "-D", "--defined-only", _lib.LIB_PATH], capture_output=True, text=True).stdout
    names = [ln.split()[-1] for ln in out.splitlines() if name in ln]
    assert len(names) == 1, names
    f = getattr(_lib.lib(), names[0])
    f.restype, f.argtypes = None, args
    return f


@pytest.fixture(scope="module")
def problem(gpu_lib):
    import numpy as np
    import torch
    n = BSEG * NSEG
    seg = np.zeros(NSEG, dtype=[("base", "i8"), ("count", "i4"), ("prob", "i4"), ("comp", "i4"), ("first", "i4"),
                                ("pitch", "i4"), ("row", "i4")])
    seg["base"] = seg["first"] = BSEG * np.arange(NSEG)
    seg["count"] = seg["pitch"] = seg["row"] = BSEG
    d = torch.from_numpy(seg.view(np.uint8)).cuda()
    cnt = torch.tensor([NSEG], dtype=torch.int32, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(1)
    a = [0.5 + torch.rand(n, device="cuda", generator=gen) for _ in range(4)]
    return {"list": SegList(d.data_ptr(), cnt.data_ptr(), NSEG), "keep": (d, cnt), "a": a}


def close(got, want):
    return abs(float(got) - float(want)) <= BAR * abs(float(want))


def test_component_sums(problem):
    import torch
    y = problem["a"][0]
    sums = torch.zeros(3, dtype=torch.float64, device="cuda")
    f = launcher("launch_batch_mean3If", [vp, ctypes.c_int, vp, SegList, vp, vp, vp, ctypes.c_int, vp])
    torch.cuda.synchronize()
    f(None, GRID, None, problem["list"], None, y.data_ptr(), sums.data_ptr(), 0, None)
    torch.cuda.synchronize()
    assert close(sums[0], y.double().sum())


@pytest.mark.parametrize("k", [1, 3])
def test_inner_products(problem, k):
    import torch
    x, d = problem["a"][0], problem["a"][1]
    v = problem["a"][1:1 + k]
    out = torch.zeros(16, dtype=torch.float64, device="cuda")
    vecs = Vecs((vp * 16)(*[t.data_ptr() for t in v]))
    f = launcher("launch_batch_multidot", [vp, ctypes.c_int, SegList, vp, ctypes.c_int, vp, ctypes.POINTER(Vecs), vp,
                                           vp, ctypes.c_int])
    torch.cuda.synchronize()
    f(None, GRID, problem["list"], None, k, x.data_ptr(), ctypes.byref(vecs), d.data_ptr(), out.data_ptr(), 16)
    torch.cuda.synchronize()
    for i in range(k):
        assert close(out[i], (x.double() * d.double() ** 2 * v[i].double()).sum()), i


def test_new_direction(problem):
    import torch
    w, r, d = problem["a"][:3]
    dots = torch.zeros(2, dtype=torch.float64, device="cuda")
    none = Vecs()
    ref = ctypes.POINTER(Vecs)
    f = launcher("launch_batch_gcr_orth", [vp, ctypes.c_int, SegList, vp, ctypes.c_int, vp, ctypes.c_int, vp,
                                           ctypes.c_int, ref, ref, vp, vp, vp, vp, vp])
    torch.cuda.synchronize()
    f(None, GRID, problem["list"], None, 0, None, 16, None, 1, ctypes.byref(none), ctypes.byref(none), w.data_ptr(), None,
      r.data_ptr(), d.data_ptr(), dots.data_ptr())
    torch.cuda.synchronize()
    u = w.double() * d.double() ** 2
    assert close(dots[0], (u * w.double()).sum()) and close(dots[1], (u * r.double()).sum())
