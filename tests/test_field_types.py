"""CPU: fields of another type than the call reads are refused on the host, as
numpy arrays always were: an FP32 tensor read as FP64 would be read past its end."""
import numpy as np
import pytest
import torch

from alamo_gb300.elastic import _ptr


@pytest.mark.parametrize("held,read", [("float32", "float64"), ("float64", "float32"), ("bfloat16", "float64"),
                                       ("int64", "float64"), ("complex64", "float64")])
def test_other_types_are_refused(held, read):
    with pytest.raises(TypeError):
        _ptr(torch.zeros(8, dtype=getattr(torch, held)), np.dtype(read))
    if held != "bfloat16":
        with pytest.raises(TypeError):
            _ptr(np.zeros(8, dtype=held), np.dtype(read))


@pytest.mark.parametrize("name", ["float32", "float64"])
def test_own_type_is_taken(name):
    t, a = torch.zeros(8, dtype=getattr(torch, name)), np.zeros(8, dtype=name)
    assert _ptr(t, np.dtype(name))[0].value == t.data_ptr() and _ptr(t, getattr(np, name))[1] == 0
    assert _ptr(a, np.dtype(name))[0].value == a.ctypes.data


def test_default_is_fp64():
    _ptr(torch.zeros(8, dtype=torch.float64))
    with pytest.raises(TypeError):
        _ptr(torch.zeros(8))
