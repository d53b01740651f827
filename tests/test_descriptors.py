"""The tensor descriptors handed to the C ABI."""
import ctypes

import pytest
import torch

from totri_gb300 import _lib


@pytest.mark.parametrize("t", [
    torch.zeros(()), torch.zeros(3, dtype=torch.int64), torch.zeros(2, 0, 3),
    torch.zeros(4, 5, 6).transpose(0, 2), torch.zeros(1, 2, 3, 4, 5, dtype=torch.float64),
    torch.zeros(2, 3).half(), torch.zeros(1, 1).expand(5, 7), torch.zeros(9, dtype=torch.int32)[::2]])
def test_descriptor_fields(t):
    a, n = _lib.array(t)._obj, t.dim()
    assert ctypes.sizeof(a) == 96
    assert (a.data or 0) == (t.data_ptr() if t.numel() else 0)
    assert a.ndim == n and a.dtype == _lib._DTYPES.get(t.dtype, -1)
    assert tuple(a.shape) == tuple(t.shape) + (0,) * (5 - n)
    assert tuple(a.strides) == t.stride() + (0,) * (5 - n)


def test_rank_limit():
    with pytest.raises(ValueError):
        _lib.array(torch.zeros((1,) * 6))
