"""Which arguments are taken as device tensors and which as host arrays
(focusing._ptr, focusing._stream), without a GPU."""
import sys
import types

import numpy as np
import pytest
import torch

from uncc_sar_focusing_b200 import _native as N
from uncc_sar_focusing_b200 import focusing


class HostTensor(torch.Tensor):
    """A tensor type of another package (an image toolkit's, say)."""


def test_numpy_arrays_do_not_need_torch(monkeypatch):
    """Another thread may be in the middle of `import torch`: the module is
    there, its names are not."""
    monkeypatch.setitem(sys.modules, "torch", types.ModuleType("torch"))
    a = np.arange(4.0)
    ptr, memory, keep = focusing._ptr(a, np.float64, 4)
    assert (ptr, memory) == (a.ctypes.data, N.MEMORY_HOST) and keep is a
    assert not focusing._is_torch(a)
    assert not focusing._stream(a, None)


def test_host_tensor_of_another_package_is_an_array():
    t = torch.arange(4, dtype=torch.float64).as_subclass(HostTensor)
    ptr, memory, _ = focusing._ptr(t, np.float64, 4)
    assert (ptr, memory) == (t.data_ptr(), N.MEMORY_HOST)


def test_torch_tensors_must_be_on_a_device():
    with pytest.raises(ValueError, match="CUDA device"):
        focusing._ptr(torch.zeros(4, dtype=torch.float64), np.float64)
    with pytest.raises(ValueError, match="CUDA device"):
        focusing._ptr(torch.nn.Parameter(torch.zeros(4, dtype=torch.float64)), np.float64)
