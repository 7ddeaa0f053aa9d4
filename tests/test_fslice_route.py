"""Which entry point FourierSlicePlan's normal operator takes, on the CPU: the
library and torch's allocator are stand-ins."""
import ctypes

import pytest
import torch

from spider_b200 import autograd


class _Lib:
    def __init__(self):
        self.calls = []

    def spi_fslice_normal_ws_bytes(self, h, fp64, out):
        ctypes.cast(out, ctypes.POINTER(ctypes.c_longlong))[0] = 4096
        return 0

    def __getattr__(self, name):
        return lambda *a: self.calls.append((name, a)) or 0


@pytest.mark.parametrize("room", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_normal_operator_route(monkeypatch, dtype, room):
    """With room for a slice buffer the normal operator goes through it; without,
    the entry point that keeps no slices gets the same grid, lam and output."""
    plan = object.__new__(autograd.FourierSlicePlan)
    plan._L, plan._h, plan.device = _Lib(), None, torch.device("cpu")
    monkeypatch.setattr(plan, "_stream", lambda: ctypes.c_void_p(7), raising=False)
    grid, out = torch.zeros(8, dtype=dtype), torch.zeros(8, dtype=dtype)
    if not room:
        def empty(*a, **k):
            raise torch.OutOfMemoryError("no room")
        monkeypatch.setattr(autograd.torch, "empty", empty)
    assert plan._normal(grid, 0.25, out) is out
    (name, a), = plan._L.calls
    assert (a[1].value, a[2], a[3].value) == (grid.data_ptr(), 0.25, out.data_ptr())
    assert a[-1].value == 7
    if room:
        assert name == "spi_fslice_normal_ws" and a[4] == int(dtype == torch.float64) and a[6] == 4096
    else:
        assert name == ("spi_fslice_normal64" if dtype == torch.float64 else "spi_fslice_normal") and len(a) == 5
