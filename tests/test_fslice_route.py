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


# no room; a small plan, and those just past its lines (slices, slices times area, box)
@pytest.mark.parametrize("nx,nang,room,buffered", [(40, 300, True, True), (40, 300, False, False), (16, 256, True, False),
                                                   (16, 257, True, True), (64, 32, True, False), (64, 33, True, True),
                                                   (127, 1, True, False), (128, 1, True, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_normal_operator_route(monkeypatch, dtype, nx, nang, room, buffered):
    """With room for a slice buffer the normal operator of all but small plans goes
    through it; else the entry point that keeps no slices gets the same grid, lam and output."""
    plan = object.__new__(autograd.FourierSlicePlan)
    plan.nx, plan.nang = nx, nang
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
    if buffered:
        assert name == "spi_fslice_normal_ws" and a[4] == int(dtype == torch.float64) and a[6] == 4096
    else:
        assert name == ("spi_fslice_normal64" if dtype == torch.float64 else "spi_fslice_normal") and len(a) == 5
