"""How a workspace takes its device memory."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _allocation_of(ptr):
    """(base, bytes) of the device allocation that holds ptr."""
    base, size = ctypes.c_uint64(), ctypes.c_size_t()
    assert ctypes.CDLL("libcuda.so.1").cuMemGetAddressRange_v2(ctypes.byref(base), ctypes.byref(size),
                                                                ctypes.c_uint64(ptr)) == 0
    return base.value, size.value


@pytest.mark.parametrize("n,b,form", [(64, 64, 0), (1024, 128, 1), (4096, 256, 2)])
def test_one_allocation(mxp, torch_cuda, n, b, form):
    """Creation costs one device allocation, however many buffers there are."""
    ws = mxp.Workspace(n, b, form)
    views = [ws.panel_view(side) for side in (0, 1)]
    ptrs = [v[k] for v in views for k in ("data", "scales") if v[k]]
    got = {_allocation_of(p) for p in ptrs}
    assert len(ptrs) >= 2 and len(got) == 1
    # the estimate a caller plans with holds the whole (buffers start on 256-byte boundaries)
    assert got.pop()[1] <= mxp.Workspace.bytes(n, b, form) + (2 << 20) + 32 * 256
    ws.close()
