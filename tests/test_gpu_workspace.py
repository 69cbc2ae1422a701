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


def test_memory_short_of_the_second_panel_copy(mxp, torch_cuda):
    """A workspace needs no second copy of the panel operands: where the device has room
    for all but that, it is created without, the U panel is cast into the L panel's
    buffer after the first product, and the factors are the same bits."""
    torch = torch_cuda
    n, b = 12288, 2048
    second = (n - b) * 3 * b * 2  # rows x split-BF16 operand, below the copy's own limit
    p = mxp.panel_matgen(n, 9)
    ws = mxp.Workspace(n, b, 0)
    mxp.panel_lu(p, b, ws)
    want = p.A.cpu()
    ws.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    room = mxp.Workspace.bytes(n, b, 0) - second // 2
    fill = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    ws = mxp.Workspace(n, b, 0)
    base, size = _allocation_of(ws.panel_view(0)["data"])
    assert size < mxp.Workspace.bytes(n, b, 0) - second // 2
    del fill
    torch.cuda.empty_cache()
    mxp.regenerate(p)
    mxp.panel_lu(p, b, ws)
    assert torch.equal(p.A.cpu(), want)
    ws.close()


@pytest.mark.parametrize("form,tol", [(0, 1e-6), (2, 1e-4)])
def test_panels_too_large_for_the_second_copy(mxp, torch_cuda, form, tol):
    """A first panel of 10752 x 3584 (231 MB as split BF16) against 192 MB of second copy: its
    U panel goes through the L panel's buffer, the later panels' through their own.
    Factors against a 64-bit elimination of the same matrix: the forms' own rounding
    of the panels, relative to the dominant diagonal, is 2e-7 (FP16) and 2e-5 (FP8)."""
    torch = torch_cuda
    n, b = 14336, 3584
    p = mxp.panel_matgen(n, 9)
    want, _ = torch.linalg.lu_factor(p.matrix().double(), pivot=False)
    ws = mxp.Workspace(n, b, form)
    mxp.panel_lu(p, b, ws)
    got = p.matrix().double()
    for part in (torch.tril, torch.triu):
        err = torch.linalg.norm(part(got) - part(want)) / torch.linalg.norm(want)
        assert float(err) < tol
    # the panels of the first step by themselves: the U strip, and the L strip (its
    # entries are smaller by the pivot)
    for sl in ((slice(0, b), slice(b, n)), (slice(b, n), slice(0, b))):
        assert float(torch.linalg.norm(got[sl] - want[sl]) / torch.linalg.norm(want[sl])) < 1e-4
    ws.close()
