"""The host entry's pipeline (cfft_execute_host) over a plan of HBM passes: its
ring of device buffers stays at three chunks of about 32 MB, whatever the
plan's own chunk, and its result is the device entry's bit for bit."""
import ctypes

import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("n,batch", [(10 ** 6, 24), (10 ** 6, 2), (999983, 9)])
def test_ring_is_three_small_chunks(n, batch, pinned):
    import torch
    cb = load()
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    x = torch.view_as_complex(torch.randn(batch, n, 2, dtype=torch.float32))
    y = torch.empty_like(x)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    h = vp()
    cb.check(lib.cfft_plan_create(ctypes.byref(h), n, batch, cb.C64, cb.NO_FLAG))
    xd = x.cuda()
    yd = torch.empty_like(xd)
    cb.check(lib.cfft_execute(h, vp(xd.data_ptr()), vp(yd.data_ptr()), cb.FORWARD, vp(0)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    cb.check(lib.cfft_execute_host(h, vp(x.data_ptr()), vp(y.data_ptr()), cb.FORWARD))
    ring = free - torch.cuda.mem_get_info()[0]
    one = n * 8
    chunk = max(1, (32 << 20) // one) * one
    # the three buffers, rounded up to 2 MB pages, and room for streams and events
    assert ring <= min(3, -(-batch * one // chunk)) * min(chunk, batch * one) + (16 << 20), ring
    assert torch.equal(y, yd.cpu())
    lib.cfft_plan_destroy(h)
