"""Plans of HBM passes are cached by shape: what their scratch takes beyond 64 MB
each is bounded for all of them together, and given back."""
import ctypes

import pytest

from _pkg import load

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_scratch_of_many_plans_is_bounded():
    import torch
    cb = load()
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    cb.empty_cache()
    n, batches = 10 ** 6, list(range(130, 140))      # 512 MB of scratch each on its own

    def plan(batch):
        h = vp()
        cb.check(lib.cfft_plan_create(ctypes.byref(h), n, batch, cb.C64, cb.NO_FLAG))
        return h

    plans = [plan(b) for b in batches]
    held = [lib.cfft_plan_workspace_bytes(h) for h in plans]
    assert held[0] > 256 * MB                          # the first ones are not cut
    assert sum(max(0, x - 64 * MB) for x in held) <= 2048 * MB, held
    assert held[-1] <= 64 * MB
    # a plan with small chunks gives the same result
    x = torch.randn(batches[-1], n, dtype=torch.complex64, device="cuda")
    y = torch.empty_like(x)
    cb.check(lib.cfft_execute(plans[-1], vp(x.data_ptr()), vp(y.data_ptr()), 0, vp(0)))
    torch.cuda.synchronize()
    for h in plans:
        lib.cfft_plan_destroy(h)
    h = plan(batches[-1])                              # what was destroyed counts no more
    assert lib.cfft_plan_workspace_bytes(h) > 256 * MB
    z = torch.empty_like(x)
    cb.check(lib.cfft_execute(h, vp(x.data_ptr()), vp(z.data_ptr()), 0, vp(0)))
    torch.cuda.synchronize()
    lib.cfft_plan_destroy(h)
    assert torch.equal(y, z)
