"""In place (input and output the same buffer, as the host entry runs every
chunk) equals out of place bit for bit for primes on the cluster Rader kernel:
its CTAs add x[0], which one of them overwrites with y[0], at different times."""
import ctypes

import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [4099, 7001, 10007, 12007, 16001])      # clusters of 3, 4, 5, 7 and 8 CTAs
def test_rader_clusters(n, dtype):
    import torch
    cb = load()
    batch = 700
    x = torch.randn(batch, n, dtype=getattr(torch, dtype), device="cuda")
    assert "cluster(C=" in cb.plan_fft(x).describe()
    for f, d in ((cb.fft, cb.FORWARD), (cb.ifft, cb.INVERSE)):
        y = f(x)
        for _ in range(3):
            z = x.clone()
            cb._run(z, d, out=z)
            torch.cuda.synchronize()
            assert torch.equal(z, y)
    h = x.cpu().pin_memory()
    out = torch.empty_like(h).pin_memory()
    plan = cb._get_plan(n, batch, cb.C128 if dtype == "complex128" else cb.C64, cb.NO_FLAG, 0)
    cb.check(cb._lib.LIB.cfft_execute_host(plan.handle, ctypes.c_void_p(h.data_ptr()),
                                           ctypes.c_void_p(out.data_ptr()), cb.FORWARD))
    assert torch.equal(out, cb.fft(x).cpu())
