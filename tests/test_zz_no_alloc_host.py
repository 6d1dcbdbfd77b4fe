"""Host time of cfft_fft_twopass_noalloc: a second call for a length must not
search for its split again (87 divisor pairs at 30240, few at 2^20)."""
import ctypes
import time

import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


def test_repeated_calls_do_not_search_again():
    import torch
    cb = load()

    def best(n, calls=40):
        x = torch.zeros(1, n, dtype=torch.complex128, device="cuda")
        p = ctypes.c_void_p(x.data_ptr())
        t = []
        for _ in range(calls):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            rc = cb._lib.LIB.cfft_fft_twopass_noalloc(n, 1, cb.C128, p, p, 0, None)
            t.append(time.perf_counter() - t0)
            cb.check(rc)
        torch.cuda.synchronize()
        return min(t)

    # the same three launches: within a factor of three of each other (with a
    # search per call the first took eight times the second)
    few = best(1 << 20)
    many = best(30240)
    assert many < 3 * few, (many, few)


@pytest.mark.parametrize("code,dtype,bar", [(0, "complex128", 1e-12), (1, "complex64", 2e-6)])
def test_many_lengths_in_turn(code, dtype, bar):
    # more lengths than the table keeps, both types, twice over: the split used
    # is always the length's own
    import numpy as np
    import torch
    cb = load()
    assert (cb.C128, cb.C64) == (0, 1)
    lengths = [n for n in range(600, 6000) if _smooth(n)][::3]
    assert len(lengths) > 40
    for n in lengths + lengths[:8]:
        x = torch.randn(2, n, dtype=getattr(torch, dtype), device="cuda")
        y = torch.empty_like(x)
        cb.check(cb._lib.LIB.cfft_fft_twopass_noalloc(n, 2, code, ctypes.c_void_p(x.data_ptr()),
                                                      ctypes.c_void_p(y.data_ptr()), 0, None))
        torch.cuda.synchronize()
        ref = np.fft.fft(x.cpu().numpy().astype(np.complex128))
        assert np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref) < bar, n


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1
