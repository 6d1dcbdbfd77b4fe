"""Plans of convolutions made by several threads at once: the builds of their
spectra share a transform plan per length and a buffer, and must not mix."""
import ctypes
import threading

import numpy as np
import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


def test_convolutions_planned_by_threads_at_once():
    import torch
    cb = load()
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    # pairs of lengths whose convolutions have the same number of points, long
    # (three passes) and in one CTA
    groups = [[99990 + k for k in range(1, 17)], [2506, 2508, 2510, 2511, 2513, 2514, 2515, 2516]]
    groups = [[n for n in g if not _smooth(n)] for g in groups]
    for rep in range(3):
        cb.empty_cache()
        plans, errors = {}, []

        def make(n):
            # (the Python cache would plan one at a time)
            h = ctypes.c_void_p()
            if lib.cfft_plan_create(ctypes.byref(h), n, 1, cb.C128, cb.EXACT_TWIDDLES) != 0:
                errors.append(n)
            plans[n] = h

        threads = [threading.Thread(target=make, args=(n,)) for g in groups for n in g]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        for n, h in plans.items():
            x = torch.from_numpy(_signal(n)).cuda()
            y = torch.empty_like(x)
            cb.check(lib.cfft_execute(h, vp(x.data_ptr()), vp(y.data_ptr()), cb.FORWARD, vp(0)))
            torch.cuda.synchronize()
            lib.cfft_plan_destroy(h)
            ref = np.fft.fft(_signal(n))
            assert np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-12, n


def _signal(n):
    rng = np.random.default_rng(n)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1
