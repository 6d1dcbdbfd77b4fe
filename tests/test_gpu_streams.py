"""Calls on several streams at once: a cached plan with scratch (the HBM passes,
odd real lengths, register kernels' ComplexF16 and strided plans) is not shared
between them, and a stream under capture allocates nothing."""
import ctypes

import numpy as np
import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


def _both(n, batch, f, torch, dtype, real=False):
    """f on four streams at once, several times over, equals f alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    xs = [torch.randn(batch, n, dtype=dtype, device="cuda", generator=g) for _ in range(4)]
    refs = [f(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    outs = [[] for _ in xs]
    for _ in range(6):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[i].append(f(xs[i]))
    torch.cuda.synchronize()
    for ref, out in zip(refs, outs):
        for y in out:
            assert torch.equal(y, ref)


@pytest.mark.parametrize("n,batch", [(48000, 24), (59049, 4), (1 << 16, 32), (100003, 6), (4096, 64), (30240, 4)])
def test_complex_on_four_streams(n, batch):
    import torch
    cb = load()
    _both(n, batch, cb.fft, torch, torch.complex128)
    p = cb.plan_fft(torch.zeros(batch, n, dtype=torch.complex128, device="cuda"))
    _both(n, batch, lambda x: p * x, torch, torch.complex128)


@pytest.mark.parametrize("n", [96000, 16807, 1000])
def test_real_on_four_streams(n):
    import torch
    cb = load()
    _both(n, 16, lambda x: cb.irfft(cb.rfft(x), n), torch, torch.float64)


def test_strided_on_four_streams():
    import torch
    cb = load()
    _both(300, 48000, lambda x: cb.fft(x.reshape(48000, 300), axis=0), torch, torch.complex64)
    _both(40, 8192, lambda x: cb.fft(x.reshape(8192, 40), axis=0), torch, torch.complex64)


@pytest.mark.parametrize("n", [48000, 4096, 100003])
def test_capture_on_another_stream(n):
    # planned and warmed up on one stream, captured on another
    import torch
    cb = load()
    x = torch.randn(5, n, dtype=torch.complex128, device="cuda")
    ref = cb.fft(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = cb.fft(x)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


def test_one_shot_entry_on_four_streams():
    import torch
    cb = load()
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    n, batch = 48000, 16
    xs = [torch.randn(batch, n, dtype=torch.complex128, device="cuda") for _ in range(4)]
    ys = [torch.empty_like(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(6):
        for x, y, s in zip(xs, ys, streams):
            cb.check(lib.cfft_fft(n, batch, cb.C128, 0, vp(x.data_ptr()), vp(y.data_ptr()), 0, vp(s.cuda_stream)))
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        ref = np.fft.fft(x.cpu().numpy())
        assert np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-12
