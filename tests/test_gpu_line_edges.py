"""The stage kernels of one CTA (csrc/passes.cuh) at their edges, against the
FP64 DFT: LINE and LCONV at their smallest and largest lengths, at the lengths
whose ComplexF32 sequence has the radices 18 and 20, with batches that leave a
partial CTA, in place; COLS with rows further apart than the batch and with
different strides on the two sides.

Bars: as in test_gpu_passes.py -- FP64 rounding of at most ~24 stages of ~4 eps
stays below 1e-13 (1e-12 is the library's bar); FP32 at ~4 x 6e-8 a stage over
at most 12 stages in quadrature is below 2e-6.  Convolution plans are made with
EXACT_TWIDDLES (the default Rader tables drift like the reference's)."""
import ctypes

import numpy as np
import pytest

from _pkg import load

pytestmark = pytest.mark.gpu
TOL = {"complex128": 1e-12, "complex64": 2e-6}
# LINE ends at 9000 (ComplexF32) and 6750 (ComplexF64), LCONV at M of those
LINE = {"complex64": [1, 2, 3, 7, 16, 20, 120, 324, 360, 400, 2160, 3840, 4536, 6000, 8000, 8820, 9000],
        "complex128": [1, 2, 3, 7, 16, 20, 120, 360, 2160, 3840, 6561, 6750]}
CONV = {"complex64": [11, 13, 22, 181, 509, 1022, 2003, 4001, 4093, 4498, 4499],
        "complex128": [11, 13, 22, 181, 509, 1022, 2503, 3202, 3374]}


@pytest.fixture(scope="module")
def cb():
    return load()


def _plan(cb, make):
    h = ctypes.c_void_p()
    cb.check(make(ctypes.byref(h)))
    buf = ctypes.create_string_buffer(256)
    cb._lib.LIB.cfft_plan_describe(h, buf, 256)
    return h, buf.value.decode()


def _err(got, ref):
    return float((np.linalg.norm(got - ref, axis=-1) / np.linalg.norm(ref, axis=-1)).max())


@pytest.mark.parametrize("dtype,n", [(d, n) for d in TOL for n in LINE[d] + CONV[d]])
def test_whole_transforms_in_a_cta(cb, dtype, n):
    import torch
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    code = cb.C128 if dtype == "complex128" else cb.C64
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for batch in (1, 3, 701, 2 + (1 << 21) // n // 8):
        h, desc = _plan(cb, lambda h: lib.cfft_plan_create(h, n, batch, code, cb.EXACT_TWIDDLES))
        assert "rows(V=" in desc or batch > 3, desc         # (many long convolutions take the passes)
        x = torch.randn(batch, n, dtype=getattr(torch, dtype), device="cuda", generator=g)
        xs = x.cpu().numpy().astype(np.complex128)
        for d, ref in ((cb.FORWARD, np.fft.fft(xs)), (cb.INVERSE, np.fft.ifft(xs))):
            y, z = torch.empty_like(x), x.clone()
            cb.check(lib.cfft_execute(h, vp(x.data_ptr()), vp(y.data_ptr()), d, vp(0)))
            cb.check(lib.cfft_execute(h, vp(z.data_ptr()), vp(z.data_ptr()), d, vp(0)))
            torch.cuda.synchronize()
            assert _err(y.cpu().numpy(), ref) < TOL[dtype], (desc, batch, d)
            assert torch.equal(y, z), (desc, batch, d)          # in place
        lib.cfft_plan_destroy(h)


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("n,m,istride,ostride", [(16, 5, 5, 5), (64, 64, 64, 64), (120, 31, 40, 33), (256, 256, 300, 256),
                                                 (360, 77, 77, 200), (400, 1, 3, 1), (1000, 129, 131, 140),
                                                 (2160, 50, 64, 50), (4096, 6, 7, 8), (97, 9, 11, 9),
                                                 (16, 40001, 40010, 40001), (256, 2500, 2500, 2600),
                                                 (360, 1701, 1800, 1800), (1000, 701, 701, 703), (2160, 301, 303, 333)])
def test_columns_at_any_stride(cb, dtype, n, m, istride, ostride):
    # column j of an n-row matrix whose rows are istride (ostride) elements apart
    import torch
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    code = cb.C128 if dtype == "complex128" else cb.C64
    h, desc = _plan(cb, lambda h: lib.cfft_plan_create_many(h, n, m, code, cb.EXACT_TWIDDLES, istride, 1, ostride, 1))
    cols = n not in (97, 4096) and n * m * (16 if dtype == "complex128" else 8) >= 4.5 * (1 << 20)
    assert ("cols(V=" in desc) == cols, desc
    x = torch.randn(n, istride, dtype=getattr(torch, dtype), device="cuda")
    xs = x.cpu().numpy().astype(np.complex128)[:, :m]
    for d, ref in ((cb.FORWARD, np.fft.fft(xs, axis=0)), (cb.BACKWARD, np.fft.ifft(xs, axis=0) * n)):
        y = torch.full((n, ostride), 7.0, dtype=getattr(torch, dtype), device="cuda")
        cb.check(lib.cfft_execute(h, vp(x.data_ptr()), vp(y.data_ptr()), d, vp(0)))
        torch.cuda.synchronize()
        out = y.cpu().numpy()
        assert _err(out[:, :m].T, ref.T) < TOL[dtype], desc
        assert (out[:, m:] == 7.0).all(), desc                   # nothing outside the columns
        if istride == ostride:
            z = x.clone()
            cb.check(lib.cfft_execute(h, vp(z.data_ptr()), vp(z.data_ptr()), d, vp(0)))
            torch.cuda.synchronize()
            assert torch.equal(z[:, :m], y[:, :m]) and torch.equal(z[:, m:], x[:, m:]), desc
    lib.cfft_plan_destroy(h)
