"""The HBM-pass kernels (csrc/passes.cuh) at the edges of their tiles and radix
sequences: two to six stages, single-radix halves, partial last tiles, one
row or column per tile, the shortest and longest convolutions, forward,
inverse, in place and strided, against the FP64 DFT.

Bars: FP64 rounding of at most ~24 stages of ~4 eps each stays below 1e-13, so
1e-12 (the library's ComplexF64 bar) leaves a decade; FP32 at ~4 x 6e-8 per
stage over at most 12 stages (24 with a convolution) in quadrature is below
2e-6.  Plans are made with EXACT_TWIDDLES: the default Rader tables follow the
reference's recurrence, which drifts from the exact DFT by itself."""
import ctypes

import numpy as np
import pytest

from _pkg import load

pytestmark = pytest.mark.gpu
TOL = {np.complex128: 1e-12, np.complex64: 2e-6}
SMOOTH = [16384 * 3, 3 ** 10, 7 ** 6, 5 ** 7, 2 * 5 ** 7, 10 ** 6, 2 ** 4 * 3 ** 9, 7 ** 4 * 5 ** 4, 2 ** 23]
CONV = [40009, 65537, 100003, 131073, 262147, 999983, (1 << 20) + 7]


@pytest.fixture(scope="module")
def cb():
    return load()


def _run_plan(cb, x, y, direction):
    n, batch = x.shape[1], x.shape[0]
    code = cb.C128 if x.element_size() == 16 else cb.C64
    h = ctypes.c_void_p()
    lib, vp = cb._lib.LIB, ctypes.c_void_p
    cb.check(lib.cfft_plan_create(ctypes.byref(h), n, batch, code, cb.EXACT_TWIDDLES))
    cb.check(lib.cfft_execute(h, vp(x.data_ptr()), vp(y.data_ptr()), direction, vp(0)))
    buf = ctypes.create_string_buffer(256)
    lib.cfft_plan_describe(h, buf, 256)
    import torch
    torch.cuda.synchronize()
    lib.cfft_plan_destroy(h)
    return buf.value.decode()


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", SMOOTH + CONV)
def test_pass_plans_match_fp64(cb, n, dtype):
    import torch
    batch = 1 if n > 3_000_000 else 3
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    real = torch.float64 if dtype == np.complex128 else torch.float32
    x = torch.view_as_complex(torch.randn(batch, n, 2, dtype=real, device="cuda", generator=g))
    keep = x.clone()
    for direction in (cb.FORWARD, cb.INVERSE):
        y = torch.empty_like(x)
        desc = _run_plan(cb, x, y, direction)
        ref = np.fft.fft(keep.cpu().numpy().astype(np.complex128)) if direction == cb.FORWARD else \
            np.fft.ifft(keep.cpu().numpy().astype(np.complex128))
        got = y.cpu().numpy()
        err = max(np.linalg.norm(got[b] - ref[b]) / np.linalg.norm(ref[b]) for b in range(batch))
        assert err < TOL[dtype], (n, direction, desc, err)
        assert torch.equal(x, keep), desc                      # inputs are never modified
        z = x.clone()
        _run_plan(cb, z, z, direction)                  # in place
        assert torch.equal(z, y), desc


@pytest.mark.parametrize("n,m", [(48000, 3), (100003, 2), (3 ** 10, 5)])
def test_pass_plans_strided(cb, n, m):
    # the first axis of an n x m matrix: strided loads and stores of the passes
    import torch
    x = torch.view_as_complex(torch.randn(n, m, 2, dtype=torch.float64, device="cuda"))
    y = cb.fft(x, axis=0).cpu().numpy()
    ref = np.fft.fft(x.cpu().numpy(), axis=0)
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) < TOL[np.complex128]
