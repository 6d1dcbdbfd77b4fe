"""The twiddles of the real transforms' split and merge sweeps (csrc/real.cu).

rfft of the unit impulse at 1: the half-length transform of the vector (i, 0, 0,
...) is i everywhere, exactly (for smooth lengths), so that the split leaves X[k] = w^k as the sweep
has it.  The bar is an FP64 rounding of each component: half an ulp below 1,
2^-54, and a hundredth of that for everything before the last addition.  The
inverse of (w^k) then gives the impulse back."""
import numpy as np
import pytest

from _pkg import load

pytestmark = pytest.mark.gpu


def roots(n):
    """w^k, k <= n/2, to long double accuracy."""
    pi = np.longdouble("3.14159265358979323846264338327950288")
    k = np.arange(n // 2 + 1)
    j = np.minimum(k, n // 2 - k).astype(np.longdouble)         # first quadrant
    a = 2 * pi * j / np.longdouble(n)
    c, s = np.cos(a), np.sin(a)
    return np.where(k <= n // 4, c, -c), -s


@pytest.mark.parametrize("n", [4, 6, 10, 600, 4096, 16384, 16464, 48000, 96000, 10 ** 6, 1 << 20, 2 * 3 ** 12, 1 << 22])
def test_roots_are_rounded_once(n):
    import torch
    cb = load()
    x = torch.zeros(2, n, dtype=torch.float64, device="cuda")
    x[1, 1] = 1.0
    X = cb.rfft(x)
    got = X[1].cpu().numpy()
    c, s = roots(n)
    err = max(np.abs(got.real - c).max(), np.abs(got.imag - s).max())
    assert err <= 1.01 * 2.0 ** -54, (n, float(err))
    assert not X[0].cpu().numpy().any()
    back = cb.irfft(X, n).cpu().numpy()
    want = np.zeros((2, n))
    want[1, 1] = 1.0
    assert np.abs(back - want).max() < 1e-15 * np.log2(n) + 1e-15
