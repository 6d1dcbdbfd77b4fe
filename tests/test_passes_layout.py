"""CPU check of the HBM-pass kernels' index plan (csrc/passes.cuh): the radix
sequences, in-place positions, twiddle exponents and padded row addresses of
COLPASS, ROWPASS and MIDPASS, restated here, give the DFT (and the cyclic
convolution), touch every position of a tile once per stage and stay inside
the shared memory the planner asks for."""
import numpy as np
import pytest

RADICES = (16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2)


def radices(L):
    """Fewest stages; ascending; at least two (csrc/passplan.h picks among the
    fewest-stage sequences by arithmetic, which no index depends on)."""
    best = None

    def go(rem, mx, cur):
        nonlocal best
        if rem == 1:
            if best is None or len(cur) < len(best):
                best = list(cur)
            return
        if best is not None and len(cur) + 1 >= len(best) or len(cur) == 6:
            return
        for r in RADICES:
            if r <= mx and rem % r == 0:
                go(rem // r, r, cur + [r])
    go(L, 16, [])
    return best[::-1] if len(best) > 1 else best + [1]


def index_of(r, s, b):
    """Output index of position b in digits 0 .. s-1 (sf_index)."""
    k = 0
    for i in range(s - 1, 0, -1):
        b, d = divmod(b, r[i])
        k = (k + d) * r[i - 1]
    return k + b


def w(N, e):
    return np.exp(-2j * np.pi * ((e % N) / N))


def dft(v):
    return np.fft.fft(v)


class Row:
    """One row of a tile: position t at (t // rl) qp + t % rl, with the odd run
    pitch of MIDPASS and narrow ROWPASS tiles (wider ones use qp = rl)."""

    def __init__(self, L):
        self.L, self.r = L, radices(L)
        self.rl = self.r[-1]
        self.qp = self.rl | 1
        self.qw = L // self.rl * self.qp
        self.buf = np.zeros(self.qw, complex)

    def at(self, t):
        return (t // self.rl) * self.qp + t % self.rl

    def butterflies(self, s):
        """(base address, stride, b, K, t') of stage s, every address checked."""
        r = self.r
        Ls = self.L // int(np.prod(r[:s]))
        nb = Ls // r[s]
        seen = np.zeros(self.qw, bool)
        for b in range(self.L // r[s]):
            if s == len(r) - 1:
                base, st, K, tp = b * self.qp, 1, b, 0
            else:
                K, tp = divmod(b, nb)
                base, st = self.at(K * Ls + tp), (nb // self.rl) * self.qp
            idx = base + st * np.arange(r[s])
            assert idx.min() >= 0 and idx.max() < self.qw and not seen[idx].any()
            seen[idx] = True
            yield idx, b, K, tp, nb, Ls
        assert seen.sum() == self.L


def forward(x):
    """FFT of one row through its stages; output in natural order."""
    R = Row(len(x))
    r, n = R.r, len(R.r)
    out = np.zeros(R.L, complex)
    for s in range(n):
        for idx, b, K, tp, nb, Ls in R.butterflies(s):
            v = x[b + nb * np.arange(r[0])] if s == 0 else R.buf[idx]
            v = dft(v)
            if s < n - 1:
                R.buf[idx] = v * w(Ls, tp * np.arange(r[s]))
            else:
                out[index_of(r, n - 1, b) + R.L // r[s] * np.arange(r[s])] = v
    return out


LENGTHS = [2, 4, 16, 21, 27, 81, 100, 243, 250, 256, 343, 625, 1000, 1024, 2187, 2401, 3125, 4096]


@pytest.mark.parametrize("L", LENGTHS)
def test_row_stages_are_the_dft(L):
    rng = np.random.default_rng(L)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    ref = np.fft.fft(x)
    assert np.linalg.norm(forward(x) - ref) < 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("L", [n for n in LENGTHS if len(radices(n)) > 1 and radices(n)[-1] > 1])
def test_mid_pass_is_the_cyclic_convolution(L):
    # MIDPASS on one row: FFT, spectrum in the kernel's order, conjugation,
    # second FFT over the digits in reverse order
    rng = np.random.default_rng(L + 1)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    spec = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    R = Row(L)
    r, n = R.r, len(R.r)
    per = L // r[-1]
    center = np.array([spec[index_of(r, n - 1, u % per) + per * (u // per)] for u in range(L)])
    for s in range(n - 1):
        for idx, b, K, tp, nb, Ls in R.butterflies(s):
            v = dft(x[b + nb * np.arange(r[0])] if s == 0 else R.buf[idx])
            R.buf[idx] = v * w(Ls, tp * np.arange(r[s]))
    for idx, b, *_ in R.butterflies(n - 1):
        v = np.conj(dft(R.buf[idx]) * center[np.arange(r[-1]) * per + b])
        R.buf[idx] = dft(v) * w(L, index_of(r, n - 1, b) * np.arange(r[-1]))
    out = np.zeros(L, complex)
    for s in range(n - 2, -1, -1):
        for idx, b, K, tp, nb, Ls in R.butterflies(s):
            v = dft(R.buf[idx])
            if s:
                pre = L // Ls
                R.buf[idx] = v * w(pre * r[s], index_of(r, s, K) * np.arange(r[s]))
            else:
                out[b + nb * np.arange(r[0])] = v
    ref = np.fft.fft(np.conj(np.fft.fft(x) * spec))
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)


def row_pitches(L, V, e, mid):
    """sf_qp and sf_qw (csrc/passplan.h)."""
    rl, B = radices(L)[-1], 16 if e == 8 else 8
    qp = rl if not mid and V >= B else rl | 1
    n = L // rl * qp
    if mid:
        return qp, n
    step = 1 if V >= B or B % V else B // V
    return qp, n + (step - n) % B


@pytest.mark.parametrize("e", [8, 16])
@pytest.mark.parametrize("L", [81, 256, 324, 729, 1000])
@pytest.mark.parametrize("V", [2, 4, 8, 16, 32])
def test_row_pass_banks(L, V, e):
    # the last stage's lanes (adjacent rows, then adjacent runs) fall in
    # distinct slots of a wavefront for power-of-two widths
    qp, qw = row_pitches(L, V, e, False)
    B = 16 if e == 8 else 8
    lanes = [(i % V) * qw + (i // V) * qp for i in range(B)]
    assert len({x % B for x in lanes}) == B
    assert qw >= L // radices(L)[-1] * qp


def test_quotients_by_multiplier():
    # sf_div: x / d = (x m) >> 32, m = ceil(2^32 / d), for x < 2^20, d <= 2^12
    rng = np.random.default_rng(0)
    for d in list(range(2, 300)) + [int(v) for v in rng.integers(300, 4097, 300)] + [4096]:
        m = (2 ** 32 + d - 1) // d
        q = rng.integers(0, 2 ** 20 // d, 200)
        x = np.concatenate([q * d, q * d + d - 1, [0, 2 ** 20 - 1]]).astype(object)
        assert all(int(v) * m >> 32 == int(v) // d for v in x), d


@pytest.mark.parametrize("N1,N2", [(16, 21), (27, 100), (144, 140)])
def test_three_pass_convolution(N1, N2):
    # COLPASS, MIDPASS, COLPASS over an N1 x N2 intermediate
    M = N1 * N2
    rng = np.random.default_rng(M)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    h = np.fft.fft(rng.standard_normal(M) + 1j * rng.standard_normal(M))
    z = np.fft.fft(x.reshape(N1, N2), axis=0) * w(M, np.outer(np.arange(N1), np.arange(N2)))
    for k1 in range(N1):
        y = np.fft.fft(np.conj(np.fft.fft(z[k1]) * h[k1 + N1 * np.arange(N2)]))
        z[k1] = y * w(M, k1 * np.arange(N2))
    out = np.conj(np.fft.fft(z, axis=0)).reshape(-1) / M
    ref = np.fft.ifft(np.fft.fft(x) * h)
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)


class Line(Row):
    """LINE's row: the first digit's blocks q0 further apart (line_at)."""

    def __init__(self, L):
        super().__init__(L)
        if len(self.r) == 2 and self.r[1] == 1:        # one butterfly a row: two stages where L factors
            for a in (4, 3, 2):
                if L % a == 0 and L // a >= a:
                    self.r = [a, L // a]
                    break
            self.rl = self.r[-1]
            self.qp = self.rl | 1
        self.nb0 = L // self.r[0]
        self.q0 = 0 if len(self.r) < 3 or (self.nb0 // self.rl * self.qp) % 2 else 1
        self.qw = L // self.rl * self.qp + self.r[0] * self.q0
        self.buf = np.zeros(self.qw, complex)

    def line_at(self, t):
        return self.at(t) + t // self.nb0 * self.q0


@pytest.mark.parametrize("L", LENGTHS + [3, 6, 7, 8, 9, 12, 14, 15, 120, 2160, 3840, 8192, 8748, 6561, 7776])
def test_line_stages_are_the_dft(L):
    rng = np.random.default_rng(L + 2)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    R = Line(L)
    r, n = R.r, len(R.r)
    out = np.zeros(L, complex)
    for s in range(n):
        Ls = L // int(np.prod(r[:s]))
        nb, per = Ls // r[s], L // r[s]
        seen = np.zeros(R.qw, bool)
        for i in range(per):
            K, tp = divmod(i, nb)
            if s == 0:
                base, st = R.at(i), nb // R.rl * R.qp + R.q0
            elif s < n - 1:
                base, st = R.line_at(K * Ls + tp), nb // R.rl * R.qp
            if s == n - 1:
                # i is the output index K; its digits in position order give the run
                k = d0 = b = i
                if n > 2:
                    k, d0 = divmod(i, r[0])
                    b = d0
                    for q in range(1, n - 2):
                        k, d = divmod(k, r[q])
                        b = b * r[q] + d
                    b = b * r[n - 2] + k
                base, st = b * R.qp + d0 * R.q0 if n > 2 else b * R.qp, 1
            idx = base + st * np.arange(r[s])
            assert idx.min() >= 0 and idx.max() < R.qw and not seen[idx].any()
            seen[idx] = True
            v = dft(x[i + nb * np.arange(r[0])] if s == 0 else R.buf[idx])
            if s < n - 1:
                R.buf[idx] = v * w(Ls, tp * np.arange(r[s]))
            else:
                out[i + per * np.arange(r[s])] = v
        assert seen.sum() == L
    ref = np.fft.fft(x)
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)
