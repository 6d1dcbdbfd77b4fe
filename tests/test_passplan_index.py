"""The stage kernels' index plan with the numbers of csrc/passplan.h itself
(compiled and called): radix sequences, twiddle blocks, quotient multipliers,
pitches and shared memory of every length the planner can use, and the DFT
through the addresses that csrc/passes.cuh forms from them -- rows of whole
transforms (the ComplexF32 sequences with radices 18 and 20 among them), the
three passes of a convolution, and the cluster kernel's exchange."""
import ctypes

import numpy as np
import pytest

from test_passplan_rules import SfPlan, plan, rules  # noqa: F401 (rules: the compiled probe)


def seq(S):
    return list(S.r)[:S.np]


def smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def div(x, m):
    return x * m >> 32 if m else x


def w(N, e):
    return np.exp(-2j * np.pi * ((e % N) / N))


def index_of(r, s, b):
    """sf_index"""
    k = 0
    for i in range(s - 1, 0, -1):
        b, d = divmod(b, r[i])
        k = (k + d) * r[i - 1]
    return k + b


@pytest.mark.parametrize("maxr,line,top", [(16, False, 4096), (16, True, 9216), (20, True, 9216)])
def test_every_length(rules, maxr, line, top):  # noqa: F811
    rng = np.random.default_rng(maxr + line)
    for L in [n for n in range(2, top + 1) if smooth(n)]:
        S = plan(rules, L, maxr, line)
        r = seq(S)
        assert 2 <= S.np <= 6 and int(np.prod(r)) == L and max(r) <= maxr
        # twiddle blocks: forward ones, then the second transform's, end to end
        off, Ls = 0, L
        for s in range(S.np - 1):
            assert S.off[s] == off
            off += (r[s] - 1) * (Ls // r[s])
            Ls //= r[s]
        assert S.twlen == off
        pre = 1
        for s in range(1, S.np):
            pre *= r[s - 1]
            assert S.boff[s] == off
            off += (r[s] - 1) * pre
        assert S.twall == off < 1 << 16
        # quotients of every index a tile forms (its butterflies: at most 74 KB of
        # ComplexF32 elements over the radix), by every divisor it uses
        sub = L
        for s in range(S.np):
            sub //= r[s]
            for d, m in ((sub, S.mnb[s]), (L // r[s], S.mper[s]), (r[s], S.mr[s])):
                assert m == rules.probe_magic(d) & 0xffffffff
                top_x = max(L, 74 * 1024 // 8)
                q = rng.integers(0, top_x // d + 1, 20)
                for x in [0, top_x] + [int(v) for v in np.concatenate([q * d, q * d + d - 1])]:
                    assert div(x, m) == x // d, (L, d, x)


@pytest.mark.parametrize("maxr,line", [(16, False), (16, True), (20, True)])
def test_twiddle_entries(rules, maxr, line):  # noqa: F811
    e, N = ctypes.c_longlong(), ctypes.c_int()
    for L in (21, 81, 324, 343, 360, 400, 1000, 4096 if not line else 8000):
        S = plan(rules, L, maxr, line)
        r = seq(S)

        def entry(i):
            rules.probe_tw(ctypes.byref(S), i, ctypes.byref(e), ctypes.byref(N))
            return e.value, N.value
        Ls, pre = L, 1
        for s in range(S.np - 1):
            nb = Ls // r[s]
            for k, t in ((1, 0), (1, nb - 1), (r[s] - 1, nb // 2), (r[s] - 1, nb - 1)):
                if r[s] > 1:
                    assert entry(S.off[s] + (k - 1) * nb + t) == (t * k, Ls)
            Ls = nb
        for s in range(1, S.np):
            pre *= r[s - 1]
            for n, b in ((1, 0), (1, pre - 1), (r[s] - 1, pre // 2)):
                if r[s] > 1:
                    assert entry(S.boff[s] + (n - 1) * pre + b) == (index_of(r, s, b) * n, pre * r[s])


def row_at(r, t, qp):
    return t // r[-1] * qp + t % r[-1]


def line_fft(S, x, pitch):
    """LINE on one row, every address checked."""
    L, r, n = S.L, seq(S), S.np
    qp, qw, q0, _ = pitch
    nb0, rl = L // r[0], r[-1]
    buf, out = np.zeros(qw, complex), np.zeros(L, complex)
    Ls = L
    for s in range(n):
        nb, per = Ls // r[s], L // r[s]
        seen = np.zeros(qw, bool)
        for i in range(per):
            K, tp = divmod(i, nb)
            if s == 0:
                base, st = row_at(r, i, qp), nb // rl * qp + q0
            elif s < n - 1:
                t = K * Ls + tp
                base, st = row_at(r, t, qp) + t // nb0 * q0, nb // rl * qp
            else:
                k = d0 = b = i
                if n > 2:
                    k, d0 = divmod(i, r[0])
                    b = d0
                    for q in range(1, n - 2):
                        k, d = divmod(k, r[q])
                        b = b * r[q] + d
                    b = b * r[n - 2] + k
                base, st = b * qp + (d0 * q0 if n > 2 else 0), 1
            idx = base + st * np.arange(r[s])
            assert 0 <= idx.min() and idx.max() < qw and not seen[idx].any()
            seen[idx] = True
            v = np.fft.fft(x[i + nb * np.arange(r[0])] if s == 0 else buf[idx])
            if s < n - 1:
                buf[idx] = v * w(Ls, tp * np.arange(r[s]))
            else:
                out[i + per * np.arange(r[s])] = v
        assert seen.sum() == L
        Ls = nb
    return out


@pytest.mark.parametrize("L,maxr", [(L, m) for m in (16, 20) for L in (2, 3, 16, 18, 20, 36, 324, 360, 400, 1000, 2160,
                                                                       4536, 6000, 6561, 8000, 8820, 9000)])
def test_line(rules, L, maxr):  # noqa: F811
    S = plan(rules, L, maxr, True)
    e = 8 if maxr == 20 else 16
    pitch = (ctypes.c_int * 4)()
    rules.probe_line(ctypes.byref(S), 3, e, pitch)
    assert pitch[3] >= 3 * pitch[1] * e                 # three rows, the last address inside
    rng = np.random.default_rng(L)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    ref = np.fft.fft(x)
    assert np.linalg.norm(line_fft(S, x, list(pitch)) - ref) < 1e-12 * np.linalg.norm(ref)


def stages(S, addr, buf, s, first=None, back=False):
    """One stage of a transform whose position t sits at addr(t): forward, or
    (back) on the same digit of the second transform."""
    L, r = S.L, seq(S)
    Ls = L // int(np.prod(r[:s]))
    nb, per = Ls // r[s], L // r[s]
    pre = L // Ls
    for b in range(per):
        K, tp = divmod(b, nb)
        idx = np.array([addr(K * Ls + tp + m * nb) for m in range(r[s])])
        v = np.fft.fft(first[b + nb * np.arange(r[s])] if first is not None else buf[idx])
        if back:
            yield idx, v * w(pre * r[s], index_of(r, s, K) * np.arange(r[s])) if s else v, b
        else:
            yield idx, v * w(Ls, tp * np.arange(r[s])) if s < S.np - 1 else v, b


@pytest.mark.parametrize("N1,N2", [(16, 18), (27, 100), (42, 144), (100, 343)])
def test_three_passes_of_a_convolution(rules, N1, N2):  # noqa: F811
    # COLPASS, MIDPASS, COLPASS through their tiles' addresses
    A, C = plan(rules, N1), plan(rules, N2)
    M = N1 * N2
    pitch = (ctypes.c_int * 3)()
    rules.probe_row(ctypes.byref(C), 1, 16, 1, pitch)
    qp, qw = pitch[0], pitch[1]
    assert pitch[2] >= qw * 16
    rng = np.random.default_rng(M)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    h = np.fft.fft(rng.standard_normal(M) + 1j * rng.standard_normal(M))

    def columns(z):
        """N1-point DFTs of the columns of z (N1 x N2), position-major tile."""
        out = np.zeros((N1, N2), complex)
        for c in range(N2):
            buf = np.zeros(N1, complex)
            for s in range(A.np):
                for idx, v, b in stages(A, lambda t: t, buf, s, first=z[:, c] if s == 0 else None):
                    if s < A.np - 1:
                        buf[idx] = v
                    else:
                        K = index_of(seq(A), A.np - 1, b)
                        out[K + N1 // A.r[s] * np.arange(A.r[s]), c] = v
        return out

    z = columns(x.reshape(N1, N2)) * w(M, np.outer(np.arange(N1), np.arange(N2)))
    r, n = seq(C), C.np
    per = N2 // r[-1]
    for k1 in range(N1):
        buf = np.full(qw, np.nan + 0j)
        at = lambda t: row_at(r, t, qp)  # noqa: E731
        for s in range(n - 1):
            for idx, v, _ in stages(C, at, buf, s, first=z[k1] if s == 0 else None):
                assert idx.max() < qw
                buf[idx] = v
        for idx, v, b in stages(C, at, buf, n - 1):
            K = index_of(r, n - 1, b)
            u = np.conj(v * h[k1 + N1 * (K + per * np.arange(r[-1]))])
            buf[idx] = np.fft.fft(u) * w(N2, K * np.arange(r[-1]))
        row = np.zeros(N2, complex)
        for s in range(n - 2, -1, -1):
            for idx, v, b in stages(C, at, buf, s, back=True):
                if s:
                    buf[idx] = v
                else:
                    row[b + N2 // r[0] * np.arange(r[0])] = v
        z[k1] = row * w(M, k1 * np.arange(N2))
    out = np.conj(columns(z)).reshape(-1) / M
    ref = np.fft.ifft(np.fft.fft(x) * h)
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("N1,N2,C,e", [(54, 150, 3, 16), (100, 100, 5, 16), (27, 729, 9, 16), (98, 98, 7, 8), (240, 100, 10, 16)])
def test_cluster_exchange(rules, N1, N2, C, e):  # noqa: F811
    # column i2 of CTA i2 / W; output k1 of its last stage goes to row k1 % R1 of
    # CTA k1 / R1, whose row transforms write X[k1 + N1 k2]
    A, B = plan(rules, N1), plan(rules, N2)
    W, R1, M = N2 // C, N1 // C, N1 * N2
    pitch = (ctypes.c_int * 3)()
    rules.probe_row(ctypes.byref(B), R1, e, 0, pitch)
    qp, qw = pitch[0], pitch[1]
    assert rules.probe_clus_smem(ctypes.byref(A), ctypes.byref(B), C, e) >= (N1 * W + R1 * qw) * e
    rng = np.random.default_rng(M)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    rows = np.full((C, R1 * qw), np.nan + 0j)
    ra, rb = seq(A), seq(B)
    for i2 in range(N2):
        buf = np.zeros(N1, complex)
        for s in range(A.np):
            for idx, v, b in stages(A, lambda t: t, buf, s, first=x[i2::N2] if s == 0 else None):
                if s < A.np - 1:
                    buf[idx] = v
                    continue
                K = index_of(ra, A.np - 1, b)
                for j in range(A.r[s]):
                    k1 = K + N1 // A.r[s] * j
                    d = div(k1, rules.probe_magic(R1) & 0xffffffff)
                    slot = (k1 - d * R1) * qw + row_at(rb, i2, qp)
                    assert 0 <= d < C and 0 <= slot < R1 * qw and np.isnan(rows[d, slot])
                    rows[d, slot] = v[j] * w(M, i2 * k1)
    out = np.zeros(M, complex)
    for c in range(C):
        for rr in range(R1):
            buf = rows[c, rr * qw:(rr + 1) * qw]
            for s in range(B.np):
                for idx, v, b in stages(B, lambda t: row_at(rb, t, qp), buf, s):
                    assert idx.max() < qw and not np.isnan(buf[idx]).any()
                    if s < B.np - 1:
                        buf[idx] = v
                    else:
                        K = index_of(rb, B.np - 1, b)
                        out[c * R1 + rr + N1 * (K + N2 // B.r[s] * np.arange(B.r[s]))] = v
    ref = np.fft.fft(x)
    assert np.linalg.norm(out - ref) < 1e-12 * np.linalg.norm(ref)
