"""Performance cases of the FFT library, through its public entry points.

Every case is one of the forms in which the library is used:

  c2c     plan_fft / plan_ifft objects applied to a [batch, n] device tensor:
          forward, or forward and then inverse of the spectrum
  real    rfft and irfft of a [batch, n] real device tensor
  fft2    both axes of a device matrix (the first axis is a strided plan)
  batch   Batch: many transforms of uneven lengths, packed, in one launch
  serve   Server: independent requests submitted one by one and drained
"""
import importlib
import importlib.util
import math
import os

import torch

_DT = {"c128": torch.complex128, "c64": torch.complex64}
_E = {"c128": 16, "c64": 8}
_LMAX_BATCH = 1 << 20          # longest transform of a packed batch
_LMAX_SERVE = 1 << 22          # longest served transform
_TICKETS = 1 << 20             # requests a server sees in its lifetime


def _cb():
    path = os.path.join(os.getcwd(), "catabrafft.jl_b200", "_load.py")
    spec = importlib.util.spec_from_file_location("catabra_b200_load", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m.load()


def _workloads():
    _cb()
    return importlib.import_module("catabra_b200.workloads")


def listed():
    return [
        # the smallest call: one vector, forward and back (latency and launches)
        dict(name="single_4096_c128", kind="c2c", n=4096, batch=1, dtype="c128", inverse=True),
        # very many very short transforms (120 = 2^3 3 5, the longest of the short-length sweep)
        dict(name="short_120_c64", kind="c2c", n=120, batch=400000, dtype="c64", inverse=False),
        # the plain mixed-radix batch, forward and inverse
        dict(name="mixed_30240_c128", kind="c2c", n=30240, batch=1024, dtype="c128", inverse=True),
        # the plain prime-length batch (Rader), forward and inverse
        dict(name="prime_10007_c128", kind="c2c", n=10007, batch=1024, dtype="c128", inverse=True),
        # the precision form's power of two and its power of three: the largest calls
        dict(name="pow2_65536_c64", kind="c2c", n=65536, batch=4096, dtype="c64", inverse=False),
        dict(name="pow3_19683_c64", kind="c2c", n=19683, batch=4096, dtype="c64", inverse=False),
        # long power-of-two transforms in double precision (two passes over memory)
        dict(name="pow2_1048576_c128", kind="c2c", n=1 << 20, batch=64, dtype="c128", inverse=False),
        # real signals (one second of 48 kHz audio per row), analysis and synthesis
        dict(name="real_48000_f32", kind="real", n=48000, batch=1024, dtype="c64"),
        # a 4K image's spectrum: strided transforms along the first axis
        dict(name="image_2160x3840_c64", kind="fft2", n=2160, m=3840, dtype="c64"),
        # uneven lengths, half 7-smooth and half with a large prime factor, in one launch
        dict(name="batch_1000_c64", kind="batch", count=1000, lengths_seed=1, dtype="c64"),
        dict(name="batch_1000_c128", kind="batch", count=1000, lengths_seed=1, dtype="c128"),
        # a burst of independent requests of any length, batched as they arrive
        dict(name="serve_256_c64", kind="serve", count=256, lengths_seed=1, dtype="c64"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _is_prime(n):
    if n < 4:
        return n > 1
    if n % 2 == 0:
        return False
    return all(n % d for d in range(3, int(n ** 0.5) + 1, 2))


def _length(rng, lo, hi, primes=True):
    """A power of two, a 7-smooth length, any length, or a prime."""
    t = _log_uniform(rng, lo, hi)
    kind = rng.choice(["pow2", "smooth", "smooth", "any", "prime"] if primes else ["pow2", "smooth", "smooth"])
    if kind == "pow2":
        return min(max(1 << round(math.log2(t)), lo), hi)
    if kind == "smooth":
        return _workloads().nearest_smooth(t, lo, hi)
    n = int(t)
    if kind == "prime":
        while not _is_prime(n):
            n -= 1
    return max(n, 2)


def draw(rng):
    kind = rng.choice(["c2c", "c2c", "c2c", "real", "fft2", "batch", "serve"])
    dtype = rng.choice(["c64", "c128"])
    if kind == "c2c":
        n = _length(rng, 16, 1 << 22)
        # up to 2^25 elements, 2^23 where a length outside the 7-smooth ones costs a convolution
        smooth = n
        for q in (2, 3, 5, 7):
            while smooth % q == 0:
                smooth //= q
        most = max(1, (1 << (25 if smooth == 1 else 23)) // n)
        return dict(kind=kind, n=n, batch=max(1, round(_log_uniform(rng, 1, most))), dtype=dtype,
                    inverse=rng.random() < 0.5)
    if kind == "real":
        n = _length(rng, 64, 1 << 20, primes=False)
        return dict(kind=kind, n=n, batch=max(1, round(_log_uniform(rng, 1, (1 << 25) / n))), dtype=dtype)
    if kind == "fft2":
        return dict(kind=kind, n=_length(rng, 64, 4096, primes=False), m=_length(rng, 64, 4096, primes=False),
                    dtype=dtype)
    if kind == "batch":
        return dict(kind=kind, count=round(_log_uniform(rng, 100, 1000)), lengths_seed=rng.randrange(1 << 30),
                    dtype=dtype)
    return dict(kind=kind, count=round(_log_uniform(rng, 16, 256)), lengths_seed=rng.randrange(1 << 30),
                dtype="c64")


def _lengths(case):
    w = _workloads()
    if case["kind"] == "batch":
        return [int(n) for n in w.batch_lengths(case["count"], case["lengths_seed"], hi=_LMAX_BATCH)]
    return [int(n) for _, n in w.request_stream(case["count"], 50000.0, case["lengths_seed"], hi=_LMAX_SERVE)]


def _input(case, seed):
    """Seeded N(0,1) parts (uniform(-1, 1) for the single-precision c2c form)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    real = torch.float64 if case["dtype"] == "c128" else torch.float32
    kind = case["kind"]
    if kind == "real":
        return torch.randn(case["batch"], case["n"], dtype=real, device="cuda", generator=g)
    if kind == "c2c":
        shape = (case["batch"], case["n"]) if case["batch"] > 1 else (case["n"],)
    elif kind == "fft2":
        shape = (case["n"], case["m"])
    else:
        shape = (sum(_lengths(case)),)
    if kind == "c2c" and case["dtype"] == "c64":
        x = torch.rand(*shape, 2, dtype=real, device="cuda", generator=g) * 2 - 1
    else:
        x = torch.randn(*shape, 2, dtype=real, device="cuda", generator=g)
    return torch.view_as_complex(x)


def prepare(case, seed):
    cb = _cb()
    kind = case["kind"]
    s = {"cb": cb, "case": case, "x": _input(case, seed)}
    if kind == "c2c":
        s["p"] = cb.plan_fft(s["x"])
        if case["inverse"]:
            s["pi"] = cb.plan_ifft(s["x"])
    elif kind == "real":
        s["p"] = cb.plan_rfft(s["x"])
    elif kind == "batch":
        s["b"] = cb.Batch(_lengths(case), _DT[case["dtype"]])
        s["y"] = torch.empty_like(s["x"])
    elif kind == "serve":
        s["y"] = torch.empty_like(s["x"])
        s["srv"] = cb.Server(_DT[case["dtype"]], max_requests=_TICKETS)
        lengths = _lengths(case)
        s["srv"].prepare(sorted(set(lengths)))
        s["reqs"] = list(zip(s["x"].split(lengths), s["y"].split(lengths)))
    torch.cuda.synchronize()
    return s


def run(s):
    cb, case, x = s["cb"], s["case"], s["x"]
    kind = case["kind"]
    if kind == "c2c":
        y = s["p"] * x
        return (y, s["pi"] * y) if case["inverse"] else y
    if kind == "real":
        X = s["p"] * x
        return X, cb.irfft(X, case["n"])
    if kind == "fft2":
        return cb.fft2(x)
    if kind == "batch":
        return s["b"].execute(x, out=s["y"])
    submit = s["srv"].submit
    for a, b in s["reqs"]:
        submit(a, b)
    s["srv"].drain()
    return s["y"]


def _fft_flops(n):
    return 5.0 * n * math.log2(n) if n > 1 else 0.0


def work(case):
    kind, e = case["kind"], _E[case["dtype"]]
    if kind == "c2c":
        k = 2 if case["inverse"] else 1
        return {"bytes": k * 2.0 * case["batch"] * case["n"] * e, "flops": k * case["batch"] * _fft_flops(case["n"])}
    if kind == "real":
        n, b = case["n"], case["batch"]
        return {"bytes": 2.0 * b * (n * e / 2 + (n // 2 + 1) * e), "flops": b * _fft_flops(n)}
    if kind == "fft2":
        n, m = case["n"], case["m"]
        return {"bytes": 2.0 * n * m * e, "flops": m * _fft_flops(n) + n * _fft_flops(m)}
    lengths = _lengths(case)
    return {"bytes": 2.0 * e * sum(lengths), "flops": sum(_fft_flops(n) for n in lengths)}


def exact(case, seed):
    x = _input(case, seed)
    kind = case["kind"]
    if kind == "real":
        x = x.to(torch.float64)
        X = torch.fft.rfft(x)
        return X, torch.fft.irfft(X, n=case["n"])
    x = x.to(torch.complex128)
    if kind == "c2c":
        y = torch.fft.fft(x)
        return (y, torch.fft.ifft(y)) if case["inverse"] else y
    if kind == "fft2":
        return torch.fft.fft2(x)
    torch.backends.cuda.cufft_plan_cache[torch.cuda.current_device()].max_size = 16
    return torch.cat([torch.fft.fft(v) for v in x.split(_lengths(case))])
