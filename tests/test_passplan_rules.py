"""The host rules of the stage kernels (csrc/passplan.h), compiled here and
called: which lengths a kernel takes, without a GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

from _pkg import PKG_DIR, load

MAXS = 6


class SfPlan(ctypes.Structure):
    """engine_types.h"""
    _fields_ = [("L", ctypes.c_int), ("np", ctypes.c_int), ("r", ctypes.c_ubyte * (MAXS + 2)),
                ("off", ctypes.c_ushort * MAXS), ("boff", ctypes.c_ushort * MAXS),
                ("twlen", ctypes.c_int), ("twall", ctypes.c_int),
                ("mnb", ctypes.c_uint * MAXS), ("mper", ctypes.c_uint * MAXS), ("mr", ctypes.c_uint * MAXS),
                ("tw", ctypes.c_void_p)]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = tmp_path_factory.mktemp("probe") / "passplan_probe.so"
    nvcc = os.path.realpath(shutil.which(os.environ.get("NVCC", "nvcc")))
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "passplan_probe.cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", cuda, "-I", os.path.join(PKG_DIR, "csrc"),
                    src, "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.probe_mid_cost.restype = ctypes.c_double
    lib.probe_mid_cost.argtypes = [ctypes.POINTER(SfPlan), ctypes.c_longlong, ctypes.c_int]
    lib.probe_cols_pays.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    lib.probe_tile.argtypes = [ctypes.POINTER(SfPlan), ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_longlong]
    assert lib.probe_plan_bytes() == ctypes.sizeof(SfPlan)
    return lib


def plan(rules, L, maxr=16, line=False):
    S = SfPlan()
    return S if rules.probe_plan(L, maxr, int(line), ctypes.byref(S)) else None


def test_convolution_rows_end_in_a_radix(rules):
    # mid_center has no radix-1 form: a row length whose sequence ends in 1 (one
    # radix) must not be priced as a row of a convolution
    single = 0
    for L in range(2, 4097):
        S = plan(rules, L)
        if S is None:
            continue
        costs = [rules.probe_mid_cost(ctypes.byref(S), 1 << 16, e) for e in (8, 16)]
        if S.r[S.np - 1] < 2:
            single += 1
            assert min(costs) >= 1e9, (L, costs)
        else:
            assert max(costs) < 1e9, (L, costs)
    assert single == 13          # 2 .. 10, 12, 14, 15 and 16


def test_small_images_stay_on_one_kernel(rules):
    # both axes of a small image in LINE: a second kernel for the columns costs
    # more than its whole segments save
    for n, m, e, cols in ((64, 64, 8, 0), (256, 256, 8, 0), (256, 256, 16, 0), (512, 512, 8, 0), (2000, 256, 8, 0),
                          (768, 768, 8, 1), (640, 640, 16, 1), (1000, 1000, 8, 1), (2160, 3840, 8, 1), (4096, 4096, 16, 1)):
        assert rules.probe_cols_pays(n, m, e) == cols, (n, m, e)


@pytest.mark.parametrize("e", [8, 16])
def test_a_few_transforms_get_many_tiles(rules, e):
    # a pass over few transforms must not leave SMs idle for wide tiles of several
    # rounds: 343 rows made 22 tiles or fewer
    for L, count, nb in ((343, 343, 1), (625, 625, 1), (81, 729, 1), (81, 729, 2), (160, 225, 1), (400, 500, 1)):
        S = plan(rules, L)
        for row in (0, 1):
            few = rules.probe_tile(ctypes.byref(S), count, e, row, nb)
            many = rules.probe_tile(ctypes.byref(S), count, e, row, 0)
            assert 1 <= few <= many
            rounds = max(-(-(L // r) // (256 // few)) for r in list(S.r)[:S.np])
            assert -(-count // few) * nb >= 40 or rounds == 1, (L, count, nb, row, few, many)
            # enough transforms: the width for many
            assert rules.probe_tile(ctypes.byref(S), count, e, row, 1000) == many


@pytest.mark.parametrize("n,expect", [(19683, "four(C=9,"), (24000, "four(C=10,"), (59049, "twopass("), (48000, "twopass("),
                                      (77760, "four(C=1")])
def test_one_long_transform(n, expect):
    # one ComplexF64 transform: as many CTAs as shorten it, or two passes where
    # clusters of few large CTAs are slower
    assert expect in load().describe_strategy(n), load().describe_strategy(n)


@pytest.mark.parametrize("n,expect", [(2801, "four(C=4,N1=56,"), (3109, "four(C=5,"), (3301, "four(C=3,"), (2557, "four(C=2,"),
                                      (2503, "rows(V=1)"), (2411, "rows(V=1)"), (1511, "rows(V=1)")])
def test_one_long_prime(n, expect):
    # one ComplexF64 prime: on a cluster where that is shorter than one CTA
    assert expect in load().describe_strategy(n), load().describe_strategy(n)


def test_convolutions_use_radices_up_to_16():
    # 18 and 20 pay in LINE; in LCONV they made every convolution slower
    m = load()
    for n in (163, 181, 1511, 2503, 2506, 3001, 4001):
        d = m.describe_strategy(n, "complex64")
        assert "rows(" in d and max(int(x) for x in d[d.rindex("[") + 1:-1].split(",")) <= 16, d
    assert m.describe_strategy(360, "complex64").endswith("[18,20]")
