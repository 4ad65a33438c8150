"""The host side of native launches in a process with several devices: what the runtime keeps or answers per device is set and
asked on each. Against a stand-in for the CUDA runtime, in a child process without a GPU."""
import os
import shutil
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

from tensorplay_b200 import _build

ROOT = Path(__file__).resolve().parent.parent
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    """Runs code over ``L`` (the kernel library) and ``F`` (the stand-in); returns what it prints."""
    built = _build.LIBDIR / "libtpb200.so"
    if not built.exists():
        _build.build_kernels()
    work = tmp_path_factory.mktemp("fake")
    lib = work / "libfake.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(_build._cuda_home() / "include"),
                    str(ROOT / "tests" / "cpp" / "fake_cuda_runtime.cpp"), "-o", str(lib)], check=True)
    head = textwrap.dedent(f"""
        import ctypes
        from ctypes import c_void_p as P, c_int as I, c_longlong as LL, c_float as FL
        F = ctypes.CDLL({str(lib)!r})
        L = ctypes.CDLL({str(built)!r})
        def decode(D, B=1, Tk=64, splits=0):
            a = P(4096)
            s = LL(8 * D)
            return L.tpb_flash_decode(a, a, a, a, a, None, None, I(B), I(1), I(Tk), I(8), I(8), I(D), *[s] * 12, I(128), I(1), FL(1.0),
                                      I(0), I(splits), None)
    """)

    def run(code):
        out = subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True, timeout=120,
                             env=dict(os.environ, LD_PRELOAD=str(lib), LD_LIBRARY_PATH=str(_build._cuda_home() / "lib64")))
        assert out.returncode == 0, out.stdout + out.stderr
        return out.stdout.split()

    return run


@pytest.mark.parametrize("D", [64, 128])
def test_few_row_attention_on_every_device(child, D):
    assert child(f"""
        for d in (0, 1, 7, 0):
            F.fake_set_device(d)
            print(decode({D}))
    """) == ["0"] * 4


@pytest.mark.parametrize("D", [64, 128])
def test_splits_by_the_device_at_hand(child, D):
    """Two devices that hold different numbers of clusters: each gets the splits that it gets as the first one."""
    code = f"""
        F.fake_set_clusters(0, 40)
        F.fake_set_clusters(1, 1)
        for d in %s:
            F.fake_set_device(d)
            assert decode({D}, 8, 2000) == 0
            print(F.fake_last_grid_x())
    """
    both = child(code % "(0, 1)")
    assert both == child(code % "(0,)") + child(code % "(1,)") and both[0] != both[1]


@pytest.mark.parametrize("D", [64, 128])
def test_long_caches_of_few_heads_take_two_launches(child, D):
    """Where eight CTAs to a head are few for the keys; a short cache stays one launch."""
    assert child(f"""
        F.fake_set_clusters(0, 48)
        for B, Hkv, Tk in ((1, 1, 9000), (1, 2, 9000), (1, 8, 14000), (2, 8, 30000), (1, 1, 2100), (1, 8, 3000), (8, 8, 16381)):
            print(int(L.tpb_flash_decode_splits(I(B), I(1), I(Tk), I(4 * Hkv), I(Hkv), I({D})) > 8))
    """) == list("1111000")


@pytest.mark.parametrize("bits,group", [(4, 128), (8, 0)])
def test_packed_weights_on_every_device(child, bits, group):
    assert child(f"""
        a = P(4096)
        for d in (0, 1, 63, 64, 0):
            F.fake_set_device(d)
            print(L.tpb_wq_gemm(a, a, a, None, None, a, I(64), I(256), I(512), I({bits}), I({group}), LL(512), LL(256), None, None))
    """) == ["0"] * 5


def test_packed_weights_host_time_of_many_rows(child):
    """What is asked on every call of more rows than the GEMV takes is answered in the same time for any number of rows."""
    few, many = (float(t) for t in child("""
        import time
        for M in (1000, 1 << 30):
            best = 1.0
            for _ in range(5):
                t = time.perf_counter()
                L.tpb_wq_gemm_pays(I(M), I(14336), I(4096), I(4), I(128))
                best = min(best, time.perf_counter() - t)
            print(best)
    """))
    assert many < 20 * few + 1e-4   # by the number of row tiles it is a million times


def test_packed_weights_tile_rows(child):
    """The tiles that a launch takes are the cheapest of those with any number of row tiles: its grid says how many there are."""
    SMS = 148
    rows = [1, 5, 16, 17, 31, 32, 33, 48, 49, 100, 128, 129, 191, 192, 193, 200, 333, 384, 385, 512, 577, 777, 1000, 1024, 3000]
    widths = [8, 136, 1000, 4096, 14336, 28672]
    got = child(f"""
        a = P(4096)
        for N in {widths}:
            for M in {rows}:
                assert L.tpb_wq_gemm(a, a, a, None, None, a, I(M), I(N), I(256), I(4), I(128), LL(256), LL(N), None, None) == 0
                print(F.fake_last_grid_x())
    """)
    want = []
    for N in widths:
        for M in rows:
            best = None
            n_tiles = (N + 127) // 128
            for t in range((M + 191) // 192, (M + 15) // 16 + 1):
                nt = ((M + t - 1) // t + 15) // 16 * 16
                if nt > 192:
                    continue
                tiles = n_tiles * ((M + nt - 1) // nt)
                cost = (tiles + SMS - 1) // SMS * (0.42 + 0.0016 * nt)
                if best is None or cost < best[0]:
                    best = (cost, tiles)
            want.append(str(min(best[1], SMS)))
    assert got == want


def test_packed_weights_where_it_pays(child):
    """Sizes at which one of the two ways was measured to be the faster by more than runs differ."""
    here = [(56, 1656, 1280, 8), (20, 4336, 1152, 4), (27, 7560, 1280, 4), (79, 6336, 1152, 4), (87, 3800, 2816, 8), (128, 4096, 4096, 8),
            (22, 10568, 3968, 8), (111, 18568, 7424, 8), (513, 1880, 1792, 4), (777, 14336, 4096, 4), (552, 27880, 2688, 8)]
    there = [(73, 2152, 3200, 8), (35, 2216, 1664, 8), (21, 2136, 3200, 4), (4096, 14336, 4096, 4)]
    got = child(f"""
        for M, N, K, bits in {here + there}:
            print(L.tpb_wq_gemm_pays(I(M), I(N), I(K), I(bits), I(128 if bits == 4 else 0)))
    """)
    assert got == ["1"] * len(here) + ["0"] * len(there)
