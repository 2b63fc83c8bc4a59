"""The thread counts of the in-place mixed-radix kernel's column tiles
(jvsip_gb300/csrc/jv_dif_tile.h, compiled here by the host compiler): for every
length and every number of transforms per tile that the autotuner, its cache
file or a caller can ask for, the threads are a multiple of the tile's
transforms, so that every loop over butterflies advances and no two threads
share a butterfly.  No GPU."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jvsip_gb300", "csrc")
SMEM = 227 * 1024 // 8  # complex values of the largest tile


@pytest.fixture(scope="module")
def tile(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile")
    (d / "t.cpp").write_text('#include "jv_dif_tile.h"\nusing namespace jv;\nextern "C" {\n'
                             "int tuned(long t, long nvec) { return dif_col_tuned(t, nvec); }\n"
                             "long threads(long N, int lgv, int f32, int few) { return dif_col_threads(N, lgv, f32 != 0, few != 0); }\n"
                             "int narrow(int lgv, long nvec, long sms) { return dif_col_narrow(lgv, nvec, sms); }\n"
                             "int batch(int nthr) { return dif_batch_threads(nthr); }\n}\n")
    so = str(d / "t.so")
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", so])
    lib = C.CDLL(so)
    lib.tuned.argtypes = [C.c_long, C.c_long]
    lib.narrow.argtypes = [C.c_int, C.c_long, C.c_long]
    lib.threads.argtypes, lib.threads.restype = [C.c_long, C.c_int, C.c_int, C.c_int], C.c_long
    return lib


def runs_every_butterfly_once(nthr, V, nb):
    """The loops of dif_first / dif_mid / dif_last: (transform, butterfly) pairs."""
    step = nthr // V
    if step < 1:
        return False  # would never end
    seen = set()
    for i in range(nthr):
        for b in range(i // V, nb, step):
            if (i % V, b) in seen:
                return False
            seen.add((i % V, b))
    return len(seen) == V * nb


@pytest.mark.parametrize("f32", [0, 1])
@pytest.mark.parametrize("few", [0, 1])
def test_every_length_and_tuned_tile(tile, f32, few):
    for N in list(range(4, 65)) + [100, 256, 1000, 1024, 2187, 4096, 16384]:
        for tuned in [1 << k for k in range(15)] + [3, 100, 1 << 40, (1 << 63) - 1]:
            for nvec in (2, 5, 64, 1 << 20):
                lgv = tile.tuned(tuned, nvec)
                assert 0 <= lgv <= 9 and (lgv == 0 or (1 << lgv) <= tuned)
                while lgv > 0 and (N << lgv) > SMEM:
                    lgv -= 1
                V, n = 1 << lgv, tile.threads(N, lgv, f32, few)
                assert 64 <= n <= (1024 if f32 else 512) and n >= V and n % V == 0 and n % 32 == 0, (N, tuned, n)
                m = tile.batch(n)
                assert m <= 1024 and m % 64 == 0 and m % V == 0, (N, tuned, n, m)


def test_few_columns_are_spread_over_the_sms(tile):
    for nvec in range(2, 1300):
        for lgv in range(5):
            n = tile.narrow(lgv, nvec, 152)
            tiles = [-(-nvec >> k) for k in range(lgv + 1)]
            assert n == lgv if 2 * tiles[lgv] > 152 else tiles[n] <= 152 and (n == 0 or 2 * tiles[n] > 152), (nvec, lgv)


@pytest.mark.parametrize("N,tuned", [(8, 128), (12, 256), (16, 1024), (20, 256), (24, 128), (36, 256), (64, 256)])
def test_tiles_of_short_lengths_run_each_butterfly_once(tile, N, tuned):
    lgv = tile.tuned(tuned, 1 << 20)
    V, n = 1 << lgv, tile.threads(N, lgv, 1, 0)
    for R in (2, 3, 4):
        if N % R == 0:
            assert runs_every_butterfly_once(n, V, N // R)
            assert runs_every_butterfly_once(tile.batch(n), V, N // R)


@pytest.mark.parametrize("N,V,nthr", [(8, 128, 64), (16, 1024, 512), (20, 256, 320)])
def test_the_oracle_sees_too_few_or_uneven_threads(N, V, nthr):
    assert not runs_every_butterfly_once(nthr, V, N // 2)
