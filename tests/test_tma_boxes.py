"""The boxes of the TMA-staged column tiles (jvsip_gb300/csrc/jv_tma_box.h, compiled
here by the host compiler): every box starts on a 128-byte boundary of shared
memory, has at most 256 rows, and together they hold the tile and fit it -- for
every even number of transforms a CTA can have, powers of two or not.  No GPU."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jvsip_gb300", "csrc")


@pytest.fixture(scope="module")
def boxes(tmp_path_factory):
    d = tmp_path_factory.mktemp("tma")
    (d / "t.cpp").write_text('#include "jv_tma_box.h"\nextern "C" int boxes(long N, long vpb, long esz, long ld, long *b, long *r) '
                             "{ return jv::tma_boxes(N, vpb, esz, ld, b, r); }\n")
    so = str(d / "t.so")
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", so])
    f = C.CDLL(so).boxes
    f.argtypes = [C.c_long] * 4 + [C.POINTER(C.c_long)] * 2

    def call(N, vpb, esz):
        b, r = C.c_long(), C.c_long()
        ld = (N - 1) + (N - 1) // 16 + 1
        return f(N, vpb, esz, ld + (ld % 2 == 0), C.byref(b), C.byref(r)), b.value, r.value, ld + (ld % 2 == 0)
    return call


@pytest.mark.parametrize("esz", [4, 8])
def test_every_box_is_aligned(boxes, esz):
    taken = 0
    for N in list(range(4, 2100)) + [2187, 2400, 3000, 3072, 4096, 5000, 7776, 8192, 12288, 16384]:
        for vpb in range(2, 65, 2):
            ok, nb, rows, ld = boxes(N, vpb, esz)
            if not ok:
                continue
            taken += 1
            assert rows <= 256 and nb * rows >= N and nb * rows <= ld, (N, vpb, nb, rows)
            assert nb == 1 or rows * vpb * 2 * esz % 128 == 0, (N, vpb, nb, rows)
    assert taken > 10000


def test_tiles_of_powers_of_two_keep_their_boxes(boxes):
    """The rule for row bytes that divide 128 (or are a multiple) is what it was."""
    for esz in (4, 8):
        for N in (64, 1000, 1536, 1600, 2400, 4096, 10000):
            for vpb in (2, 4, 8, 16, 32):
                q = max(1, 128 // (vpb * 2 * esz))
                nb = -(-N // 256)
                rows = -(-(-(-N // nb)) // q) * q
                ok, b, r, ld = boxes(N, vpb, esz)
                assert (b, r) == (nb, rows) and bool(ok) == (rows <= 256 and nb * rows <= ld)
