"""Double-precision transforms whose passes have radix 2, 4, 8 and 16 (twiddles
and constants folded into multiply-adds): each radix first, in the middle and
last, beside other codelets, one and many transforms, rows, columns and real
rows, against numpy in extended precision.

Tolerance: a pass of radix 16 rounds an element about 10 times, each by at most
1.1e-16 of it and 0.6e-16 in the mean square of random data, so four passes
stay below 0.6e-16 sqrt(40) = 4e-16 in rel-L2; 5e-16 for one transform, 1e-15
with the real rows' split (and 2e-15 there and back)."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu

LENGTHS = [2, 4, 8, 16, 32, 64, 128, 256, 512, 768, 1024, 1280, 2048, 4096, 8192]


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("N", LENGTHS)
@pytest.mark.parametrize("m,col", [(1, False), (37, False), (19, True)])
def test_complex(N, m, col):
    g = np.random.default_rng(N)
    z = g.standard_normal(m * N) + 1j * g.standard_normal(m * N)
    y = np.zeros(2 * m * N)
    bx, by = J.CBlock(z.view(np.float64).copy(), admit=True), J.CBlock(y, admit=True)
    shape = (0, m, N, 1, m) if col else (0, N, m, 1, N)
    vx, vy = bx.view(*shape), by.view(*shape)
    a, b = (N, m) if col else (m, N)
    p = J.FFTM(J.KIND_CCOP, a, b, 1.0, J.VSIP_FFT_FWD, J.VSIP_COL if col else J.VSIP_ROW, dtype=np.float64)
    p.ccfftmop(vx, vy)
    by.sync()
    ref = np.fft.fft(z.astype(np.clongdouble).reshape(a, b), axis=0 if col else 1)
    assert rel(y.view(np.complex128).reshape(a, b), ref) <= 5e-16
    for v in (vx, vy):
        v.destroy()
    for blk in (bx, by):
        blk.destroy()


@pytest.mark.parametrize("N", [n for n in LENGTHS if n > 2])
def test_real(N):
    m, h = 9, N // 2 + 1
    x = np.random.default_rng(N).standard_normal((m, N))
    z, out = np.zeros(2 * m * h), np.zeros(m * N)
    bx, bz, bo = J.RBlock(x.reshape(-1).copy(), admit=True), J.CBlock(z, admit=True), J.RBlock(out, admit=True)
    vx, vz, vo = bx.view(0, N, m, 1, N), bz.view(0, h, m, 1, h), bo.view(0, N, m, 1, N)
    p = J.FFTM(J.KIND_RCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, dtype=np.float64)
    p.rcfftmop(vx, vz)
    bz.sync()
    assert rel(z.view(np.complex128).reshape(m, h), np.fft.rfft(x.astype(np.longdouble))) <= 1e-15
    q = J.FFTM(J.KIND_CROP, m, N, 1.0 / N, J.VSIP_FFT_INV, J.VSIP_ROW, dtype=np.float64)
    q.crfftmop(vz, vo)
    bo.sync()
    assert rel(out.reshape(m, N), x) <= 2e-15
    for v in (vx, vz, vo):
        v.destroy()
    for blk in (bx, bz, bo):
        blk.destroy()
