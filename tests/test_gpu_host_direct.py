"""Calls on host blocks (not admitted) that the kernels run on the host arrays
themselves, and calls that must keep the copies: bit for bit what a plan with
the copies (JVSIP_GPU_NO_PIPELINE) gives, nothing outside the views written --
pitched rows, in place, split blocks, real rows, both precisions, unaligned
arrays, arrays that overlap."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


def both(monkeypatch, make, run):
    """The arrays after run(plan, ...) with and without device copies."""
    out = []
    for env in (None, "1"):
        if env:
            monkeypatch.setenv("JVSIP_GPU_NO_PIPELINE", env)
        else:
            monkeypatch.delenv("JVSIP_GPU_NO_PIPELINE", raising=False)
        out.append(run(*make()))
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
    return out[0]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,m,pitch", [(64, 1, 64), (1000, 37, 1003), (768, 300, 768), (5632, 3, 5640), (97, 5, 97)])
@pytest.mark.parametrize("inplace,split,skew", [(False, False, 0), (True, False, 0), (False, True, 0), (False, False, 1)])
def test_c2c(monkeypatch, dtype, N, m, pitch, inplace, split, skew):
    """skew: the arrays start one scalar past an aligned address."""
    data = np.random.default_rng(N).standard_normal(2 * m * pitch + 2).astype(dtype)

    def make():
        x, y = data.copy(), np.full_like(data, 3.0)
        return [a[skew:skew + 2 * m * pitch] for a in (x, y)]

    def run(x, y):
        h = m * pitch
        bx = J.CBlock(x[:h], x[h:]) if split else J.CBlock(x)
        by = bx if inplace else J.CBlock(y[:h], y[h:]) if split else J.CBlock(y)
        vx, vy = bx.view(0, pitch, m, 1, N), by.view(0, pitch, m, 1, N)
        p = J.FFTM(J.KIND_CCIP if inplace else J.KIND_CCOP, m, N, 0.5, J.VSIP_FFT_INV, J.VSIP_ROW, dtype=dtype)
        for _ in range(2):
            if inplace:
                p.ccfftmip(vx)
            else:
                p.ccfftmop(vx, vy)
        for v in (vx, vy):
            v.destroy()
        for b in {bx, by}:
            b.destroy()
        return x, y

    x, y = both(monkeypatch, make, run)
    if not inplace and not split:
        z, src = y.view(np.complex64 if dtype == np.float32 else np.complex128).reshape(m, pitch) if not skew else (
            y.copy().view(np.complex64 if dtype == np.float32 else np.complex128).reshape(m, pitch)), data[skew:skew + 2 * m * pitch]
        ref = np.fft.ifft(src.astype(np.float64).view(np.complex128).reshape(m, pitch)[:, :N]) * N * 0.5
        tol = (1e-6 if dtype == np.float32 else 1e-14) * max(1.0, np.log2(N))
        assert np.linalg.norm(z[:, :N] - ref) <= tol * np.linalg.norm(ref)
        assert np.all(z[:, N:] == 3 + 3j)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,m,pad", [(1536, 33, 0), (600, 5, 6), (22, 100, 0)])
def test_real_rows_there_and_back(monkeypatch, dtype, n, m, pad):
    h = n // 2 + 1
    data = np.random.default_rng(n).standard_normal(m * (n + pad)).astype(dtype)

    def run(x, z, o):
        bx, bz, bo = J.RBlock(x), J.CBlock(z), J.RBlock(o)
        vx, vz, vo = bx.view(0, n + pad, m, 1, n), bz.view(0, h, m, 1, h), bo.view(0, n + pad, m, 1, n)
        J.FFTM(J.KIND_RCOP, m, n, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, dtype=dtype).rcfftmop(vx, vz)
        J.FFTM(J.KIND_CROP, m, n, 1.0 / n, J.VSIP_FFT_INV, J.VSIP_ROW, dtype=dtype).crfftmop(vz, vo)
        for v in (vx, vz, vo):
            v.destroy()
        for b in (bx, bz, bo):
            b.destroy()
        return x, z, o

    x, z, o = both(monkeypatch, lambda: (data.copy(), np.zeros(2 * m * h, dtype), np.zeros_like(data)), run)
    tol = (2e-6 if dtype == np.float32 else 2e-14) * np.log2(n)
    r, e = o.reshape(m, -1)[:, :n], data.reshape(m, -1)[:, :n]
    assert np.linalg.norm(r - e) <= tol * np.linalg.norm(e)
    assert not o.reshape(m, -1)[:, n:].any()


def test_blocks_on_overlapping_arrays_keep_the_copies(monkeypatch):
    """Two blocks bound to ranges of one array that overlap: the input is copied
    before any output is written."""
    N, m = 500, 8
    data = np.random.default_rng(3).standard_normal(2 * N * (m + 1)).astype(np.float32)

    def run(a):
        bx, by = J.CBlock(a[:2 * N * m]), J.CBlock(a[2 * N:])
        vx, vy = bx.view(0, N, m, 1, N), by.view(0, N, m, 1, N)
        J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW).ccfftmop(vx, vy)
        for v in (vx, vy):
            v.destroy()
        for b in (bx, by):
            b.destroy()
        return (a,)

    a, = both(monkeypatch, lambda: (data.copy(),), run)
    ref = np.fft.fft(data[:2 * N * m].astype(np.float64).view(np.complex128).reshape(m, N))
    got = a[2 * N:].view(np.complex64).reshape(m, N)
    assert np.linalg.norm(got - ref) <= 1e-6 * np.log2(N) * np.linalg.norm(ref)
