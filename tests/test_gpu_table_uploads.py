"""Tables of new plans while batches are queued whose device queues are back in
the buffer pool: the copies into pool buffers take their turn behind the work
that still reads them, and the plan's own first call, queued right after, finds
its tables.  Results against numpy in 64 bits; tolerance rel-L2 1e-6 log2 N."""
import ctypes as C

import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def test_plans_made_behind_queued_batches():
    g = np.random.default_rng(5)
    N, m, calls = 1000, 40, 48
    z = (g.standard_normal((calls, m, N)) + 1j * g.standard_normal((calls, m, N))).astype(np.complex64)
    bx, by = J.CBlock(z.reshape(-1).view(np.float32).copy(), admit=True), J.CBlock(np.zeros(2 * z.size, np.float32), admit=True)
    p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, ntimes=1)
    xs, ys = ([b.view(i * m * N, N, m, 1, N) for i in range(calls)] for b in (bx, by))
    arr = [(C.c_void_p * calls)(*h) for h in ([p.h] * calls, [v.h for v in xs], [v.h for v in ys])]
    # work that keeps the stream busy while the batch and the plans are queued
    big = J.CBlock(g.standard_normal(2 << 24).astype(np.float32), admit=True)
    vb = big.vview(0, 1, 1 << 24)
    pb = J.FFT(J.KIND_CCIP, 1 << 24, 1.0 / 4096, ntimes=1)
    pb.ccfftip(vb)
    ref = np.fft.fft(z.astype(np.complex128))
    plans = []
    for k in range(12):
        for _ in range(6):
            pb.ccfftip(vb)
        assert J.lib().jvsip_fftm_batch_f(calls, *arr) == 0, J.last_error()
        # tables of 2 to 128 KB: the size classes of the batch's calls and tiles
        plans += [(n + 64 * k, J.FFTM(J.KIND_CCOP, 3, n + 64 * k, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, ntimes=1))
                  for n in (256, 1024, 2048, 4096, 8192)]
        by.sync()
        assert rel(by.re.view(np.complex64).reshape(z.shape), ref) <= 1e-6 * np.log2(N)
    for n, q in plans:
        v = bx.view(0, n, 3, 1, n)
        o = by.view(0, n, 3, 1, n)
        q.ccfftmop(v, o)
        by.sync()
        src = z.reshape(-1)[:3 * n].reshape(3, n).astype(np.complex128)
        assert rel(by.re.view(np.complex64)[:3 * n].reshape(3, n), np.fft.fft(src)) <= 1e-6 * np.log2(n), n
        v.destroy()
        o.destroy()
    for o in xs + ys + [vb]:
        o.destroy()
    for o in (bx, by, big):
        o.destroy()
