"""Batches whose calls are cut for their share of the GPU: many equal small calls,
one large among small ones, few columns of a long length among many (tiles) and
many (two steps), rows and columns in place -- against numpy in 64 bits, captured
and not.  Tolerance: rel-L2 1e-6 log2 N, the library's acceptance bound."""
import ctypes as C

import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu
R, K = J.VSIP_ROW, J.VSIP_COL


@pytest.mark.parametrize("jobs", [
    [(64, 200, R)] * 64, [(100, 7, K)] * 40, [(1000, 4000, R)] + [(128, 3, K), (250, 5, R)] * 20,
    [(3000, 3, K)] * 12 + [(3125, 31, K), (3125, 33, K)], [(3000, 40, K)] * 3, [(8192, 2, K)] * 6 + [(81, 500, K)],
    [(7, 90, R), (4, 1000, K), (16, 333, K), (15, 64, R)] * 3], ids=str)
@pytest.mark.parametrize("inplace", [False, True])
def test_batch(jobs, inplace):
    g = np.random.default_rng(len(jobs))
    total = sum(n * m for n, m, _ in jobs)
    x = (g.standard_normal(total) + 1j * g.standard_normal(total)).astype(np.complex64)
    for captured in (False, True):
        bx = J.CBlock(x.view(np.float32).copy(), admit=True)
        by = bx if inplace else J.CBlock(np.zeros(2 * total, np.float32), admit=True)
        plans, vx, vy, off = [], [], [], 0
        for n, m, major in jobs:
            plans.append(J.FFTM(J.KIND_CCIP if inplace else J.KIND_CCOP, *((m, n) if major == R else (n, m)), 1.0,
                                J.VSIP_FFT_FWD, major))
            shape = (off, n, m, 1, n) if major == R else (off, m, n, 1, m)
            vx.append(bx.view(*shape))
            vy.append(by.view(*shape))
            off += n * m
        arr = [(C.c_void_p * len(jobs))(*[o.h for o in some]) for some in (plans, vx, vy)]
        if captured:
            b = J.lib().jvsip_fftm_batch_create_f(len(jobs), *arr)
            assert b, J.last_error()
            assert J.lib().jvsip_fftm_batch_run_f(b) == 0, J.last_error()
        else:
            assert J.lib().jvsip_fftm_batch_f(len(jobs), *arr) == 0, J.last_error()
        by.sync()
        got, off = by.re.view(np.complex64), 0
        for n, m, major in jobs:
            z = x[off:off + n * m].astype(np.complex128)
            ref = np.fft.fft(z.reshape(m, n)) if major == R else np.fft.fft(z.reshape(n, m), axis=0)
            err = np.linalg.norm(got[off:off + n * m] - ref.reshape(-1)) / np.linalg.norm(ref)
            assert err <= 1e-6 * max(1.0, np.log2(n)), (n, m, major)
            off += n * m
        if captured:
            J.lib().jvsip_fftm_batch_destroy_f(b)
        for o in plans + vx + vy:
            o.destroy()
        for o in {bx, by}:
            o.destroy()
