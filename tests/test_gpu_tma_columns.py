"""TMA-staged column tiles whose transforms per CTA are not a power of two (the CTA's
threads or shared memory do not hold eight): columns into rows, which only the
shared-memory kernel takes, and columns of plans that ask for TMA.  Against numpy in
64 bits; tolerance rel-L2 1e-6 log2 N (double: 1e-14 log2 N)."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m,dtype,force", [(1600, 5242, np.float32, False), (2400, 4866, np.float32, False),
                                             (1500, 4866, np.float32, True), (1300, 4866, np.float64, True),
                                             (1280, 4866, np.float64, True)])
@pytest.mark.parametrize("transposing", [True, False])
def test_columns(monkeypatch, N, m, dtype, force, transposing):
    if force:
        monkeypatch.setenv("JVSIP_GPU_TMA_COLUMNS", "1")
    monkeypatch.setenv("JVSIP_GPU_NO_FAST", "1")
    g = np.random.default_rng(N)
    x = g.standard_normal(2 * N * m, dtype=dtype)
    y = np.zeros_like(x)
    bx, by = J.CBlock(x, admit=True), J.CBlock(y, admit=True)
    vx = bx.view(0, 1, m, m, N)  # transform i down column i of an N x m matrix
    vy = by.view(0, N, m, 1, N) if transposing else by.view(0, 1, m, m, N)
    p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, dtype=dtype, ntimes=1)
    p.ccfftmop(vx, vy)
    by.sync()
    c = np.complex64 if dtype == np.float32 else np.complex128
    pick = np.unique(np.r_[0:24, m // 2:m // 2 + 12, m - 24:m])
    ref = np.fft.fft(x.view(c).reshape(N, m)[:, pick].astype(np.complex128), axis=0)
    got = y.view(c).reshape(m, N)[pick].T if transposing else y.view(c).reshape(N, m)[:, pick]
    assert np.linalg.norm(got - ref) <= (1e-6 if dtype == np.float32 else 1e-14) * np.log2(N) * np.linalg.norm(ref)
    for o in (vx, vy, bx, by):
        o.destroy()
