"""Columns too few to give every SM a tile of four: tiles of two and one, which
the kernel that reads its schedule takes (split complex, lengths without
compiled-in columns) -- one transform, a last tile that is not full, both sides
of the counts where tiles become narrower (76 and 152 of 152 SMs), in place --
against numpy in 64 bits.  Tolerance: rel-L2 1e-6 log2 N (double: 1e-14 log2 N)."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [100, 1000, 2197, 2750])
@pytest.mark.parametrize("m", [2, 3, 76, 77, 151, 153, 301, 305])
@pytest.mark.parametrize("split,inplace,dtype", [(True, False, np.float32), (True, True, np.float32),
                                                 (False, False, np.float32), (False, True, np.float64)])
def test_columns(N, m, split, inplace, dtype):
    g = np.random.default_rng(N + m)
    z = g.standard_normal((N, m)) + 1j * g.standard_normal((N, m))
    z = z.astype(np.complex64 if dtype == np.float32 else np.complex128)

    def block(a):
        a = np.ascontiguousarray(a.reshape(-1))
        return J.CBlock(a.real.copy(), a.imag.copy(), admit=True) if split else J.CBlock(a.view(dtype).copy(), admit=True)

    bx = block(z)
    by = bx if inplace else block(np.zeros_like(z))
    vx, vy = bx.view(0, m, N, 1, m), by.view(0, m, N, 1, m)
    p = J.FFTM(J.KIND_CCIP if inplace else J.KIND_CCOP, N, m, 1.0 / N, J.VSIP_FFT_INV, J.VSIP_COL, dtype=dtype, ntimes=1)
    if inplace:
        p.ccfftmip(vx)
    else:
        p.ccfftmop(vx, vy)
    by.sync()
    got = (by.re + 1j * by.im if split else by.re.view(z.dtype)).reshape(N, m)
    ref = np.fft.ifft(z.astype(np.complex128), axis=0)
    tol = (1e-6 if dtype == np.float32 else 1e-14) * np.log2(N)
    assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)
    for v in (vx, vy):
        v.destroy()
    for b in {bx, by}:
        b.destroy()


@pytest.mark.parametrize("N,m", [(7000, 5), (7000, 200), (13312, 9), (14641, 3)])
def test_long_split_columns(N, m):
    test_columns(N, m, True, False, np.float32)
