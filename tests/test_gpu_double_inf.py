"""Infinities in double-precision rows of 2^k points: an infinite element leaves
finite what its exactly zero factors leave out of a component, and other rows
alone.  Tolerance of the finite parts: rel-L2 1e-14 log2 N."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


def transform(z):
    m, N = z.shape
    y = np.zeros(2 * m * N)
    bx, by = J.CBlock(z.reshape(-1).view(np.float64).copy(), admit=True), J.CBlock(y, admit=True)
    vx, vy = bx.view(0, N, m, 1, N), by.view(0, N, m, 1, N)
    p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, dtype=np.float64)
    p.ccfftmop(vx, vy)
    by.sync()
    for o in (vx, vy, bx, by):
        o.destroy()
    return y.view(np.complex128).reshape(m, N)


def data(m, N):
    g = np.random.default_rng(N)
    return g.standard_normal((m, N)) + 1j * g.standard_normal((m, N))


def close(a, b, N):
    assert np.linalg.norm(a - b) <= 1e-14 * np.log2(N) * np.linalg.norm(b)


@pytest.mark.parametrize("N", [16, 64, 128, 256, 1024, 4096])
def test_infinite_first_element(N):
    """x_0 = inf: every output has real part inf and the imaginary part of the rest."""
    z = data(5, N)
    z[1, 0] = 0
    rest = np.fft.fft(z)
    z[1, 0] = np.inf
    y = transform(z)
    assert np.all(y[1].real == np.inf) and np.all(np.isfinite(y[1].imag))
    close(y[1].imag, rest[1].imag, N)
    for r in (0, 2, 3, 4):
        close(y[r], rest[r], N)


def test_exact_factors_of_a_later_pass():
    """64 points as 16 x 4, x_1 = inf: X_0, X_16, X_32, X_48 get it times 1, -i, -1, i."""
    z = data(3, 64)
    z[1, 1] = 0
    rest = np.fft.fft(z)
    z[1, 1] = np.inf
    y = transform(z)[1]
    got = np.array([y[0].imag, y[16].real, y[32].imag, y[48].real])
    close(got, np.array([rest[1, 0].imag, rest[1, 16].real, rest[1, 32].imag, rest[1, 48].real]), 64)
    assert [y[0].real, y[16].imag, y[32].real, y[48].imag] == [np.inf, -np.inf, -np.inf, np.inf]
