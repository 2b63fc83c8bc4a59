"""Which calls on host blocks run on the host arrays themselves: long rows and small
calls do (where the GPU reaches pageable memory through the host's page tables), and
pitched rows; many short rows, rows that overlap in bulk, unaligned and overlapping
arrays keep the copies -- and every call's result matches numpy in 64 bits (rel-L2 1e-6 log2 N,
double 1e-14 log2 N)."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu


def host_access():
    import torch
    return "GB300" in torch.cuda.get_device_name()  # the attribute has no Python name


def run(N, m, dtype=np.float32, pitch=None, skew=0):
    pitch = pitch or N
    g = np.random.default_rng(N + m)
    n = (m - 1) * pitch + N
    x = g.standard_normal(2 * n + 2).astype(dtype)[skew:skew + 2 * n]
    y = np.zeros(2 * m * N, dtype)
    bx, by = J.CBlock(x), J.CBlock(y)
    vx, vy = bx.view(0, pitch, m, 1, N), by.view(0, N, m, 1, N)
    p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, dtype=dtype)
    n0 = J.lib().jvsip_gpu_host_direct_calls()
    p.ccfftmop(vx, vy)
    direct = J.lib().jvsip_gpu_host_direct_calls() - n0
    c = np.complex64 if dtype == np.float32 else np.complex128
    rows = np.lib.stride_tricks.sliding_window_view(x.copy().view(c), N)[::pitch][:m]
    ref = np.fft.fft(rows.astype(np.complex128))
    tol = (1e-6 if dtype == np.float32 else 1e-14) * max(1.0, np.log2(N))
    assert np.linalg.norm(y.view(c).reshape(m, N) - ref) <= tol * np.linalg.norm(ref)
    for o in (vx, vy, bx, by):
        o.destroy()
    return direct


@pytest.mark.parametrize("N,m,dtype,pitch,skew,direct", [
    (1000, 256, np.float32, None, 0, 1), (200, 20000, np.float32, None, 0, 1), (64, 1000, np.float32, None, 0, 1),
    (64, 20000, np.float32, None, 0, 0), (128, 4096, np.float32, None, 0, 1), (128, 4097, np.float32, None, 0, 0),
    (16, 4096, np.float64, None, 0, 1), (16, 4097, np.float64, None, 0, 0), (24, 20000, np.float64, None, 0, 1),
    (1000, 400, np.float32, 250, 0, 1), (1000, 530, np.float32, 250, 0, 0),
    (960, 700, np.float32, 240, 0, 1), (8, 20000, np.float32, 2, 0, 0),
    (64, 20000, np.float32, 256, 0, 1), (1000, 256, np.float32, None, 1, 0), (1500, 40, np.float64, 1502, 0, 1)])
def test_route_and_result(N, m, dtype, pitch, skew, direct):
    if not host_access():
        direct = 0
    assert run(N, m, dtype, pitch, skew) == direct


def test_overlapping_arrays_keep_the_copies():
    N, m = 500, 8
    a = np.random.default_rng(3).standard_normal(2 * N * (m + 1)).astype(np.float32)
    bx, by = J.CBlock(a[:2 * N * m]), J.CBlock(a[2 * N:])
    vx, vy = bx.view(0, N, m, 1, N), by.view(0, N, m, 1, N)
    p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW)
    n0 = J.lib().jvsip_gpu_host_direct_calls()
    p.ccfftmop(vx, vy)
    assert J.lib().jvsip_gpu_host_direct_calls() == n0
    for o in (vx, vy, bx, by):
        o.destroy()
