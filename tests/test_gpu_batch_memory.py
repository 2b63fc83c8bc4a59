"""A batch of long columns when the device memory left does not hold the scratch
of its plans: the calls run as tiles (no scratch) instead of being refused, and
with the memory back the same batch runs as two steps.  In a process of its own,
which holds most of the device memory for the time; against numpy in 64 bits,
tolerance rel-L2 1e-6 log2 N."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r'''
import ctypes as C, numpy as np, torch, jvsip_gb300 as J
N, m = int(__import__("sys").argv[1]), 1440000000 // 8 // int(__import__("sys").argv[1])
z = np.random.default_rng(N).standard_normal(2 * N * m, dtype=np.float32)
want = [0, 1, m // 2, m - 2, m - 1]
src = z.view(np.complex64).reshape(N, m)[:, want].astype(np.complex128)
blk = J.CBlock(z, admit=True)
v = blk.view(0, m, N, 1, m)
p = J.FFTM(J.KIND_CCIP, N, m, 1.0 / N, J.VSIP_FFT_INV, J.VSIP_COL, ntimes=1)
arr = [(C.c_void_p * 1)(o.h) for o in (p, v)]
free = torch.cuda.mem_get_info()[0]
hold = torch.empty(free - (700 << 20), dtype=torch.uint8, device="cuda")  # less than the scratch stays free
for step in range(2):
    n0 = J.lib().jvsip_gpu_kernel_launches()
    assert J.lib().jvsip_fftm_batch_f(1, arr[0], arr[1], arr[1]) == 0, J.last_error()
    assert J.lib().jvsip_gpu_kernel_launches() - n0 == 1 + step  # tiles, then two steps
    blk.sync()
    ref = np.fft.ifft(src, axis=0)
    err = np.linalg.norm(z.view(np.complex64).reshape(N, m)[:, want] - ref) / np.linalg.norm(ref)
    assert err <= 1e-6 * np.log2(N), err
    src = z.view(np.complex64).reshape(N, m)[:, want].astype(np.complex128)
    hold = None
    torch.cuda.empty_cache()
print("ok")
'''


@pytest.mark.parametrize("N", [3000, 10000])
def test_columns_without_scratch_run_as_tiles(N):
    out = subprocess.run([sys.executable, "-c", CODE, str(N)], cwd=ROOT, text=True, capture_output=True, timeout=300)
    assert out.returncode == 0 and out.stdout.split()[-1] == "ok", out.stderr[-2000:]
