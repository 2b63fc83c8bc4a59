"""Batches of short columns whose transforms per tile come from the autotuner or
its cache file, more of them than the tile has threads to spare, against numpy
in 64 bits.  Each in a process of its own (tuned entries are process-wide).
Tolerance: rel-L2 1e-6 log2 N, the library's acceptance bound."""
import os
import subprocess
import sys

import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def child(code, cache):
    env = dict(os.environ, JVSIP_GPU_TUNE_CACHE=str(cache))
    pre = "import sys; sys.path.insert(0, 'tests'); import test_gpu_batch_tuned_columns as T; "
    return subprocess.check_output([sys.executable, "-c", pre + code], env=env, cwd=ROOT, text=True, timeout=120)


def worst(lengths, counts):
    """The largest error of batched column calls over its tolerance."""
    bad = 0.0
    for N in lengths:
        for m in counts:
            g = np.random.default_rng(N + m)
            z = (g.standard_normal((N, m)) + 1j * g.standard_normal((N, m))).astype(np.complex64)
            bx, by = (J.CBlock(a, admit=True) for a in (z.reshape(-1).view(np.float32).copy(), np.zeros(2 * N * m, np.float32)))
            vx, vy = bx.view(0, m, N, 1, m), by.view(0, m, N, 1, m)
            p = J.FFTM(J.KIND_CCOP, N, m, 1.0, J.VSIP_FFT_FWD, J.VSIP_COL)
            arr = [(J.C.c_void_p * 1)(o.h) for o in (p, vx, vy)]
            assert J.lib().jvsip_fftm_batch_f(1, *arr) == 0, J.last_error()
            by.sync()
            ref = np.fft.fft(z.astype(np.complex128), axis=0)
            err = np.linalg.norm(by.re.view(np.complex64).reshape(N, m) - ref) / np.linalg.norm(ref)
            bad = max(bad, err / (1e-6 * max(1.0, np.log2(N))))
            for o in (vx, vy, bx, by, p):
                o.destroy()
    return bad


LENGTHS = [4, 6, 8, 9, 10, 12, 14, 15, 16, 20, 24, 36, 40, 64, 100]


@pytest.mark.parametrize("per", [1, 32, 64, 128, 256, 1024, 1 << 40])
def test_cache_entries(tmp_path, per):
    import torch
    name = torch.cuda.get_device_name().replace(" ", "_")
    cache = tmp_path / "tune.txt"
    cache.write_text("".join("B %s %d 0 1 %d\n" % (name, N, per) for N in LENGTHS))
    out = child("assert T.J.lib().jvsip_fftm_autotune_entries() == %d; print(T.worst(%r, (2, 63, 700)))" % (len(LENGTHS), LENGTHS), cache)
    assert float(out.split()[-1]) <= 1.0


def test_the_autotuner_on_short_columns(tmp_path):
    out = child("import ctypes as C; L = (C.c_ulong * 6)(4, 8, 12, 16, 20, 100); "
                "assert T.J.lib().jvsip_fftm_autotune_f(6, L, 1) == 0, T.J.last_error(); "
                "print(T.worst([4, 8, 12, 16, 20, 100], (2, 63, 700)))", tmp_path / "tune.txt")
    assert float(out.split()[-1]) <= 1.0
    assert len((tmp_path / "tune.txt").read_text().splitlines()) == 6
