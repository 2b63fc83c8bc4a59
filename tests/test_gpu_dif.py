"""The in-place mixed-radix kernel (lengths that the register-resident kernel
does not take) where it can go wrong: two to five passes, every codelet from 2
to 16, the smallest and the largest length, one transform, a last CTA that is
not full, pitched and descending rows, in place, split complex, columns, real
rows of every spectrum layout -- against numpy in 64 bits and, for routes, the
general kernels (JVSIP_GPU_NO_FAST).  Tolerance: rel-L2 1e-6 log2 N, the
library's acceptance bound for single precision."""
import numpy as np
import pytest

import jvsip_gb300 as J

pytestmark = pytest.mark.gpu

LENGTHS = [4, 6, 22, 26, 72, 121, 130, 143, 169, 210, 300, 441, 1001, 1331, 1500, 2197, 2310, 3000, 3125, 3600, 5632,
           6561, 12000, 13312, 14641, 15625, 16380, 16384]


def tol(N):
    return 1e-6 * max(1.0, np.log2(N))


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def rnd(n, seed):
    g = np.random.default_rng(seed)
    return (g.standard_normal(n) + 1j * g.standard_normal(n)).astype(np.complex64)


def run_rows(N, m, pitch, d, inplace, split, descending=False):
    """One c2c call on m rows `pitch` apart; the whole blocks before and after."""
    z = rnd(m * pitch, N + m)
    scale = 1.0 if d < 0 else 1.0 / N
    fill = np.full(m * pitch, 7 - 5j, np.complex64)

    def block(v):
        if split:
            return J.CBlock(v.real.copy(), v.imag.copy(), admit=True)
        return J.CBlock(v.copy().view(np.float32), admit=True)

    def values(b):
        b.sync()
        return b.re + 1j * b.im if split else b.re.view(np.complex64)

    bx = block(z)
    by = bx if inplace else block(fill)
    args = ((m - 1) * pitch, -pitch, m, 1, N) if descending else (0, pitch, m, 1, N)
    vx = bx.view(*args)
    vy = vx if inplace else by.view(*args)
    p = J.FFTM(J.KIND_CCIP if inplace else J.KIND_CCOP, m, N, scale, d, J.VSIP_ROW, ntimes=1)
    if inplace:
        p.ccfftmip(vx)
    else:
        p.ccfftmop(vx, vy)
    got = values(by).reshape(m, pitch)
    src = z.reshape(m, pitch)
    ref = np.fft.fft(src[:, :N].astype(np.complex128)) if d < 0 else np.fft.ifft(src[:, :N].astype(np.complex128))
    assert rel(got[:, :N], ref) <= tol(N)
    assert np.array_equal(got[:, N:], (src if inplace else fill.reshape(m, pitch))[:, N:])
    for v in {vx, vy}:
        v.destroy()
    for b in {bx, by}:
        b.destroy()


@pytest.mark.parametrize("N", LENGTHS)
@pytest.mark.parametrize("split", [False, True], ids=["interleaved", "split"])
def test_rows(N, split):
    run_rows(N, 1, N, J.VSIP_FFT_FWD, False, split)
    run_rows(N, 37, N + 3, J.VSIP_FFT_INV, False, split)
    run_rows(N, 37, N + 3, J.VSIP_FFT_FWD, True, split)
    run_rows(N, 700 if N < 4000 else 5, N, J.VSIP_FFT_INV, True, split, descending=True)


@pytest.mark.parametrize("N", [n for n in LENGTHS if n < 3000])
@pytest.mark.parametrize("cols,extra,inplace", [(2, 0, False), (19, 3, True), (64, 0, False)])
def test_columns(N, cols, extra, inplace):
    pitch = cols + extra
    z = rnd(N * pitch, N + cols)
    bx = J.CBlock(z.copy().view(np.float32), admit=True)
    by = bx if inplace else J.CBlock(np.zeros(2 * N * pitch, np.float32), admit=True)
    vx, vy = bx.view(0, pitch, N, 1, cols), by.view(0, pitch, N, 1, cols)
    p = J.FFTM(J.KIND_CCIP if inplace else J.KIND_CCOP, N, cols, 1.0 / N, J.VSIP_FFT_INV, J.VSIP_COL, ntimes=1)
    n0 = J.lib().jvsip_gpu_kernel_launches()
    if inplace:
        p.ccfftmip(vx)
    else:
        p.ccfftmop(vx, vy)
    assert J.lib().jvsip_gpu_kernel_launches() - n0 == 1
    by.sync()
    got, src = by.re.view(np.complex64).reshape(N, pitch), z.reshape(N, pitch)
    assert rel(got[:, :cols], np.fft.ifft(src[:, :cols].astype(np.complex128), axis=0)) <= tol(N)
    assert np.array_equal(got[:, cols:], (src if inplace else np.zeros_like(src))[:, cols:])
    for v in (vx, vy):
        v.destroy()
    for b in {bx, by}:
        b.destroy()


# large calls: power-of-two columns go back to the register-resident tiles, tiles
# of 4 columns become 8; ragged counts, first, middle and last columns
@pytest.mark.parametrize("N,cols", [(64, 16391), (256, 4099), (512, 32773), (128, 262147), (1350, 24859), (1792, 18727)])
def test_large_column_calls(N, cols):
    z = rnd(N * cols, N)
    bx = J.CBlock(z.copy().view(np.float32), admit=True)
    by = J.CBlock(np.zeros(2 * N * cols, np.float32), admit=True)
    vx, vy = bx.view(0, cols, N, 1, cols), by.view(0, cols, N, 1, cols)
    p = J.FFTM(J.KIND_CCOP, N, cols, 1.0, J.VSIP_FFT_FWD, J.VSIP_COL, ntimes=1)
    n0 = J.lib().jvsip_gpu_kernel_launches()
    p.ccfftmop(vx, vy)
    assert J.lib().jvsip_gpu_kernel_launches() - n0 == 1
    by.sync()
    pick = np.unique(np.r_[0:17, cols // 2 - 8:cols // 2 + 9, cols - 17:cols])
    got, src = by.re.view(np.complex64).reshape(N, cols)[:, pick], z.reshape(N, cols)[:, pick]
    assert rel(got, np.fft.fft(src.astype(np.complex128), axis=0)) <= tol(N)
    for v in (vx, vy):
        v.destroy()
    for b in (bx, by):
        b.destroy()


@pytest.mark.parametrize("N", LENGTHS)
@pytest.mark.parametrize("m,pad,colmajor", [(1, 0, False), (53, 4, False), (6, 0, True)])
def test_real_rows(N, m, pad, colmajor):
    """R2C into rows `pad` apart or a column-major spectrum, then C2R back from rows (2N real points)."""
    n, h = 2 * N, N + 1
    x = np.random.default_rng(N).standard_normal((m, n + pad)).astype(np.float32)
    bx = J.RBlock(x.reshape(-1).copy(), admit=True)
    z = np.zeros(2 * m * (h + pad), np.float32)
    bz = J.CBlock(z, admit=True)
    vx = bx.view(0, n + pad, m, 1, n)
    vz = bz.view(0, 1, m, m, h) if colmajor else bz.view(0, h + pad, m, 1, h)
    p = J.FFTM(J.KIND_RCOP, m, n, 0.5, J.VSIP_FFT_FWD, J.VSIP_ROW, ntimes=1)
    p.rcfftmop(vx, vz)
    bz.sync()
    zc = z.view(np.complex64)
    got = zc[:m * h].reshape(h, m).T if colmajor else zc.reshape(m, h + pad)[:, :h]
    assert rel(got, 0.5 * np.fft.rfft(x[:, :n].astype(np.float64))) <= tol(n)
    if not colmajor:
        assert not zc.reshape(m, h + pad)[:, h:].any()
        out = np.full(m * (n + pad), 3.0, np.float32)
        bo = J.RBlock(out, admit=True)
        vo = bo.view(0, n + pad, m, 1, n)
        q = J.FFTM(J.KIND_CROP, m, n, 2.0 / n, J.VSIP_FFT_INV, J.VSIP_ROW, ntimes=1)
        q.crfftmop(vz, vo)
        bo.sync()
        assert rel(out.reshape(m, -1)[:, :n], x[:, :n].astype(np.float64)) <= 2 * tol(n)
        assert np.all(out.reshape(m, -1)[:, n:] == 3.0)
        vo.destroy()
        bo.destroy()
    for v in (vx, vz):
        v.destroy()
    for b in (bx, bz):
        b.destroy()


@pytest.mark.parametrize("N", [72, 1500, 6000])
def test_routes_agree_with_the_general_kernels(monkeypatch, N):
    """Views that take the kernel and views that do not (strided elements,
    overlapping rows, odd real offsets) give what JVSIP_GPU_NO_FAST plans give."""
    m = 9
    for cs, rs in ((N, 1), (2 * N, 2), (N // 2, 1), (1, m), (1, m + 2)):
        z = rnd(2 * (m + 2) * N, 3)
        outs = []
        for env in (None, "1"):
            if env:
                monkeypatch.setenv("JVSIP_GPU_NO_FAST", env)
            else:
                monkeypatch.delenv("JVSIP_GPU_NO_FAST", raising=False)
            bx, by = J.CBlock(z.copy().view(np.float32), admit=True), J.CBlock(np.zeros(2 * z.size, np.float32), admit=True)
            ocs, ors = (cs, rs) if cs != N // 2 else (N, 1)
            vx, vy = bx.view(0, cs, m, rs, N), by.view(0, ocs, m, ors, N)
            p = J.FFTM(J.KIND_CCOP, m, N, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, ntimes=1)
            p.ccfftmop(vx, vy)
            by.sync()
            outs.append(by.re.view(np.complex64).copy())
            for v in (vx, vy):
                v.destroy()
            for b in (bx, by):
                b.destroy()
        assert rel(outs[0], outs[1]) <= tol(N), (cs, rs)
        assert np.array_equal(outs[0] == 0, outs[1] == 0)


@pytest.mark.parametrize("N", [8748, 9000, 59049, 100842, 234375, 823543, 1953125, 1 << 21, 3 << 20, 2 * 3 ** 13])
@pytest.mark.parametrize("inplace", [False, True])
def test_single_vectors(N, inplace):
    """Two and three passes over one vector, last tiles that are not full, an
    offset, both directions; then R2C of 2N real points and C2R back."""
    z = rnd(N + 2, N)
    bx = J.CBlock(z.copy().view(np.float32), admit=True)
    by = bx if inplace else J.CBlock(np.zeros(2 * (N + 2), np.float32), admit=True)
    vx, vy = bx.vview(1, 1, N), by.vview(1, 1, N)
    p = J.FFT(J.KIND_CCIP if inplace else J.KIND_CCOP, N, 1.0 / N, J.VSIP_FFT_INV, ntimes=1)
    if inplace:
        p.ccfftip(vx)
    else:
        p.ccfftop(vx, vy)
    by.sync()
    got = by.re.view(np.complex64)
    assert rel(got[1:-1], np.fft.ifft(z[1:-1].astype(np.complex128))) <= tol(N)
    assert np.array_equal(got[[0, -1]], z[[0, -1]] if inplace else np.zeros(2))
    for v in (vx, vy):
        v.destroy()
    for b in {bx, by}:
        b.destroy()
    if inplace:
        return
    x = np.random.default_rng(N).standard_normal(2 * N).astype(np.float32)
    out = np.zeros(2 * N, np.float32)
    bx, bz, bo = (J.RBlock(x, admit=True), J.CBlock(np.zeros(2 * (N + 1), np.float32), admit=True),
                  J.RBlock(out, admit=True))
    vx, vz, vo = bx.vview(0, 1, 2 * N), bz.vview(0, 1, N + 1), bo.vview(0, 1, 2 * N)
    J.FFT(J.KIND_RCOP, 2 * N, 1.0, ntimes=1).rcfftop(vx, vz)
    J.FFT(J.KIND_CROP, 2 * N, 0.5 / N, ntimes=1).crfftop(vz, vo)
    bz.sync()
    bo.sync()
    assert rel(bz.re.view(np.complex64), np.fft.rfft(x.astype(np.float64))) <= tol(2 * N)
    assert rel(out, x.astype(np.float64)) <= 2 * tol(2 * N)
    for v in (vx, vz, vo):
        v.destroy()
    for b in (bx, bz, bo):
        b.destroy()


@pytest.mark.parametrize("ns,nt", [(2, 8), (36, 60), (250, 500), (162, 3000), (700, 1050), (75, 8192), (1029, 128)])
def test_komega_column_major(ns, nt):
    """k-omega (lengths 2^a 3^b 5^c 7^d, as the call takes) in tiles that are not full, one row per tile, compiled-in schedules
    and others: tapered data bit for bit (products rounded in order), power,
    imaginary part and gram against numpy in 64 bits."""
    g = np.random.default_rng(ns + nt)
    nf = nt // 2 + 1
    x = g.standard_normal((ns, nt)).astype(np.float32)
    ts, arr = (g.uniform(0.5, 1.0, n).astype(np.float32) for n in (nt, ns))
    gram = g.uniform(0, 1, (nf, ns)).astype(np.float32)
    scale = np.float32(1.0 / (ns * nt))
    bx, bg = J.RBlock(x.reshape(-1).copy(), admit=True), J.RBlock(gram.reshape(-1).copy(), admit=True)
    bf = J.CBlock(np.zeros(2 * nf * ns, np.float32), admit=True)
    bt, ba = J.RBlock(ts, admit=True), J.RBlock(arr, admit=True)
    vx, vf, vg = bx.view(0, nt, ns, 1, nt), bf.view(0, 1, ns, ns, nf), bg.view(0, 1, ns, ns, nf)
    vt, va = bt.vview(0, 1, nt), ba.vview(0, 1, ns)
    rc = J.FFTM(J.KIND_RCOP, ns, nt, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW, ntimes=1)
    cc = J.FFTM(J.KIND_CCIP, ns, nf, 1.0, J.VSIP_FFT_FWD, J.VSIP_COL, ntimes=1)
    assert J.lib().jvsip_komega_f(rc.h, cc.h, vt.h, va.h, vx.h, vf.h, float(scale), vg.h) == 0, J.last_error()
    for b in (bx, bf, bg):
        b.sync()
    tapered = (ts[None, :] * x) * arr[:, None]
    assert np.array_equal(bx.a.reshape(ns, nt), tapered)
    z = np.fft.fft(np.fft.rfft(tapered.astype(np.float64)).T)
    power = float(scale) * np.abs(z) ** 2
    f = bf.re.reshape(nf, ns, 2)
    assert rel(f[..., 0], power) <= 2 * tol(ns * nt)
    assert rel(f[..., 1], z.imag) <= tol(ns * nt)
    assert rel(bg.a.reshape(nf, ns), gram.astype(np.float64) + power) <= 2 * tol(ns * nt)
    for v in (vx, vf, vg, vt, va):
        v.destroy()
    for b in (bx, bf, bg, bt, ba):
        b.destroy()


@pytest.mark.parametrize("N", [22, 81, 100, 143, 600, 1000, 2197, 5632, 6561, 8125])
def test_double_rows_and_columns(N):
    """Double precision: rows that fill their warps better here than in the
    shared-memory kernel, and lengths with factors 11 and 13 (columns too).
    Tolerance: rel-L2 1e-14 log2 N, the library's bound for double precision."""
    g = np.random.default_rng(N)
    for m, col in ((1, False), (37, False), (3, True)):
        z = g.standard_normal(m * N) + 1j * g.standard_normal(m * N)
        y = np.zeros(2 * m * N)
        bx, by = J.CBlock(z.view(np.float64).copy(), admit=True), J.CBlock(y, admit=True)
        shape = (0, m, N, 1, m) if col else (0, N, m, 1, N)
        vx, vy = bx.view(*shape), by.view(*shape)
        a, b = (N, m) if col else (m, N)
        p = J.FFTM(J.KIND_CCOP, a, b, 1.0 / N, J.VSIP_FFT_INV, J.VSIP_COL if col else J.VSIP_ROW, dtype=np.float64)
        p.ccfftmop(vx, vy)
        by.sync()
        ref = np.fft.ifft(z.reshape(a, b), axis=0 if col else 1)
        assert rel(y.view(np.complex128).reshape(a, b), ref) <= 1e-14 * np.log2(N)
        for v in (vx, vy):
            v.destroy()
        for blk in (bx, by):
            blk.destroy()
