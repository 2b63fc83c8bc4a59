"""The work that users of this library give it, as measurable cases.

Each case is a dict of plain values; its "family" says which public call it makes:

  rows     vsip_ccfftmop_f / vsip_ccfftmip_f, VSIP_ROW, on admitted blocks
  cols     vsip_ccfftmop_f, VSIP_COL, on admitted blocks
  r2c      vsip_rcfftmop_f, VSIP_ROW, on admitted blocks
  c2r      vsip_crfftmop_f, VSIP_ROW, on admitted blocks
  vector   vsip_ccfftop_f on one admitted vector
  double   vsip_ccfftmop_d, VSIP_ROW, on admitted blocks
  batch    jvsip_fftm_batch_run_f: many uneven calls as one
  komega   jvsip_komega_f: the k-omega power estimate of sensor data
  host     the pyJvsip-style FFT class on numpy-backed (not admitted) blocks

Admitted blocks stay on the GPU from call to call, so a pass returns a
`Resident`: it reads an output back (jvsip_cblocksync_*) when the output is
looked at, as a VSIPL program does with vsip_cblockrelease_*.
"""
import ctypes as C
import math

import numpy as np
import torch

import jvsip_gb300 as J
from jvsip_gb300 import pyjvsip, synth

# lengths of real use are products of small primes; the library's own
# generators (synth.smooth_lengths) draw from the same set
SMOOTH = synth.smooth_lengths(64, 16384)


def listed():
    return [
        # a small matrix, as one processing interval of a streaming program has it:
        # the launch and the latency of a few blocks count, not bytes
        {"name": "rows_64x1024", "family": "rows", "count": 64, "length": 1024, "dir": "fwd",
         "in_place": False, "storage": "interleaved"},
        # the large plain batch that the library's headline figure is quoted on
        {"name": "rows_65536x4096", "family": "rows", "count": 65536, "length": 4096, "dir": "fwd",
         "in_place": False, "storage": "interleaved"},
        # records of a decimal length transformed in place and back (inverse), an odd number of them
        {"name": "rows_ip_6001x2400", "family": "rows", "count": 6001, "length": 2400, "dir": "inv",
         "in_place": True, "storage": "interleaved"},
        # lengths with a factor that has no power-of-two schedule (8 x 8 x 8 x 11)
        {"name": "rows_4096x5632", "family": "rows", "count": 4096, "length": 5632, "dir": "fwd",
         "in_place": False, "storage": "interleaved"},
        # transforms down the columns of a row-major matrix (Doppler processing)
        {"name": "cols_1000x4096", "family": "cols", "count": 4096, "length": 1000, "dir": "fwd"},
        # real records to spectra, and spectra back to real records of another length and an odd count
        {"name": "r2c_4096x1536", "family": "r2c", "count": 4096, "length": 1536},
        {"name": "c2r_5001x3000", "family": "c2r", "count": 5001, "length": 3000},
        # one long vector (spectrum analysis of a whole recording)
        {"name": "vector_16777216", "family": "vector", "length": 1 << 24, "dir": "fwd"},
        # double precision records
        {"name": "double_16384x4096", "family": "double", "count": 16384, "length": 4096, "dir": "fwd"},
        # many small independent jobs of uneven lengths, counts, directions and majors
        {"name": "batch_160", "family": "batch", "instances": 160, "mix": 6},
        # the k-omega power estimate of a sensor array
        {"name": "komega_4096x4096", "family": "komega", "sensors": 4096, "samples": 4096},
        # a Python program that keeps its data in numpy arrays and transforms them now and then
        {"name": "host_256x1000", "family": "host", "count": 256, "length": 1000, "dir": "fwd"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _smooth(rng, lo, hi, even=False):
    """Half powers of two, half any product of 2, 3 and 5, spread over the logarithm."""
    v = _log(rng, lo, hi)
    if rng.random() < 0.4:
        return 1 << max(math.ceil(math.log2(lo)), min(math.floor(math.log2(hi)), round(math.log2(v))))
    return min((n for n in SMOOTH if lo <= n <= hi and not (even and n % 2)), key=lambda n: abs(math.log(n / v)))


def _count(rng, length, lo, hi):
    """How many transforms make between lo and hi points together."""
    return max(1, round(_log(rng, lo, hi) / length))


def draw(rng):
    family = rng.choice(["rows", "rows", "rows", "cols", "cols", "r2c", "c2r", "vector", "double", "batch", "komega",
                         "host"])
    way = rng.choice(["fwd", "inv"])
    if family == "rows":
        if rng.random() < 0.25:
            p = rng.choice([11, 13])
            length = p * round(_log(rng, 8, 1024) / 8) * 8 if rng.random() < 0.5 else p << rng.randint(3, 10)
            while max(_prime_factors(length)) > 13:
                length += 8 * p
        else:
            length = _smooth(rng, 64, 16384)
        return {"family": family, "count": _count(rng, length, 1 << 16, 1 << 25), "length": length, "dir": way,
                "in_place": rng.random() < 0.3, "storage": "split" if rng.random() < 0.2 else "interleaved"}
    if family == "cols":
        length = _smooth(rng, 64, 16384)
        return {"family": family, "count": max(16, _count(rng, length, 1 << 18, 1 << 24)), "length": length, "dir": way}
    if family in ("r2c", "c2r"):
        length = _smooth(rng, 128, 16384, even=True)
        return {"family": family, "count": _count(rng, length, 1 << 18, 1 << 25), "length": length}
    if family == "vector":
        n = round(_log(rng, 14, 24.4))
        length = 1 << min(24, n)
        if rng.random() < 0.4:  # a decimal or three-smooth length of the same order
            length = min((v * s for v in (1000, 3 << 10, 5 << 10, 10000) for s in SMOOTH if v * s <= 1 << 24),
                         key=lambda m: abs(math.log(m / (length * 0.8))))
        return {"family": family, "length": length, "dir": way}
    if family == "double":
        length = _smooth(rng, 64, 8192)
        return {"family": family, "count": _count(rng, length, 1 << 16, 1 << 24), "length": length, "dir": way}
    if family == "batch":
        return {"family": family, "instances": round(_log(rng, 20, 160)), "mix": rng.randint(100, 9999)}
    if family == "komega":
        return {"family": family, "sensors": 4096 if rng.random() < 0.1 else _smooth(rng, 64, 2560),
                "samples": _smooth(rng, 256, 8192, even=True)}
    length = _smooth(rng, 64, 4096)
    return {"family": family, "count": _count(rng, length, 1 << 13, 1 << 21), "length": length, "dir": way}


def _prime_factors(n):
    out, p = [], 2
    while n > 1:
        while n % p == 0:
            out.append(p)
            n //= p
        p += 1
    return out or [1]


# ---------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(n, seed, dtype=torch.float32):
    """n samples of N(0,1) on the GPU."""
    return torch.randn(n, device="cuda", dtype=dtype, generator=_generator(seed))


def _spectra(count, length, seed):
    """Hermitian-consistent spectra of `count` real rows, as interleaved scalars."""
    z = torch.fft.rfft(_normal(count * length, seed).view(count, length) / math.sqrt(length))
    z[:, 0].imag.zero_()
    z[:, -1].imag.zero_()
    return torch.view_as_real(z).reshape(-1)


def _taper(n):
    """A Tukey window (a tenth cosine, flat between), so that data tapered again and again stays at its level."""
    k = torch.arange(n, dtype=torch.float64)
    edge = max(1, n // 20)
    d = torch.minimum(k, n - 1 - k)
    return torch.where(d < edge, 0.5 * (1 - torch.cos(math.pi * (d + 1) / (edge + 1))), torch.ones(())).float()


def _host(t):
    return t.cpu().numpy()


class Resident(dict):
    """A pass's outputs by name, still on the GPU; looking one up reads it back. Keeps the state that holds them."""

    def __init__(self, state):
        super().__init__(state.out)
        self.state = state

    def __getitem__(self, name):
        block, arrays = super().__getitem__(name)
        block.sync()
        return arrays


class State:
    """The blocks, views and plans that a program holds between calls, released with it."""

    def __init__(self):
        self.blocks, self.views, self.plans, self.batch = [], [], [], None
        self.call, self.out, self.host = None, None, None

    def cblock(self, re, im=None, upload=True):
        self.blocks.append(J.CBlock(re, im, admit=True, update=upload))
        return self.blocks[-1]

    def rblock(self, a, upload=True):
        self.blocks.append(J.RBlock(a, admit=True, update=upload))
        return self.blocks[-1]

    def view(self, block, *a):
        self.views.append(block.view(*a))
        return self.views[-1]

    def vview(self, block, *a):
        self.views.append(block.vview(*a))
        return self.views[-1]

    def plan(self, p):
        self.plans.append(p)
        return p

    def __del__(self):
        if self.batch:
            J.lib().jvsip_fftm_batch_destroy_f(self.batch)
        for p in self.plans:
            p.destroy()
        for v in self.views:
            v.destroy()
        for b in self.blocks:
            b.destroy()


def _dir(case):
    return J.VSIP_FFT_FWD if case["dir"] == "fwd" else J.VSIP_FFT_INV


def _scale(case):
    """1 forward, 1/N back; in place 1/sqrt(N) each way, which keeps the data's level from call to call."""
    n = case["length"]
    if case.get("in_place"):
        return float(np.float32(1.0 / math.sqrt(n)))
    return 1.0 if case["dir"] == "fwd" else float(np.float32(1.0 / n)) if case["family"] != "double" else 1.0 / n


def prepare(case, seed):
    return globals()["_prepare_" + case["family"]](case, seed)


def _prepare_rows(case, seed):
    m, n, s = case["count"], case["length"], State()
    split, ip = case["storage"] == "split", case["in_place"]
    x = _normal(2 * m * n, seed)
    if split:
        x = [_host(x[: m * n]), _host(x[m * n:])]
        y = x if ip else [np.empty_like(x[0]), np.empty_like(x[1])]
    else:
        x = [_host(x)]
        y = x if ip else [np.empty_like(x[0])]
    bx = s.cblock(*x)
    vx = s.view(bx, 0, n, m, 1, n)
    p = s.plan(J.FFTM(J.KIND_CCIP if ip else J.KIND_CCOP, m, n, _scale(case), _dir(case), J.VSIP_ROW))
    if ip:
        s.call, by = (lambda: p.ccfftmip(vx)), bx
    else:
        by = s.cblock(*y, upload=False)
        vy = s.view(by, 0, n, m, 1, n)
        s.call = lambda: p.ccfftmop(vx, vy)
    s.out = {"y": (by, y if split else y[0])}
    return s


def _prepare_cols(case, seed):
    m, n, s = case["count"], case["length"], State()
    x = _host(_normal(2 * m * n, seed))
    y = np.empty_like(x)
    bx, by = s.cblock(x), s.cblock(y, upload=False)
    vx, vy = (s.view(b, 0, m, n, 1, m) for b in (bx, by))
    p = s.plan(J.FFTM(J.KIND_CCOP, n, m, _scale(case), _dir(case), J.VSIP_COL))
    s.call, s.out = (lambda: p.ccfftmop(vx, vy)), {"y": (by, y)}
    return s


def _prepare_r2c(case, seed):
    m, n, s = case["count"], case["length"], State()
    h = n // 2 + 1
    x, z = _host(_normal(m * n, seed)), np.empty(2 * m * h, np.float32)
    bx, bz = s.rblock(x), s.cblock(z, upload=False)
    vx, vz = s.view(bx, 0, n, m, 1, n), s.view(bz, 0, h, m, 1, h)
    p = s.plan(J.FFTM(J.KIND_RCOP, m, n, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW))
    s.call, s.out = (lambda: p.rcfftmop(vx, vz)), {"z": (bz, z)}
    return s


def _prepare_c2r(case, seed):
    m, n, s = case["count"], case["length"], State()
    h = n // 2 + 1
    z, x = _host(_spectra(m, n, seed)), np.empty(m * n, np.float32)
    bz, bx = s.cblock(z), s.rblock(x, upload=False)
    vz, vx = s.view(bz, 0, h, m, 1, h), s.view(bx, 0, n, m, 1, n)
    p = s.plan(J.FFTM(J.KIND_CROP, m, n, float(np.float32(1.0 / n)), J.VSIP_FFT_INV, J.VSIP_ROW))
    s.call, s.out = (lambda: p.crfftmop(vz, vx)), {"x": (bx, x)}
    return s


def _prepare_vector(case, seed):
    n, s = case["length"], State()
    x = _host(_normal(2 * n, seed))
    y = np.empty_like(x)
    bx, by = s.cblock(x), s.cblock(y, upload=False)
    vx, vy = s.vview(bx, 0, 1, n), s.vview(by, 0, 1, n)
    p = s.plan(J.FFT(J.KIND_CCOP, n, _scale(case), _dir(case)))
    s.call, s.out = (lambda: p.ccfftop(vx, vy)), {"y": (by, y)}
    return s


def _prepare_double(case, seed):
    m, n, s = case["count"], case["length"], State()
    x = _host(_normal(2 * m * n, seed, torch.float64))
    y = np.empty_like(x)
    bx, by = s.cblock(x), s.cblock(y, upload=False)
    vx, vy = (s.view(b, 0, n, m, 1, n) for b in (bx, by))
    p = s.plan(J.FFTM(J.KIND_CCOP, m, n, _scale(case), _dir(case), J.VSIP_ROW, dtype=np.float64))
    s.call, s.out = (lambda: p.ccfftmop(vx, vy)), {"y": (by, y)}
    return s


def _jobs(case):
    return synth.batch_sequence(case["instances"], seed=case["mix"])


def _prepare_batch(case, seed):
    s, jobs, off = State(), _jobs(case), 0
    total = sum(n * m for n, m, _, _ in jobs)
    x = _host(_normal(2 * total, seed))
    y = np.empty_like(x)
    bx, by = s.cblock(x), s.cblock(y, upload=False)
    for n, m, way, major in jobs:
        if major == J.VSIP_ROW:
            s.plan(J.FFTM(J.KIND_CCOP, m, n, 1.0 if way < 0 else 1.0 / n, way, major))
            shape = (off, n, m, 1, n)
        else:
            s.plan(J.FFTM(J.KIND_CCOP, n, m, 1.0 if way < 0 else 1.0 / n, way, major))
            shape = (off, m, n, 1, m)
        s.view(bx, *shape)
        s.view(by, *shape)
        off += n * m
    lists = [(C.c_void_p * len(jobs))(*[o.h for o in some]) for some in (s.plans, s.views[0::2], s.views[1::2])]
    s.batch = J.lib().jvsip_fftm_batch_create_f(len(jobs), *lists)
    if not s.batch:
        J.check("jvsip_fftm_batch_create_f")

    def call():
        if J.lib().jvsip_fftm_batch_run_f(s_batch):
            J.check("jvsip_fftm_batch_run_f")

    s_batch = s.batch
    s.call, s.out = call, {"y": (by, y)}
    return s


def _prepare_komega(case, seed):
    ns, nt, s = case["sensors"], case["samples"], State()
    nf = nt // 2 + 1
    x = _host(_normal(ns * nt, seed))
    f = np.zeros(2 * ns * nf, np.float32)
    g = _host(torch.rand(ns * nf, device="cuda", generator=_generator(seed + 1)))
    bx, bf, bg = s.rblock(x), s.cblock(f), s.rblock(g)
    bt, ba = s.rblock(_host(_taper(nt))), s.rblock(_host(_taper(ns)))
    vx, vf, vg = s.view(bx, 0, nt, ns, 1, nt), s.view(bf, 0, 1, ns, ns, nf), s.view(bg, 0, 1, ns, ns, nf)
    vt, va = s.vview(bt, 0, 1, nt), s.vview(ba, 0, 1, ns)
    rc = s.plan(J.FFTM(J.KIND_RCOP, ns, nt, 1.0, J.VSIP_FFT_FWD, J.VSIP_ROW))
    cc = s.plan(J.FFTM(J.KIND_CCIP, ns, nf, 1.0, J.VSIP_FFT_FWD, J.VSIP_COL))
    scale = _power_scale(case)

    def call():
        if J.lib().jvsip_komega_f(rc.h, cc.h, vt.h, va.h, vx.h, vf.h, scale, vg.h):
            J.check("jvsip_komega_f")

    s.call, s.out = call, {"data": (bx, x), "freq": (bf, f), "gram": (bg, g)}
    return s


def _power_scale(case):
    return float(np.float32(1.0 / (case["sensors"] * case["samples"])))


def _prepare_host(case, seed):
    m, n, s = case["count"], case["length"], State()
    x, y = pyjvsip.create("cmview_f", m, n), pyjvsip.create("cmview_f", m, n)
    x.block.array[:] = _host(_normal(2 * m * n, seed))
    p = pyjvsip.FFT("ccfftmop_f", m, n, _scale(case), _dir(case), J.VSIP_ROW, 0, 0)
    s.call, s.host = (lambda: p.dft(x, y)), y.block.array
    return s


def run(state):
    state.call()
    return state.host if state.out is None else Resident(state)


# ---------------------------------------------------------------------------- what a pass cannot do without
def _c2c_flops(n, count=1):
    return 5.0 * n * math.log2(n) * count


def work(case):
    f = case["family"]
    if f == "batch":
        jobs = _jobs(case)
        return {"bytes": 16.0 * sum(n * m for n, m, _, _ in jobs), "flops": sum(_c2c_flops(n, m) for n, m, _, _ in jobs)}
    if f == "komega":
        ns, nt = case["sensors"], case["samples"]
        nf = nt // 2 + 1
        return {"bytes": 8.0 * ns * nt + 8.0 * ns * nf + 8.0 * ns * nf + 4.0 * (ns + nt),
                "flops": _c2c_flops(nt, ns) / 2 + _c2c_flops(ns, nf) + 2.0 * ns * nt + 5.0 * ns * nf}
    n, m = case["length"], case.get("count", 1)
    if f in ("r2c", "c2r"):
        return {"bytes": m * (4.0 * n + 8.0 * (n // 2 + 1)), "flops": _c2c_flops(n, m) / 2}
    return {"bytes": (32.0 if f == "double" else 16.0) * m * n, "flops": _c2c_flops(n, m)}


# ---------------------------------------------------------------------------- the same in 64 bits
def _fft64(z, case, dim=-1):
    """The unnormalised transform of the case's direction times its scale."""
    y = torch.fft.fft(z, dim=dim) if case["dir"] == "fwd" else torch.fft.ifft(z, dim=dim, norm="forward")
    return y.mul_(_scale(case))


def _scalars(z):
    return torch.view_as_real(z).reshape(-1)


def exact(case, seed):
    f = case["family"]
    if f == "batch":
        x = _normal(2 * sum(n * m for n, m, _, _ in _jobs(case)), seed).double()
        out, off = [], 0
        for n, m, way, major in _jobs(case):
            z = torch.view_as_complex(x[2 * off:2 * (off + n * m)].view(-1, 2))
            z = z.view(m, n) if major == J.VSIP_ROW else z.view(n, m)
            dim = 1 if major == J.VSIP_ROW else 0
            y = torch.fft.fft(z, dim=dim) if way < 0 else torch.fft.ifft(z, dim=dim)
            out.append(_scalars(y.contiguous()))
            off += n * m
        return {"y": torch.cat(out)}
    if f == "komega":
        ns, nt = case["sensors"], case["samples"]
        nf = nt // 2 + 1
        x = _normal(ns * nt, seed).view(ns, nt).double() * _taper(nt).cuda().double() * _taper(ns).cuda().double()[:, None]
        g = torch.rand(ns * nf, device="cuda", generator=_generator(seed + 1)).double().view(nf, ns)
        z = torch.fft.fft(torch.fft.rfft(x).t().contiguous())
        power = _power_scale(case) * (z.real.square() + z.imag.square())
        return {"data": x.reshape(-1), "freq": torch.stack([power, z.imag], -1).reshape(-1), "gram": (g + power).reshape(-1)}
    n, m = case["length"], case.get("count", 1)
    if f == "r2c":
        return {"z": _scalars(torch.fft.rfft(_normal(m * n, seed).view(m, n).double()))}
    if f == "c2r":
        z = torch.view_as_complex(_spectra(m, n, seed).double().view(m, n // 2 + 1, 2))
        return {"x": torch.fft.irfft(z, n, norm="forward").mul_(float(np.float32(1.0 / n))).reshape(-1)}
    if f == "rows" and case["storage"] == "split":
        x = _normal(2 * m * n, seed).double()
        y = _fft64(torch.complex(x[: m * n].view(m, n), x[m * n:].view(m, n)), case)
        return {"y": [y.real.reshape(-1), y.imag.reshape(-1)]}
    x = _normal(2 * m * n, seed, torch.float64 if f == "double" else torch.float32).double()
    z = torch.view_as_complex(x.view(-1, 2))
    if f == "cols":
        return {"y": _scalars(_fft64(z.view(n, m), case, dim=0).contiguous())}
    y = _scalars(_fft64(z.view(m, n), case))
    return y if f == "host" else {"y": y}
