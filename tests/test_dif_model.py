"""The in-place mixed-radix decomposition of jvsip_gb300/csrc/jv_dif.cuh
restated in numpy: positions, twiddles and output order of every pass, the
block pitch, and the pair passes of the real transforms, against numpy's FFT
for schedules of two to five passes in several orders (no GPU needed)."""
import os
import re

import numpy as np
import pytest

SCHEDULES = [[2, 2], [3, 5], [13, 11], [16, 16], [10, 10, 10], [8, 15, 10], [5, 3, 2, 7], [2, 3, 2, 2, 5],
             [12, 5, 4], [4, 5, 12], [11, 2, 13]]


def passes(x, rad, P1):
    """The shared-memory image after every pass but the last; index k1*P1 + rest."""
    N = len(x)
    s = np.full(rad[0] * P1, np.nan + 0j)
    M = N
    for p, R in enumerate(rad[:-1]):
        S = M // R
        w = np.exp(-2j * np.pi * np.outer(np.arange(R), np.arange(S)) / M)
        F = np.exp(-2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
        if p == 0:
            y = F @ x.reshape(R, S) * w
            for k in range(R):
                s[k * P1:k * P1 + S] = y[k]
        else:
            NB1, seen = N // rad[0] // R, set()
            for j in range(N // R):
                k1, u = divmod(j, NB1)
                c, n = divmod(u, S)
                pos = k1 * P1 + u + c * (M - S) + S * np.arange(R)
                assert not seen.intersection(pos)
                seen.update(pos)
                s[pos] = (F @ s[pos]) * w[:, n]
        M = S
    return s


def last(s, rad, P1, q):
    """Butterfly q of the last pass: outputs q + r*N/R."""
    N, R = int(np.prod(rad)), rad[-1]
    k1, rem = q % rad[0], q // rad[0]
    pos, S = k1 * P1, N // rad[0]
    for r in rad[1:-1]:
        S //= r
        pos += rem % r * S
        rem //= r
    F = np.exp(-2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
    return F @ s[pos:pos + R]


@pytest.mark.parametrize("rad", SCHEDULES, ids=str)
@pytest.mark.parametrize("pad", [0, 3])
def test_passes_give_the_dft(rad, pad):
    N = int(np.prod(rad))
    rng = np.random.default_rng(N)
    x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    P1 = N // rad[0] + pad
    s = passes(x, rad, P1)
    Q, y = N // rad[-1], np.empty(N, complex)
    for q in range(Q):
        y[q::Q] = last(s, rad, P1, q)
    assert np.linalg.norm(y - np.fft.fft(x)) <= 1e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("rad", SCHEDULES, ids=str)
def test_r2c_pair_pass(rad):
    N = int(np.prod(rad))
    x = np.random.default_rng(N).standard_normal(2 * N)
    P1 = N // rad[0] + 1
    s = passes(x[0::2] + 1j * x[1::2], rad, P1)
    R = rad[-1]
    Q = N // R
    X = np.full(N + 1, np.nan + 0j)
    for q in range(Q // 2 + 1):
        u, v = last(s, rad, P1, q), last(s, rad, P1, Q - q if q else 0)
        for r in range(R):
            k = q + r * Q
            z, n = u[r], v[(R - r) % R] if q == 0 else v[R - 1 - r]
            w = np.exp(-1j * np.pi * k / N)
            a, b = z + np.conj(n), -1j * w * (z - np.conj(n))
            X[k] = (a + b) / 2
            if (q and 2 * q != Q) or (q == 0 and r == 0):
                X[N - k] = np.conj(a - b) / 2
    assert np.linalg.norm(X - np.fft.rfft(x)) <= 1e-12 * np.linalg.norm(X)


@pytest.mark.parametrize("rad", SCHEDULES, ids=str)
def test_c2r_pair_pass_partners(rad):
    """Butterflies n' and S - n' of the first pass hold each other's X_{N-n}."""
    N = int(np.prod(rad))
    R, S = rad[0], N // rad[0]
    done = []
    for j in range(S // 2 + 1):
        u, w = [j + r * S for r in range(R)], [S - j + r * S for r in range(R)]
        assert max(w) <= N and all(u[r] + w[R - 1 - r] == N for r in range(R))
        done += u + (w if j and 2 * j != S else [])
    assert sorted(done) == list(range(N))


# ---------------------------------------------------------------- compiled-in schedules
def table():
    src = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jvsip_gb300", "csrc",
                            "jv_dif_table.h")).read()
    out = {}
    for name, body in re.findall(r"#define (JV_DIF_\w+)\(X\) \\\n((?:    X\([\d, ]+\)(?: \\)?\n?)+)", src):
        kind = "c2c" if "LENGTHS" in name else name.split("_")[2].lower()
        out.setdefault(kind, []).extend([int(v) for v in row.split(",")] for row in re.findall(r"X\(([\d, ]+)\)", body))
    return out


def test_table_covers_its_lengths_once():
    smooth = [n for n in range(40, 16385) if _smooth(n)]
    t = table()
    assert [r[0] for r in t["c2c"]] == smooth
    for kind in ("r2c", "c2r"):
        assert [r[0] for r in t[kind]] == [n for n in smooth if n <= 8192]
    assert [r[0] for r in t["rows"]] == [n for n in range(40, 16385) if any(n % p == 0 and _smooth(n // p) for p in (7, 11, 13))]


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


@pytest.mark.parametrize("kind", ["c2c", "r2c", "c2r", "rows"])
def test_table_entries_fit_the_kernel(kind):
    """Radices give the length and are codelets (pair passes at most 10), blocks
    do not overlap, every CTA's threads and shared memory exist, and index
    products stay below the multiply-high limit."""
    for row in table()[kind]:
        N, P1, T, VPB = row[:4]
        VC, TC, TV, TL, rad = (*row[4:8], row[8:]) if kind == "c2c" else (0, 0, 0, 0, row[4:])
        assert int(np.prod(rad)) == N and len(rad) >= 2 and all(2 <= r <= 16 for r in rad), row
        assert N // rad[0] <= P1 < N // rad[0] + 16, row
        if kind == "r2c":
            assert rad[-1] <= 10, row
        if kind == "c2r":
            assert rad[0] <= 10, row
        tiles = [(VPB, T)] + [(v, t) for v, t in ((VC, TC), (16, TV), (4, TL)) if v and t]
        for v, t in tiles:
            assert t % 32 == 0 and 64 <= t <= 1024, row
            # the long vectors' first pass keeps N more elements behind its tile of 16
            assert (v * (rad[0] * P1 + 1) + (N if v == 16 and t == TV else 0)) * 8 <= 227 * 1024, row
            assert v * N // min(rad) * (N // min(rad)) < 2 ** 32, row
        for v, t in tiles[1:]:
            assert v & (v - 1) == 0 and t % v == 0, row
